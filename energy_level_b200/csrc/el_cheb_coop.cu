// One Chebyshev step exp(-i CONV H tau) psi on a small full basis as a single
// cooperative launch.
//
// With one launch per term a step on 2^16 rows is a chain of launches that
// each wait for the previous one to drain (6 to 9 us a term, of which the
// arithmetic is a fraction).  Here a CTA keeps a tile of consecutive rows for
// the whole step: t_m, t_{m-1} and the accumulated state of a row stay in its
// thread's registers, flips of the tile's bits are gathers from shared memory,
// flips of the higher bits coalesced reads of the other tiles' rows, which
// every CTA publishes in global memory before the grid barrier that ends a
// term.  Bases of one tile need no grid barrier.  Same recurrence as
// el_cheb_step:
//     t_{m+1} = (2/a) H t_m - (2b/a) t_m - t_{m-1},  acc += c_{m+1} t_{m+1}.
// Bound: per term the barrier and one round trip to L2; 16 sites, complex128:
// 9.0 us (row kernel) and 6.9 us (tiled kernel) per term before, 3.2 us here.
#include "el_coop.cuh"

#include <algorithm>

namespace el {

namespace {

constexpr int CHEB_TERMS = 1024;   // coefficients passed with the launch
constexpr int CHEB_THREADS = 512;

struct ChebArgs {
  int n, tb, M, nctas, poll_limit, cplx;   // tb: bits of a tile
  double a, b;
  const double *diagV;
  const float *diagV32;
  double delta[18], up_re[18], up_im[18];
  void *psi;
  void *pub;                // [2][2^n] published vectors
  unsigned *bar;
  int *err;
  double c[2 * (CHEB_TERMS + 1)];
};

// RA: real amplitudes.  R rows per thread, CHEB_THREADS (or fewer, R = 1)
// rows apart.
template <typename S, bool RA, int R>
__global__ void __launch_bounds__(CHEB_THREADS, 1) k_cheb_coop(const __grid_constant__ ChebArgs P) {
  typedef typename VecT<S, true>::type V2;
  extern __shared__ __align__(16) unsigned char cheb_smem[];
  V2 *const tile = reinterpret_cast<V2 *>(cheb_smem);      // [2][2^tb]
  const int rows = 1 << P.tb, nt = (int)blockDim.x;
  const int64_t dim = (int64_t)1 << P.n, base = (int64_t)blockIdx.x << P.tb;
  V2 *const psi = reinterpret_cast<V2 *>(P.psi) + base;
  V2 *const pub = reinterpret_cast<V2 *>(P.pub);
  const S a = (S)P.a, b = (S)P.b;
  unsigned gen = 0;
  V2 x[R], z[R], acc[R];
  S d[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int i = threadIdx.x + q * nt;
    x[q] = psi[i];
    z[q].x = z[q].y = S(0);
    acc[q].x = (S)P.c[0] * x[q].x - (S)P.c[1] * x[q].y;
    acc[q].y = (S)P.c[0] * x[q].y + (S)P.c[1] * x[q].x;
    S s = S(0);
    for (int k = 0; k < P.n; ++k)
      if (((base + i) >> k) & 1) s += (S)P.delta[k];
    if constexpr (sizeof(S) == 4) d[q] = s + P.diagV32[base + i];
    else d[q] = s + P.diagV[base + i];
    tile[i] = x[q];
  }
  __syncthreads();
  for (int m = 1; m <= P.M; ++m) {
    // t_{m-1} of the other tiles: the state itself, then the published terms
    const V2 *other = m == 1 ? reinterpret_cast<const V2 *>(P.psi) : pub + ((m & 1) ? dim : 0);
    const V2 *mine = tile + ((m & 1) ? 0 : rows);
    V2 h[R];
#pragma unroll
    for (int q = 0; q < R; ++q) h[q].x = h[q].y = S(0);
#pragma unroll 4
    for (int k = P.tb; k < P.n; ++k) {
      const S ar = (S)P.up_re[k];
      const bool set = (blockIdx.x >> (k - P.tb)) & 1;
      const S ai = RA ? S(0) : (S)(set ? P.up_im[k] : -P.up_im[k]);
      if (ar == S(0) && (RA || ai == S(0))) continue;
      const V2 *p = other + (base ^ ((int64_t)1 << k));
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const V2 v = p[threadIdx.x + q * nt];
        h[q].x += ar * v.x;
        h[q].y += ar * v.y;
        if constexpr (!RA) { h[q].x -= ai * v.y; h[q].y += ai * v.x; }
      }
    }
#pragma unroll 4
    for (int k = 0; k < P.tb; ++k) {
      const S ar = (S)P.up_re[k];
      if (ar == S(0) && (RA || P.up_im[k] == 0.0)) continue;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int i = threadIdx.x + q * nt;
        const V2 v = mine[i ^ (1 << k)];
        h[q].x += ar * v.x;
        h[q].y += ar * v.y;
        if constexpr (!RA) {
          const S ai = (S)(((i >> k) & 1) ? P.up_im[k] : -P.up_im[k]);
          h[q].x -= ai * v.y;
          h[q].y += ai * v.x;
        }
      }
    }
    const S al = (m == 1 ? S(1) : S(2)) / a, be = (m == 1 ? -b : S(-2) * b) / a;
    const S cr = (S)P.c[2 * m], ci = (S)P.c[2 * m + 1];
    V2 *const next = tile + ((m & 1) ? rows : 0);
    V2 *const out = pub + ((m & 1) ? 0 : dim) + base;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int i = threadIdx.x + q * nt;
      V2 y;
      y.x = al * (d[q] * x[q].x + h[q].x) + be * x[q].x - z[q].x;
      y.y = al * (d[q] * x[q].y + h[q].y) + be * x[q].y - z[q].y;
      acc[q].x += cr * y.x - ci * y.y;
      acc[q].y += cr * y.y + ci * y.x;
      z[q] = x[q];
      x[q] = y;
      if (m < P.M) {
        next[i] = y;
        if (P.nctas > 1) out[i] = y;
      }
    }
    // the last term needs no publication; after the first one every CTA has
    // to be done with psi before it is overwritten
    if (m < P.M || m == 1) {
      if (P.nctas > 1) coop_sync(P.bar, P.err, P.nctas, P.poll_limit, gen);
      else __syncthreads();
    }
  }
#pragma unroll
  for (int q = 0; q < R; ++q) psi[threadIdx.x + q * nt] = acc[q];
}

template <typename S>
const void *cheb_fn(bool ra, int R) {
  if (ra) return R == 1 ? (const void *)k_cheb_coop<S, true, 1> : R == 2 ? (const void *)k_cheb_coop<S, true, 2>
                                                                          : (const void *)k_cheb_coop<S, true, 4>;
  return R == 1 ? (const void *)k_cheb_coop<S, false, 1> : R == 2 ? (const void *)k_cheb_coop<S, false, 2>
                                                                  : (const void *)k_cheb_coop<S, false, 4>;
}

}  // namespace

// Full bases of 5 to 18 sites, sigma^x channels and a real diagonal, a GPU
// with an SM for every tile.
bool cheb_coop_ok(const el_ctx *ctx, const el_ham *h, int dtype, const void *psi, int M) {
  return (uintptr_t)psi % dtype_size(dtype) == 0 && h->basis->layout == EL_LAYOUT_FULL && h->px.empty() && !h->lossy && h->n >= 5 && h->n <= 18 &&
         M <= CHEB_TERMS && sm_count(ctx) >= 128;
}

int cheb_coop(el_ctx *ctx, el_ham *h, int dtype, void *psi, const ChebPlan &plan) {
  const int n = h->n;
  // one tile up to 2^10 rows (no grid barrier), then tiles of 512 rows until
  // they number 128, then more rows per thread
  const int tb = n <= 10 ? n : std::max(9, n - 7);
  const int R = std::max(1, (1 << tb) / CHEB_THREADS);
  const int threads = (1 << tb) / R;
  const int nctas = 1 << (n - tb);
  const size_t es = dtype_size(dtype);
  char *pub = (char *)workspace(ctx, 17, 2 * es * ((size_t)1 << n) + 16);
  if (!pub) return EL_ENOMEM;
  if (dtype == EL_C64) {
    const int rc = ham_diag32(ctx, h);
    if (rc) return rc;
  }
  ChebArgs P;
  memset(&P, 0, offsetof(ChebArgs, c));
  P.n = n; P.tb = tb; P.M = plan.M; P.nctas = nctas; P.poll_limit = 1 << 22;
  P.a = plan.a; P.b = plan.b;
  P.diagV = h->d_diagV64; P.diagV32 = h->d_diagV32;
  for (int k = 0; k < n; ++k) {
    P.delta[k] = h->delta[k];
    P.up_re[k] = 0.5 * h->om_re[k];
    P.up_im[k] = 0.5 * h->om_im[k];
  }
  P.psi = psi; P.pub = pub;
  P.bar = (unsigned *)(pub + 2 * es * ((size_t)1 << n));
  P.err = (int *)(P.bar + 1);
  for (int m = 0; m <= plan.M; ++m) { P.c[2 * m] = plan.c_re[m]; P.c[2 * m + 1] = plan.c_im[m]; }
  const size_t smem = 2 * es * ((size_t)1 << tb);
  const void *fn = dtype == EL_C64 ? cheb_fn<float>(!h->drive_complex, R) : cheb_fn<double>(!h->drive_complex, R);
  if (smem > 48 * 1024)
    EL_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  EL_CUDA_TRY(ctx, cudaMemsetAsync(P.bar, 0, 2 * sizeof(unsigned), ctx->stream));
  void *kargs[] = {(void *)&P};
  EL_CUDA_TRY(ctx, cudaLaunchCooperativeKernel(fn, dim3(nctas), dim3(threads), kargs, smem, ctx->stream));
  ctx->launches++;
  if (nctas > 1) {
    unsigned err = 0;
    EL_CUDA_TRY(ctx, el::copy(ctx, ctx->h_scalars, P.err, sizeof err, cudaMemcpyDeviceToHost));
    EL_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    memcpy(&err, ctx->h_scalars, sizeof err);
    if (err) return fail(ctx, EL_ECUDA, "cooperative Chebyshev step: grid barrier timed out");
  }
  return EL_OK;
}

}  // namespace el
