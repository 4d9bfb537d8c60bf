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
// 9.0 us (row kernel) and 6.9 us (tiled kernel) per term before, 2.9 us here.
#include "el_coop.cuh"

#include <algorithm>

namespace el {

namespace {

constexpr int CHEB_TERMS = 1024;   // coefficients passed with the launch
constexpr int CHEB_THREADS = 512;

template <typename S>
struct ChebArgs {
  int n, tb, M, nctas, poll_limit;         // tb: bits of a tile
  S al[2], be[2];           // t_{m+1} = (al H + be) t_m - t_{m-1}: first term, later ones
  const S *diagV;
  S delta[18], up_re[18], up_im[18];
  void *psi;
  void *pub;                // [2][2^n] published vectors
  unsigned *bar;
  int *err;
  double c0[2];
  S c[2 * (CHEB_TERMS + 1)];
};

// RA: real amplitudes.  R rows per thread, CHEB_THREADS (or fewer, R = 1)
// rows apart.  Tiles of a basis with several have 2^9 R rows.
//
// Over many steps the digits of a complex64 state depend on how every term
// rounds: coefficients one FP32 unit off are another H, and its phase grows
// with the time.  So al and be are formed in FP64 and rounded once, the
// multiply-adds are spelled out, and flips and detunings are summed in a stated
// order: bits k, k + G, ... ascending, then the G sums in a butterfly (G = 4
// below 17 sites, as where four lanes share a row in the row kernel).
template <typename S, bool RA, int R, int G>
__global__ void __launch_bounds__(CHEB_THREADS, 1) k_cheb_coop(const __grid_constant__ ChebArgs<S> P) {
  typedef typename VecT<S, true>::type V2;
  constexpr int TB = 9 + (R == 2) + 2 * (R == 4);          // bits of a tile, where there are several
  constexpr int NH = R == 2 && G == 4 ? 0 : 7;             // bits above it, at most (2 rows below 17 sites: one tile)
  constexpr bool AHEAD = NH && R <= 2;                     // read the other tiles' rows first: registers for NH R values
  extern __shared__ __align__(16) unsigned char cheb_smem[];
  V2 *const tile = reinterpret_cast<V2 *>(cheb_smem);      // [2][2^tb]
  const int rows = 1 << P.tb, nt = (int)blockDim.x;
  const int64_t dim = (int64_t)1 << P.n, base = (int64_t)blockIdx.x << P.tb;
  V2 *const psi = reinterpret_cast<V2 *>(P.psi) + base;
  V2 *const pub = reinterpret_cast<V2 *>(P.pub);
  unsigned gen = 0;
  V2 x[R], z[R], acc[R];
  S d[R];
  auto butterfly = [](const S (&v)[G]) -> S {
    if constexpr (G == 4) return (v[0] + v[2]) + (v[1] + v[3]);
    else return v[0];
  };
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const int i = threadIdx.x + q * nt;
    x[q] = psi[i];
    z[q].x = z[q].y = S(0);
    acc[q].x = (S)(P.c0[0] * (double)x[q].x - P.c0[1] * (double)x[q].y);
    acc[q].y = (S)(P.c0[0] * (double)x[q].y + P.c0[1] * (double)x[q].x);
    S s[G];
#pragma unroll
    for (int l = 0; l < G; ++l) {
      s[l] = S(0);
      for (int k = l; k < P.n; k += G)
        if (((base + i) >> k) & 1) s[l] += P.delta[k];
    }
    d[q] = butterfly(s) + P.diagV[base + i];
    tile[i] = x[q];
  }
  __syncthreads();
  for (int m = 1; m <= P.M; ++m) {
    // t_{m-1} of the other tiles: the state itself, then the published terms
    const V2 *other = m == 1 ? reinterpret_cast<const V2 *>(P.psi) : pub + ((m & 1) ? dim : 0);
    const V2 *mine = tile + ((m & 1) ? 0 : rows);
    S hx[R][G], hy[R][G];
#pragma unroll
    for (int q = 0; q < R; ++q)
#pragma unroll
      for (int l = 0; l < G; ++l) hx[q][l] = hy[q][l] = S(0);
    // h += the flip with amplitude (ar, +- ai) of a row with value v there
    auto add = [](S &h0, S &h1, S ar, S ai, V2 v) {
      if constexpr (RA) {
        h0 = fma(ar, v.x, h0);
        h1 = fma(ar, v.y, h1);
      } else {
        h0 += fma(ar, v.x, -(ai * v.y));
        h1 += fma(ar, v.y, ai * v.x);
      }
    };
    auto skip = [&](int k) { return P.up_re[k] == S(0) && (RA || P.up_im[k] == S(0)); };
    V2 far[AHEAD ? NH : 1][R];
    if (AHEAD && P.nctas > 1) {
#pragma unroll
      for (int j = 0; j < NH; ++j) {
        if (TB + j >= P.n) continue;
        const V2 *p = other + (base ^ ((int64_t)1 << (TB + j)));
#pragma unroll
        for (int q = 0; q < R; ++q) far[j][q] = p[threadIdx.x + q * nt];
      }
    }
    auto near = [&](int k, int l) {
      if (skip(k)) return;
      const S ar = P.up_re[k], im = RA ? S(0) : P.up_im[k];
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int i = threadIdx.x + q * nt;
        add(hx[q][l % G], hy[q][l % G], ar, ((i >> k) & 1) ? im : -im, mine[i ^ (1 << k)]);
      }
    };
    const int whole = P.tb & ~3;
    for (int k = 0; k < whole; k += 4) { near(k, 0); near(k + 1, 1); near(k + 2, 2); near(k + 3, 3); }
    if (P.tb > whole) near(whole, 0);
    if (P.tb > whole + 1) near(whole + 1, 1);
    if (P.tb > whole + 2) near(whole + 2, 2);
    if (P.nctas > 1) {
#pragma unroll
      for (int j = 0; j < NH; ++j) {
        const int k = TB + j;
        if (k >= P.n || skip(k)) continue;
        const S ar = P.up_re[k], im = RA ? S(0) : P.up_im[k];
        const S ai = ((blockIdx.x >> j) & 1) ? im : -im;
        const V2 *p = other + (base ^ ((int64_t)1 << k));
#pragma unroll
        for (int q = 0; q < R; ++q) {
          V2 v;
          if constexpr (AHEAD) v = far[j][q];
          else v = p[threadIdx.x + q * nt];
          add(hx[q][k % G], hy[q][k % G], ar, ai, v);
        }
      }
    }
    const S al = P.al[m > 1], be = P.be[m > 1];
    const S cr = P.c[2 * m], ci = P.c[2 * m + 1];
    V2 *const next = tile + ((m & 1) ? rows : 0);
    V2 *const out = pub + ((m & 1) ? 0 : dim) + base;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int i = threadIdx.x + q * nt;
      V2 y;
      y.x = fma(al, fma(d[q], x[q].x, butterfly(hx[q])), be * x[q].x) - z[q].x;
      y.y = fma(al, fma(d[q], x[q].y, butterfly(hy[q])), be * x[q].y) - z[q].y;
      acc[q].x += fma(cr, y.x, -(ci * y.y));
      acc[q].y += fma(cr, y.y, ci * y.x);
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

// n: sites; R: rows per thread
template <typename S, bool RA>
const void *cheb_fn(int n, int R) {
  if (R == 1) return (const void *)k_cheb_coop<S, RA, 1, 4>;
  if (R == 4) return (const void *)k_cheb_coop<S, RA, 4, 1>;
  return n <= 16 ? (const void *)k_cheb_coop<S, RA, 2, 4> : (const void *)k_cheb_coop<S, RA, 2, 1>;
}

template <typename S>
int launch_cheb(el_ctx *ctx, const el_ham *h, const S *diagV, void *psi, const ChebPlan &plan) {
  const int n = h->n;
  // one tile up to 2^10 rows (no grid barrier), then tiles of 512 rows until
  // they number 128, then more rows per thread
  const int tb = n <= 10 ? n : std::max(9, n - 7);
  const int R = std::max(1, (1 << tb) / CHEB_THREADS);
  const int threads = (1 << tb) / R;
  const int nctas = 1 << (n - tb);
  const size_t es = 2 * sizeof(S);
  char *pub = (char *)workspace(ctx, 17, 2 * es * ((size_t)1 << n) + 16);
  if (!pub) return EL_ENOMEM;
  ChebArgs<S> P;
  memset(&P, 0, offsetof(ChebArgs<S>, c));
  P.n = n; P.tb = tb; P.M = plan.M; P.nctas = nctas; P.poll_limit = 1 << 22;
  P.al[0] = (S)(1.0 / plan.a); P.be[0] = (S)(-plan.b / plan.a);
  P.al[1] = (S)(2.0 / plan.a); P.be[1] = (S)(-2.0 * plan.b / plan.a);
  P.diagV = diagV;
  for (int k = 0; k < n; ++k) {
    P.delta[k] = (S)h->delta[k];
    P.up_re[k] = (S)(0.5 * h->om_re[k]);
    P.up_im[k] = (S)(0.5 * h->om_im[k]);
  }
  P.psi = psi; P.pub = pub;
  P.bar = (unsigned *)(pub + 2 * es * ((size_t)1 << n));
  P.err = (int *)(P.bar + 1);
  P.c0[0] = plan.c_re[0]; P.c0[1] = plan.c_im[0];
  for (int m = 0; m <= plan.M; ++m) { P.c[2 * m] = (S)plan.c_re[m]; P.c[2 * m + 1] = (S)plan.c_im[m]; }
  const size_t smem = 2 * es * ((size_t)1 << tb);
  const void *fn = h->drive_complex ? cheb_fn<S, false>(n, R) : cheb_fn<S, true>(n, R);
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

}  // namespace

// Full bases of 5 to 18 sites, sigma^x channels and a real diagonal, a GPU
// with an SM for every tile.
bool cheb_coop_ok(const el_ctx *ctx, const el_ham *h, int dtype, const void *psi, int M) {
  return (uintptr_t)psi % dtype_size(dtype) == 0 && h->basis->layout == EL_LAYOUT_FULL && h->px.empty() &&
         !h->lossy && h->n >= 5 && h->n <= 18 && M <= CHEB_TERMS && sm_count(ctx) >= 128;
}

int cheb_coop(el_ctx *ctx, el_ham *h, int dtype, void *psi, const ChebPlan &plan) {
  if (dtype == EL_C128) return launch_cheb<double>(ctx, h, h->d_diagV64, psi, plan);
  const int rc = ham_diag32(ctx, h);
  if (rc) return rc;
  return launch_cheb<float>(ctx, h, h->d_diagV32, psi, plan);
}

}  // namespace el
