// Fused H-apply on the full 2^n basis.
//
// Rows are codes, so bit k flips row r to r ^ 2^k.  A tile is 2^(L + 2)
// consecutive rows; a thread holds one setting of the L low bits and one
// 16-byte chunk of the row for all four settings of the next two bits:
//   - low bits are gathers from the tile in shared memory, one address per
//     bit for all four rows;
//   - the two middle bits are the thread's own registers;
//   - a high bit moves the whole tile by +- 2^k rows: coalesced reads of x.
// Bound: latency of the high bits' reads (10 of 21 bits at n = 21; x is read
// that often from L2) at 32 to 40 warps per SM; DRAM moves x and y once while
// x fits L2.  Four rows per thread keep enough warps: eight rows measured 46
// against 39 us (complex128, n = 21), two rows 49.  A pass of its own for the
// top bits over strided tiles (five vector moves for any n) measured 45 us at
// n = 21 and 418 against 355 at n = 24: half-used sectors and a second
// launch cost more than the reads.  H x against a kernel with one thread per
// row: complex128 n = 21 65.6 -> 39.0 us, complex64 57.5 -> 26.7, float64 54.7
// -> 27.9, n = 23 216 -> 116; complex128 n = 24 556 -> 354; 16 float32 vectors
// n = 20 352 -> 74.
#include "el_tile.cuh"

#include <algorithm>

namespace {

using namespace el;

constexpr int FSUB = 256;      // chunks per sub-block in shared memory (= threads per CTA)

constexpr int MB = 2;          // middle bits

// CTAs of 256 threads per SM that the register budget is set for.
template <typename S, int CW>
constexpr int full_ctas(int nd) { return nd ? 3 : CW * sizeof(S) >= 16 ? 4 : 5; }

struct FullGeom {
  int n, L, nch, lognch;       // L: low bits of a tile (thread bits)
  int bits;                    // bits of the tile, L + MB
  uint64_t amps;               // bits with a nonzero amplitude
};

template <typename S, bool C, int CW, bool RA, int ND>
__global__ void __launch_bounds__(FSUB, full_ctas<S, CW>(ND))
k_full_block(const __grid_constant__ FullGeom G, const __grid_constant__ HamArgs<S> H,
             const __grid_constant__ KArgs K, int64_t ntiles) {
  typedef Chunk<S, CW> V;
  constexpr int CV = C ? CW / 2 : CW;
  constexpr int NS = 1 << MB;
  extern __shared__ __align__(16) unsigned char full_smem[];
  V *const xs = reinterpret_cast<V *>(full_smem) + threadIdx.x;
  const int L = G.L, nch = G.nch;
  const int i = (int)threadIdx.x >> G.lognch, q = (int)threadIdx.x & (nch - 1);
  const int64_t sub = (int64_t)nch << L;            // chunks from one sub-block to the next
  const V *__restrict__ xg = reinterpret_cast<const V *>(K.x);
  S dlow = S(0);
  for (int k = 0; k < L; ++k)
    if ((i >> k) & 1) dlow += H.delta[k];
  double dots[CV][ND ? ND : 1];
#pragma unroll
  for (int v = 0; v < CV; ++v)
#pragma unroll
    for (int d = 0; d < ND; ++d) dots[v][d] = 0.0;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t row = (t << G.bits) + i;
    const int64_t e = row * nch + q;
    V x[NS], h[NS];
#pragma unroll
    for (int c = 0; c < NS; ++c) x[c] = xg[e + c * sub];
#pragma unroll
    for (int c = 0; c < NS; ++c) h[c] = V{};
    __syncthreads();   // the previous tile's gathers are done
#pragma unroll
    for (int c = 0; c < NS; ++c) xs[c * FSUB] = x[c];
    __syncthreads();
#pragma unroll 2
    for (int k = G.bits; k < G.n; ++k) {
      if (!((G.amps >> k) & 1u)) continue;
      const bool set = (t >> (k - G.bits)) & 1;
      const int64_t d = (int64_t)nch << k;
      const V *__restrict__ xp = xg + (set ? e - d : e + d);
      const S are = H.up_re[k], aim = C ? (set ? H.up_im[k] : -H.up_im[k]) : S(0);
      V p[NS];
#pragma unroll
      for (int c = 0; c < NS; ++c) p[c] = xp[c * sub];
#pragma unroll
      for (int c = 0; c < NS; ++c) add_flip<S, C, CW, RA>(h[c], are, aim, p[c]);
    }
#pragma unroll 2
    for (int k = 0; k < L; ++k) {
      if (!((G.amps >> k) & 1u)) continue;
      const bool set = (i >> k) & 1;
      const int d = nch << k;
      const V *__restrict__ xp = xs + (set ? -d : d);
      const S are = H.up_re[k], aim = C ? (set ? H.up_im[k] : -H.up_im[k]) : S(0);
      V p[NS];
#pragma unroll
      for (int c = 0; c < NS; ++c) p[c] = xp[c * FSUB];
#pragma unroll
      for (int c = 0; c < NS; ++c) add_flip<S, C, CW, RA>(h[c], are, aim, p[c]);
    }
#pragma unroll
    for (int b = 0; b < MB; ++b) {
      const int k = L + b;
      if (!((G.amps >> k) & 1u)) continue;
      const S are = H.up_re[k], im = C ? H.up_im[k] : S(0);
#pragma unroll
      for (int c = 0; c < NS; ++c) add_flip<S, C, CW, RA>(h[c], are, (c >> b) & 1 ? im : -im, x[c ^ (1 << b)]);
    }
    S dt = dlow;
    for (int k = G.bits; k < G.n; ++k)
      if ((t >> (k - G.bits)) & 1) dt += H.delta[k];
#pragma unroll
    for (int c = 0; c < NS; ++c) {
      if (!K.skip_diag) {
        S dm = dt;
#pragma unroll
        for (int b = 0; b < MB; ++b)
          if ((c >> b) & 1) dm += H.delta[L + b];
        dm += H.diagV[row + ((int64_t)c << L)];
#pragma unroll
        for (int w = 0; w < CW; ++w) h[c].v[w] += dm * x[c].v[w];
      }
      finish_chunk<S, C, CW, ND>(K, e + c * sub, h[c], x[c], dots);
    }
  }
  if constexpr (ND > 0) block_dots<CV, ND>(K, nch, dots, reinterpret_cast<double *>(full_smem));
}

template <typename S, bool C, int CW, bool RA, int ND>
int launch_full_t(el_ctx *ctx, const FullGeom &G, const HamArgs<S> &H, KArgs K) {
  const int threads = G.nch << G.L;
  const int nout = (int)K.nvec * 4;
  size_t smem = (size_t)(1 << MB) * FSUB * sizeof(Chunk<S, CW>);
  if (ND) smem = std::max(smem, (size_t)std::max((threads / 32) * nout, threads) * sizeof(double));
  auto *fn = k_full_block<S, C, CW, RA, ND>;
  if (smem > 48 * 1024)
    EL_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t ntiles = (int64_t)1 << (G.n - G.bits);
  const int per_sm = full_ctas<S, CW>(ND) * (FSUB / threads);
  const int grid = (int)std::min<int64_t>(ntiles, (int64_t)sm_count(ctx) * per_sm);
  if (ND) {
    const int rc = ensure_partials(ctx, (size_t)(grid + DOT_GROUPS) * nout);
    if (rc) return rc;
    K.partials = ctx->d_partials;
  }
  fn<<<grid, threads, smem, ctx->stream>>>(G, H, K, ntiles);
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

template <typename S, bool C, int CW, bool RA>
int launch_full_r(el_ctx *ctx, const FullGeom &G, const HamArgs<S> &H, const KArgs &K) {
  if (!K.want) return launch_full_t<S, C, CW, RA, 0>(ctx, G, H, K);
  if (CW > (C ? 2 : 1) && K.want == 3 && !K.probe) return launch_full_t<S, C, CW, RA, 2>(ctx, G, H, K);
  return launch_full_t<S, C, CW, RA, 4>(ctx, G, H, K);
}

template <typename S, bool C, int CW>
int launch_full_c(el_ctx *ctx, const FullGeom &G, const HamArgs<S> &H, const KArgs &K) {
  if constexpr (C) {
    if (H.real_amp) return launch_full_r<S, C, CW, true>(ctx, G, H, K);
  }
  return launch_full_r<S, C, CW, false>(ctx, G, H, K);
}

int ilog2i(int64_t v) {
  int l = 0;
  while ((1LL << l) < v) ++l;
  return l;
}

bool full_geom(const el_ham *h, const ApplyArgs &A, FullGeom *g) {
  memset(g, 0, sizeof *g);
  const int n = h->n;
  if (h->basis->layout != EL_LAYOUT_FULL) return false;
  g->n = n;
  g->nch = chunks_per_row(A);
  if (g->nch > 32) return false;
  g->lognch = ilog2i(g->nch);
  // 256 threads per CTA, fewer where the basis has no more rows
  g->L = std::min(8 - g->lognch, n - MB);
  g->bits = g->L + MB;
  if (g->L < 0 || (g->nch << g->L) < 32) return false;
  for (int k = 0; k < n; ++k)
    if (h->om_re[k] != 0.0 || h->om_im[k] != 0.0) g->amps |= 1ULL << k;
  return true;
}

}  // namespace

namespace el {

bool full_block_ok(const el_ham *h, const ApplyArgs &A) {
  if (!h->px.empty() || h->lossy) return false;   // sigma^x channels and a real diagonal only
  if (!chunks_aligned(A)) return false;
  FullGeom G;
  return full_geom(h, A, &G);
}

int launch_full_block(el_ctx *ctx, el_ham *h, const ApplyArgs &A, const KArgs &K) {
  FullGeom G;
  if (!full_geom(h, A, &G)) return fail(ctx, EL_EINVAL, "no full-basis tile for this shape");
  const int nv = A.nvec;
  switch (A.dtype) {
    case EL_F32: {
      const HamArgs<float> H = ham_args<float>(h, h->d_diagV32);
      if (nv == 1) return launch_full_c<float, false, 1>(ctx, G, H, K);
      if (nv == 2) return launch_full_c<float, false, 2>(ctx, G, H, K);
      return launch_full_c<float, false, 4>(ctx, G, H, K);
    }
    case EL_F64: {
      const HamArgs<double> H = ham_args<double>(h, h->d_diagV64);
      if (nv == 1) return launch_full_c<double, false, 1>(ctx, G, H, K);
      return launch_full_c<double, false, 2>(ctx, G, H, K);
    }
    case EL_C64: {
      const HamArgs<float> H = ham_args<float>(h, h->d_diagV32);
      if (nv == 1) return launch_full_c<float, true, 2>(ctx, G, H, K);
      return launch_full_c<float, true, 4>(ctx, G, H, K);
    }
    case EL_C128:
      return launch_full_c<double, true, 2>(ctx, G, ham_args<double>(h, h->d_diagV64), K);
    default:
      return fail(ctx, EL_EINVAL, "unknown dtype %d", A.dtype);
  }
}

}  // namespace el
