// Fused H-apply on general blockade sectors (TABLE bases of a graph, at most
// 32 sites): one thread per row and 16-byte chunk of its vectors.
//
// A row's flips are a mask (set bits, and clear ones without a set
// neighbour; the neighbour mask and the detuning sum come from tables of the
// sums over each byte of the code), so no target has to be tested.  A flip of
// a suffix bit keeps the row's prefix group and costs one look-up in its
// suffix ranks, a flip of a prefix bit looks up the other group's offset and
// class and then the rank.  Four flips are looked up, gathered and added at a
// time: the look-ups are a chain of two or three reads from L1 or L2, and what
// bounds the kernel is how many of these chains are in flight.  5 x 6 lattice
// (454,385 rows), float64: 39 us one flip after the other with 64-bit codes,
// 28.5 us here; 16 float32 vectors 434 -> 74.
#include "el_tile.cuh"

#include <algorithm>

namespace {

using namespace el;

constexpr int TT = 256;      // threads per CTA
constexpr int TU = 4;        // flips in flight

struct TableGeom {
  int nch, lognch;
  uint32_t amps;             // bits with a nonzero amplitude
};

template <typename S, bool C, int CW, bool RA, int ND>
__global__ void __launch_bounds__(TT) k_table_block(const __grid_constant__ BasisDev B, const __grid_constant__ TableGeom G,
                                                    const __grid_constant__ HamArgs<S> H, const __grid_constant__ KArgs K) {
  typedef Chunk<S, CW> V;
  constexpr int CV = C ? CW / 2 : CW;
  extern __shared__ __align__(16) unsigned char table_smem[];   // the dot products' sums
  __shared__ S td[4][256];
  __shared__ uint32_t tn[4][256];
  __shared__ S s_re[32], s_im[32];
  const int n = B.n, L = B.L;
  for (int e = threadIdx.x; e < 1024; e += TT) {
    const int byte = e >> 8, v = e & 255;
    S d = S(0);
    uint32_t nb = 0;
    for (int q = 0; q < 8; ++q) {
      const int k = byte * 8 + q;
      if (k >= n || !((v >> q) & 1)) continue;
      d += H.delta[k];
      nb |= (uint32_t)B.adj[k];
    }
    td[byte][v] = d;
    tn[byte][v] = nb;
  }
  if (threadIdx.x < 32) {
    s_re[threadIdx.x] = H.up_re[threadIdx.x];
    s_im[threadIdx.x] = C ? H.up_im[threadIdx.x] : S(0);
  }
  __syncthreads();
  const int q = threadIdx.x & (G.nch - 1);
  const uint32_t lowmask = (1u << L) - 1u;
  const V *__restrict__ xg = reinterpret_cast<const V *>(K.x);
  double dots[CV][ND ? ND : 1];
#pragma unroll
  for (int v = 0; v < CV; ++v)
#pragma unroll
    for (int d = 0; d < ND; ++d) dots[v][d] = 0.0;
  const int rpb = TT >> G.lognch;
  for (int64_t row = (int64_t)blockIdx.x * rpb + (threadIdx.x >> G.lognch); row < B.dim; row += (int64_t)gridDim.x * rpb) {
    const uint32_t code = (uint32_t)B.codes[row];
    const uint32_t p = code >> L;
    const V x = xg[row * G.nch + q];
    S dm = K.skip_diag ? S(0) : H.diagV[row];
    const int2 own = B.pre_pack[p];
    uint32_t nb = 0;
    S dsum = S(0);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int v = (code >> (8 * b)) & 255;
      nb |= tn[b][v];
      dsum += td[b][v];
    }
    V h = V{};
    uint32_t m = G.amps & (code | ~nb);
    while (m) {
      int k[TU], tg[TU];
      bool ok[TU];
#pragma unroll
      for (int u = 0; u < TU; ++u) {
        // past the last flip: the row itself.  No branch between the reads,
        // so that the four chains overlap.
        ok[u] = m != 0;
        k[u] = ok[u] ? __ffs(m) - 1 : 0;
        const uint32_t c = ok[u] ? code ^ (1u << k[u]) : code;
        m &= m - 1;          // 0 stays 0
        const int2 pk = (k[u] < L || !ok[u]) ? own : B.pre_pack[c >> L];
        tg[u] = pk.x + B.suf_rank[((uint32_t)pk.y << L) + (c & lowmask)];
      }
      V xv[TU];
#pragma unroll
      for (int u = 0; u < TU; ++u) xv[u] = xg[(int64_t)tg[u] * G.nch + q];
#pragma unroll
      for (int u = 0; u < TU; ++u) {
        if (!ok[u]) continue;
        const S aim = C ? (((code >> k[u]) & 1u) ? s_im[k[u]] : -s_im[k[u]]) : S(0);
        add_flip<S, C, CW, RA>(h, s_re[k[u]], aim, xv[u]);
      }
    }
    if (!K.skip_diag) {
      dm += dsum;
#pragma unroll
      for (int w = 0; w < CW; ++w) h.v[w] += dm * x.v[w];
    }
    finish_chunk<S, C, CW, ND>(K, row * G.nch + q, h, x, dots);
  }
  if constexpr (ND > 0) block_dots<CV, ND>(K, G.nch, dots, reinterpret_cast<double *>(table_smem));
}

template <typename S, bool C, int CW, bool RA, int ND>
int launch_table_t(el_ctx *ctx, const BasisDev &B, const TableGeom &G, const HamArgs<S> &H, KArgs K) {
  const int nout = (int)K.nvec * 4;
  const size_t smem = ND ? (size_t)std::max((TT / 32) * nout, TT) * sizeof(double) : 0;
  auto *fn = k_table_block<S, C, CW, RA, ND>;
  if (smem > 32 * 1024)
    EL_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t blocks = (B.dim * G.nch + TT - 1) / TT;
  const int grid = (int)std::min<int64_t>(blocks, 8 * (int64_t)sm_count(ctx));
  if (ND) {
    const int rc = ensure_partials(ctx, (size_t)(grid + DOT_GROUPS) * nout);
    if (rc) return rc;
    K.partials = ctx->d_partials;
  }
  fn<<<grid, TT, smem, ctx->stream>>>(B, G, H, K);
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

template <typename S, bool C, int CW, bool RA>
int launch_table_r(el_ctx *ctx, const BasisDev &B, const TableGeom &G, const HamArgs<S> &H, const KArgs &K) {
  if (!K.want) return launch_table_t<S, C, CW, RA, 0>(ctx, B, G, H, K);
  if (CW > (C ? 2 : 1) && K.want == 3 && !K.probe) return launch_table_t<S, C, CW, RA, 2>(ctx, B, G, H, K);
  return launch_table_t<S, C, CW, RA, 4>(ctx, B, G, H, K);
}

template <typename S, bool C, int CW>
int launch_table_c(el_ctx *ctx, const BasisDev &B, const TableGeom &G, const HamArgs<S> &H, const KArgs &K) {
  if constexpr (C) {
    if (H.real_amp) return launch_table_r<S, C, CW, true>(ctx, B, G, H, K);
  }
  return launch_table_r<S, C, CW, false>(ctx, B, G, H, K);
}

}  // namespace

namespace el {

bool table_block_ok(const el_ham *h, const ApplyArgs &A) {
  const el_basis *b = h->basis;
  if (!h->px.empty() || h->lossy) return false;   // sigma^x channels and a real diagonal only
  // every flip the neighbour mask allows is in the basis: blockade sectors
  if (b->layout != EL_LAYOUT_TABLE || b->kind != EL_BASIS_BLOCKADE) return false;
  if (h->n > 32 || b->dim >= ((int64_t)1 << 31)) return false;
  return chunks_aligned(A) && chunks_per_row(A) <= 32;
}

int launch_table_block(el_ctx *ctx, el_ham *h, const ApplyArgs &A, const BasisDev &B, const KArgs &K) {
  TableGeom G;
  memset(&G, 0, sizeof G);
  G.nch = chunks_per_row(A);
  while ((1 << G.lognch) < G.nch) ++G.lognch;
  for (int k = 0; k < h->n; ++k)
    if (h->om_re[k] != 0.0 || h->om_im[k] != 0.0) G.amps |= 1u << k;
  const int nv = A.nvec;
  switch (A.dtype) {
    case EL_F32: {
      const HamArgs<float> H = ham_args<float>(h, h->d_diagV32);
      if (nv == 1) return launch_table_c<float, false, 1>(ctx, B, G, H, K);
      if (nv == 2) return launch_table_c<float, false, 2>(ctx, B, G, H, K);
      return launch_table_c<float, false, 4>(ctx, B, G, H, K);
    }
    case EL_F64: {
      const HamArgs<double> H = ham_args<double>(h, h->d_diagV64);
      if (nv == 1) return launch_table_c<double, false, 1>(ctx, B, G, H, K);
      return launch_table_c<double, false, 2>(ctx, B, G, H, K);
    }
    case EL_C64: {
      const HamArgs<float> H = ham_args<float>(h, h->d_diagV32);
      if (nv == 1) return launch_table_c<float, true, 2>(ctx, B, G, H, K);
      return launch_table_c<float, true, 4>(ctx, B, G, H, K);
    }
    case EL_C128:
      return launch_table_c<double, true, 2>(ctx, B, G, ham_args<double>(h, h->d_diagV64), K);
    default:
      return fail(ctx, EL_EINVAL, "unknown dtype %d", A.dtype);
  }
}

}  // namespace el
