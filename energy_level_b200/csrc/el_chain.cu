// Fused H-apply on nearest-neighbour chain and ring blockade sectors.
//
// A chain of n sites splits by code bit into L low, 3 middle and the
// remaining high bits.  Rows that share the bits >= L + 3 (a tile) are
// contiguous and ordered like the (L + 3)-site chain: 5 sub-blocks, one per
// middle code 000 001 010 100 101 in this order, of F(L+2) rows each (F(L+1)
// where middle bit 0 is set, because low bit L-1 is then clear); a tile whose
// high bit L + 3 is set has the first three only.  A CTA takes one tile at a
// time and a thread one low code i and one 16-byte chunk of the row (all
// vectors of a row are adjacent), for all sub-blocks at once:
//   - which low bits of i flip, and where to, is the same for every
//     sub-block and every tile: each thread works it out once per launch,
//     and per flip one address serves up to 5 shared-memory gathers;
//   - flips of middle bits are the thread's own rows;
//   - a flip of a high bit moves the whole tile by +- F(k+2) rows: coalesced
//     reads of x, up to 10 in flight, with one amplitude and one decision for
//     the tile (the flip of bit L + 3 reaches the first three sub-blocks).
// With 4 middle bits (8 sub-blocks) the same code spilled 200 to 800 bytes.
// One warp decodes the next tile's prefix and its flip list while the CTA
// works on the current tile.
//
// A ring of n sites is two chains by its top bit: codes with it clear are
// the chain of the n - 1 lower sites (rows [0, F(n+1))), codes with it set
// the chain of sites 1..n-3 (rows from F(n+1) on, bit k of that chain = code
// bit k + 1).  The top bit's flip couples them: a row of the first whose
// bits 0 and n - 2 are clear and the row of the second with the same code;
// the partner's rank is a sum over set bits (Zeckendorf, weights shifted by
// one), so it splits into a low, a middle and a tile part.
//
// Bound: latency of the L2 reads of high-flip partners (about 0.72 per high
// bit and row) against the instructions that issue them; DRAM moves the
// vectors once (complex64, one vector of the 31-site chain) or, with 8
// vectors (225 MB, more than L2), again for the top three bits.  H x on the
// 31-site chain (dim 3,524,578) against a kernel with one thread per row and
// a tile of 15 low bits: complex64 102 -> 61 us, x 4 vectors 227 -> 186, x 8
// 622 -> 358; complex128 137 -> 102, x 8 2247 -> 1000; float64 124 -> 65;
// 32 float32 vectors on 24 sites 198 -> 28; complex64 on the 28-site ring
// 42 -> 22.
#include "el_tile.cuh"

#include <algorithm>

namespace {

using namespace el;

constexpr int MID = 3;        // middle bits: one thread holds all their codes
constexpr int NSUB = 5;       // F(MID + 2) middle codes
constexpr int NSHORT = 3;     // F(MID + 1): those with the top middle bit clear
constexpr int SUB = 256;       // chunks per sub-block in shared memory, at most (= threads per CTA)
constexpr int MAXHIGH = 32;   // high bits (one lane each when a tile is decoded)

// Middle codes in ascending order, 000 001 010 100 101, and their sub-block's
// offset A F(L+2) + B F(L+1) rows into the tile.
__host__ __device__ constexpr int mid_code(int c) { return c < 3 ? c : c + 1; }
__host__ __device__ constexpr int mid_a(int c) { return c < 2 ? c : c - 1; }
__host__ __device__ constexpr int mid_b(int c) { return c < 2 ? 0 : 1; }
// sub-block whose middle code is that of c with bit b flipped, or -1
__host__ __device__ constexpr int mid_flip(int c, int b) {
  for (int d = 0; d < NSUB; ++d)
    if (mid_code(d) == (mid_code(c) ^ (1 << b))) return d;
  return -1;
}

// CTAs of 256 threads per SM that the register budget is set for.  The loads
// of a flip wait for L2, so more warps win even at a few spilled registers:
// complex64 on the 31-site chain, 8 vectors (16-byte chunks): 453 us with 2
// CTAs, 386 with 3, 358 with 4; one vector (8 bytes): 64.7 us with 4, 60.6
// with 5, 68.3 with 6.  Dot products keep 3 to 16 FP64 sums more.
template <typename S, int CW>
constexpr int chain_ctas(int nd) { return nd ? 3 : CW * sizeof(S) >= 16 ? 4 : 5; }

template <typename S>
struct TileHdr {
  int64_t base;             // first row
  int64_t ring;             // ring: tile part of the partner rank of the top bit's flip
  int nsub, nhf, seg, ring_ok;
  int edge;                 // the lowest high bit flips (it reaches the first NSHORT sub-blocks)
  S delta;                  // detunings of the set high bits
  S edge_re, edge_im;
  int64_t edge_off;
  int64_t off[MAXHIGH];     // per flip of the other high bits: rows to the partner
  S re[MAXHIGH], im[MAXHIGH];
};

struct ChainGeom {
  int L, nch, lognch;       // low bits; chunks per row
  uint64_t amps;            // code bits with a nonzero amplitude
  int nseg;                 // 1 chain, 2 ring
  int nbits[2];             // chain length of a segment (bit k of segment s is code bit k + s)
  int64_t row0[2];          // first row of a segment
  int64_t tiles[2];         // tiles of a segment
  uint64_t fib[EL_MAX_SITES + 3];
};

// The header of tile t, by one warp (every lane calls it).
template <typename S, bool C>
__device__ void decode_tile(const ChainGeom &G, const HamArgs<S> &H, int n, int64_t t, TileHdr<S> &T) {
  const int lane = threadIdx.x & 31;
  const int seg = t >= G.tiles[0] ? 1 : 0;
  int64_t r = seg ? t - G.tiles[0] : t;
  const int lo = G.L + MID, h = G.nbits[seg] - lo, sh = seg;
  uint32_t p = 0;
  for (int j = h - 1; j >= 0; --j) {
    const int64_t w = (int64_t)G.fib[j + 2];
    if (r >= w) { p |= 1u << j; r -= w; }
  }
  const bool mine = lane < h;
  const bool set = mine && ((p >> lane) & 1u);
  const int k = mine ? lo + lane : lo;          // bit in the segment's chain
  const int64_t w = (int64_t)G.fib[k + 2];
  int64_t base = set ? w : 0;
  int64_t ring = set ? (int64_t)G.fib[k + (seg ? 3 : 1)] : 0;
  S dl = set ? H.delta[k + sh] : S(0);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    base += __shfl_xor_sync(0xffffffffu, base, o);
    ring += __shfl_xor_sync(0xffffffffu, ring, o);
    dl += __shfl_xor_sync(0xffffffffu, dl, o);
  }
  const int nsub = (p & 1u) ? NSHORT : NSUB;
  const S are = mine ? H.up_re[k + sh] : S(0);
  const S aim = (C && mine) ? (set ? H.up_im[k + sh] : -H.up_im[k + sh]) : S(0);
  const uint32_t near = (p << 1) | (p >> 1);
  const bool flip = mine && (are != S(0) || aim != S(0)) && (set || !((near >> lane) & 1u));
  const unsigned all = __ballot_sync(0xffffffffu, flip && lane > 0);
  if (flip && lane > 0) {
    const int q = __popc(all & ((1u << lane) - 1u));
    T.off[q] = set ? -w : w;
    T.re[q] = are;
    T.im[q] = aim;
  }
  if (lane == 0) {
    T.base = G.row0[seg] + base;
    T.ring = ring;
    T.ring_ok = seg ? 1 : !((p >> (h - 1)) & 1u);   // ring: the last bit of the first chain is clear
    T.nsub = nsub;
    T.nhf = __popc(all);
    T.seg = seg;
    T.delta = dl;
    T.edge = flip;
    T.edge_off = set ? -w : w;
    T.edge_re = are;
    T.edge_im = aim;
  }
}

// One tile: the NS sub-blocks of the thread's low code.  Threads without a
// row in a sub-block work on the row of low code 0 instead (every address
// stays inside the tile and no inner loop tests for it) and store nothing.
template <typename S, bool C, int CW, bool RA, bool RING, int ND, int NS>
__device__ __forceinline__ void chain_tile(const ChainGeom &G, const HamArgs<S> &H, const KArgs &K, const TileHdr<S> &T,
                                           Chunk<S, CW> *xt, int n, uint32_t code, uint32_t flips, S dlow, int rlow,
                                           double (&dots)[C ? CW / 2 : CW][ND ? ND : 1]) {
  typedef Chunk<S, CW> V;
  const int L = G.L, nch = G.nch, sh = RING ? T.seg : 0;   // code bit of the segment's bit 0
  const int F1 = (int)G.fib[L + 1], F2 = (int)G.fib[L + 2];
  const int i = (int)threadIdx.x >> G.lognch, q = (int)threadIdx.x & (nch - 1);
  const bool act = i < F2, act1 = i < F1;
  const int me0 = act ? (int)threadIdx.x : q, me1 = act1 ? (int)threadIdx.x : q;
  const int s2 = F2 * nch, s1 = F1 * nch;
  const V *__restrict__ xg = reinterpret_cast<const V *>(K.x);
  // chunk index of the thread's row of a sub-block in x, and in shared
  // memory, where sub-blocks lie SUB chunks apart (a constant: one address
  // serves all sub-blocks)
  auto off = [&](int c) { return mid_a(c) * s2 + mid_b(c) * s1 + ((mid_code(c) & 1) ? me1 : me0); };
  V *const xs = xt + me0;
  const int64_t base = T.base * nch;
  {
    V x[NS];
#pragma unroll
    for (int c = 0; c < NS; ++c) x[c] = xg[base + off(c)];
#pragma unroll
    for (int c = 0; c < NS; ++c)
      if ((mid_code(c) & 1) ? act1 : act) xs[c * SUB] = x[c];
  }
  V h[NS];
#pragma unroll
  for (int c = 0; c < NS; ++c) h[c] = V{};
  __syncthreads();
  // high bits: partner tiles
  if (T.edge) {
    const V *__restrict__ xp = xg + (base + T.edge_off * nch);
    const S are = T.edge_re, aim = T.edge_im;
    V p[NSHORT];
#pragma unroll
    for (int c = 0; c < NSHORT; ++c) p[c] = xp[off(c)];
#pragma unroll
    for (int c = 0; c < NSHORT; ++c) add_flip<S, C, CW, RA>(h[c], are, aim, p[c]);
  }
#pragma unroll 2
  for (int f = 0; f < T.nhf; ++f) {
    const V *__restrict__ xp = xg + (base + T.off[f] * nch);
    const S are = T.re[f], aim = T.im[f];
    V p[NS];
#pragma unroll
    for (int c = 0; c < NS; ++c) p[c] = xp[off(c)];
#pragma unroll
    for (int c = 0; c < NS; ++c) add_flip<S, C, CW, RA>(h[c], are, aim, p[c]);
  }
  // ring: the flip of the top bit
  if (RING && T.ring_ok) {
    const int top = n - 1;
    const S are = H.up_re[top];
    const S aim = C ? (T.seg ? H.up_im[top] : -H.up_im[top]) : S(0);
    if (((G.amps >> top) & 1u) && (T.seg || !(code & 1u))) {
      const int64_t pb = (T.seg ? 0 : G.row0[1]) + T.ring + rlow;
#pragma unroll
      for (int c = 0; c < NS; ++c) {
        if (!((mid_code(c) & 1) ? act1 : act)) continue;
        int64_t pr = pb;
#pragma unroll
        for (int b = 0; b < MID; ++b)
          if ((mid_code(c) >> b) & 1) pr += (int64_t)G.fib[L + b + (T.seg ? 3 : 1)];
        add_flip<S, C, CW, RA>(h[c], are, aim, xg[pr * nch + q]);
      }
    }
  }
  // low bits: the tile in shared memory (bit L - 1 where middle bit 0 is clear)
  for (int k = 0; k < L - 1; ++k) {
    if (!((flips >> k) & 1u)) continue;
    const S are = H.up_re[k + sh];
    const S im = C ? H.up_im[k + sh] : S(0);
    const bool set = (code >> k) & 1u;
    const int w = (int)G.fib[k + 2] * nch;
    const V *__restrict__ xp = xs + (set ? -w : w);
    const S aim = set ? im : -im;
    V p[NS];
#pragma unroll
    for (int c = 0; c < NS; ++c) p[c] = xp[c * SUB];
#pragma unroll
    for (int c = 0; c < NS; ++c) add_flip<S, C, CW, RA>(h[c], are, aim, p[c]);
  }
  {
    if ((flips >> (L - 1)) & 1u) {
      const S are = H.up_re[L - 1 + sh];
      const S im = C ? H.up_im[L - 1 + sh] : S(0);
      const bool set = (code >> (L - 1)) & 1u;
      const int w = s1;
      const V *__restrict__ xp = xs + (set ? -w : w);
      const S aim = set ? im : -im;
#pragma unroll
      for (int c = 0; c < NS; ++c)
        if (!(mid_code(c) & 1)) add_flip<S, C, CW, RA>(h[c], are, aim, xp[c * SUB]);
    }
  }
  // middle bits: the thread's own rows of the other sub-blocks
  V x[NS];
#pragma unroll
  for (int c = 0; c < NS; ++c) x[c] = xs[c * SUB];
#pragma unroll
  for (int b = 0; b < MID; ++b) {
    if (!((G.amps >> (L + b + sh)) & 1u)) continue;
    const S are = H.up_re[L + b + sh];
    const S aim = C ? H.up_im[L + b + sh] : S(0);
#pragma unroll
    for (int c = 0; c < NS; ++c) {
      const int d = mid_flip(c, b);
      if (d < 0 || d >= NS) continue;
      const bool set = (mid_code(c) >> b) & 1;
      if (b > 0 || act1) add_flip<S, C, CW, RA>(h[c], are, set ? aim : -aim, x[d]);
    }
  }
  // diagonal and the caller's recurrence
  const S dt = T.delta + dlow;
#pragma unroll
  for (int c = 0; c < NS; ++c) {
    if (!((mid_code(c) & 1) ? act1 : act)) continue;
    const int64_t e = base + off(c);
    if (!K.skip_diag) {
      S dm = dt;
#pragma unroll
      for (int b = 0; b < MID; ++b)
        if ((mid_code(c) >> b) & 1) dm += H.delta[L + b + sh];
      dm += H.diagV[T.base + (mid_a(c) * F2 + mid_b(c) * F1 + i)];
#pragma unroll
      for (int w = 0; w < CW; ++w) h[c].v[w] += dm * x[c].v[w];
    }
    finish_chunk<S, C, CW, ND>(K, e, h[c], x[c], dots);
  }
}

// ND: dot products kept per vector: 0, 2 (xx, Re xy) or 4.
template <typename S, bool C, int CW, bool RA, bool RING, int ND>
__global__ void __launch_bounds__(SUB, chain_ctas<S, CW>(ND))
k_chain_block(const __grid_constant__ ChainGeom G, const __grid_constant__ HamArgs<S> H,
              const __grid_constant__ KArgs K, int n, int64_t ntiles) {
  typedef Chunk<S, CW> V;
  constexpr int CV = C ? CW / 2 : CW;     // vectors of a chunk
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *xt = reinterpret_cast<V *>(smem_raw);
  __shared__ TileHdr<S> hdr[2];
  const int L = G.L;
  const int i = (int)threadIdx.x >> G.lognch;
  // the low code, its and, per segment, its flippable bits (those of
  // the L-site chain that have an amplitude), its detuning sum and its part of the ring partner's rank
  uint32_t code = 0, flips[2] = {0, 0};
  S dlow[2] = {S(0), G.nseg == 2 ? H.delta[n - 1] : S(0)};   // the second segment has the top bit set
  int rlow[2] = {0, 0};
  if (i < (int)G.fib[L + 2]) {
    int r = i;
    for (int k = L - 1; k >= 0; --k) {
      const int w = (int)G.fib[k + 2];
      if (r >= w) { code |= 1u << k; r -= w; }
    }
    const uint32_t fl = code | (~((code << 1) | (code >> 1)) & ((1u << L) - 1u));
    flips[0] = fl & (uint32_t)G.amps;
    flips[1] = fl & (uint32_t)(G.amps >> 1);
    for (int k = 0; k < L; ++k) {
      if (!((code >> k) & 1u)) continue;
      dlow[0] += H.delta[k];
      dlow[1] += H.delta[k + 1];
      rlow[0] += (int)G.fib[k + 1];
      rlow[1] += (int)G.fib[k + 3];
    }
  }
  double dots[CV][ND ? ND : 1];
#pragma unroll
  for (int v = 0; v < CV; ++v)
#pragma unroll
    for (int d = 0; d < ND; ++d) dots[v][d] = 0.0;
  if (threadIdx.x < 32 && blockIdx.x < ntiles) decode_tile<S, C>(G, H, n, blockIdx.x, hdr[0]);
  int cur = 0;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x, cur ^= 1) {
    __syncthreads();   // header ready; the previous tile's gathers are done
    if (threadIdx.x < 32 && t + gridDim.x < ntiles) decode_tile<S, C>(G, H, n, t + gridDim.x, hdr[cur ^ 1]);
    const TileHdr<S> &T = hdr[cur];
    const int seg = RING ? T.seg : 0;
    if (T.nsub == NSUB)
      chain_tile<S, C, CW, RA, RING, ND, NSUB>(G, H, K, T, xt, n, code, flips[seg], dlow[seg], rlow[seg], dots);
    else
      chain_tile<S, C, CW, RA, RING, ND, NSHORT>(G, H, K, T, xt, n, code, flips[seg], dlow[seg], rlow[seg], dots);
  }
  if constexpr (ND > 0) block_dots<CV, ND>(K, G.nch, dots, reinterpret_cast<double *>(smem_raw));
}

// Low bits of the tile: F(L+2) x chunks threads, the most that fit SUB.  A
// larger L leaves fewer high bits, so fewer reads of partner tiles (one
// complex64 vector, n = 31: 64.7 us at L = 9, 62.2 at 10, 60.6 at 11; 512
// threads at L = 12 measured 81); smaller ones keep two tiles per SM on
// short chains.  Returns 0 where no L gives a tile.
int chain_low_bits(const ChainGeom &g, const BasisDev &B, int nch, int sms) {
  const int nmin = g.nseg == 2 ? g.nbits[1] : g.nbits[0];
  int best = 0;
  for (int L = 3; L + MID + 1 <= nmin && L <= 16; ++L) {
    const int64_t threads = (int64_t)B.fib[L + 2] * nch;
    int64_t tiles = 0;
    for (int s = 0; s < g.nseg; ++s) tiles += (int64_t)B.fib[g.nbits[s] - L - MID + 2];
    if (threads > SUB) break;
    if (best && tiles < 2 * sms) break;
    best = L;
  }
  return best;
}

bool chain_geom(const el_ctx *ctx, const el_ham *h, const ApplyArgs &A, const BasisDev &B, ChainGeom *g) {
  memset(g, 0, sizeof *g);
  const int n = h->n;
  memcpy(g->fib, B.fib, sizeof g->fib);
  if (h->basis->layout == EL_LAYOUT_CHAIN) {
    g->nseg = 1;
    g->nbits[0] = n;
  } else if (h->basis->layout == EL_LAYOUT_RING && n >= 6) {
    g->nseg = 2;
    g->nbits[0] = n - 1;
    g->nbits[1] = n - 3;
    g->row0[1] = (int64_t)B.fib[n + 1];
  } else {
    return false;
  }
  g->nch = chunks_per_row(A);
  if (g->nch > 32) return false;
  while ((1 << g->lognch) < g->nch) ++g->lognch;
  g->L = chain_low_bits(*g, B, g->nch, sm_count(ctx));
  if (!g->L) return false;
  for (int k = 0; k < n; ++k)
    if (h->om_re[k] != 0.0 || h->om_im[k] != 0.0) g->amps |= 1ULL << k;
  for (int s = 0; s < g->nseg; ++s) {
    if (g->nbits[s] - g->L - MID > MAXHIGH) return false;
    g->tiles[s] = (int64_t)B.fib[g->nbits[s] - g->L - MID + 2];
  }
  return true;
}

template <typename S, bool C, int CW, bool RA, bool RING, int ND>
int launch_block_t(el_ctx *ctx, const ChainGeom &G, const HamArgs<S> &H, KArgs K, int n) {
  const int threads = (((int)G.fib[G.L + 2] * G.nch + 31) / 32) * 32;
  size_t smem = (size_t)NSUB * SUB * sizeof(Chunk<S, CW>);
  const int nout = (int)K.nvec * 4;
  if (ND) smem = std::max(smem, (size_t)std::max((threads / 32) * nout, threads) * sizeof(double));
  auto *fn = k_chain_block<S, C, CW, RA, RING, ND>;
  if (smem > 48 * 1024)
    EL_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t ntiles = G.tiles[0] + G.tiles[1];
  const int per_sm = chain_ctas<S, CW>(ND) * (SUB / threads);
  const int grid = (int)std::min<int64_t>(ntiles, (int64_t)sm_count(ctx) * per_sm);
  if (ND) {
    const int rc = ensure_partials(ctx, (size_t)(grid + DOT_GROUPS) * nout);
    if (rc) return rc;
    K.partials = ctx->d_partials;
  }
  fn<<<grid, threads, smem, ctx->stream>>>(G, H, K, n, ntiles);
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

template <typename S, bool C, int CW, bool RA, bool RING>
int launch_block_r(el_ctx *ctx, const ChainGeom &G, const HamArgs<S> &H, const KArgs &K, int n) {
  if (!K.want) return launch_block_t<S, C, CW, RA, RING, 0>(ctx, G, H, K, n);
  if (CW > (C ? 2 : 1) && K.want == 3 && !K.probe) return launch_block_t<S, C, CW, RA, RING, 2>(ctx, G, H, K, n);
  return launch_block_t<S, C, CW, RA, RING, 4>(ctx, G, H, K, n);
}

template <typename S, bool C, int CW>
int launch_block_c(el_ctx *ctx, const ChainGeom &G, const HamArgs<S> &H, const KArgs &K, int n) {
  if constexpr (C) {
    if (H.real_amp)
      return G.nseg == 2 ? launch_block_r<S, C, CW, true, true>(ctx, G, H, K, n)
                         : launch_block_r<S, C, CW, true, false>(ctx, G, H, K, n);
  }
  return G.nseg == 2 ? launch_block_r<S, C, CW, false, true>(ctx, G, H, K, n)
                     : launch_block_r<S, C, CW, false, false>(ctx, G, H, K, n);
}

}  // namespace

namespace el {

bool chain_block_ok(const el_ctx *ctx, const el_ham *h, const ApplyArgs &A) {
  if (!h->px.empty() || h->lossy) return false;   // sigma^x channels and a real diagonal only
  if (!chunks_aligned(A)) return false;
  ChainGeom G;
  return chain_geom(ctx, h, A, basis_dev(h->basis), &G);
}

int launch_chain_block(el_ctx *ctx, el_ham *h, const ApplyArgs &A, const BasisDev &B, const KArgs &K) {
  ChainGeom G;
  if (!chain_geom(ctx, h, A, B, &G)) return fail(ctx, EL_EINVAL, "no chain tile for this shape");
  const int n = h->n, nv = A.nvec;
  switch (A.dtype) {
    case EL_F32: {
      const HamArgs<float> H = ham_args<float>(h, h->d_diagV32);
      if (nv == 1) return launch_block_c<float, false, 1>(ctx, G, H, K, n);
      if (nv == 2) return launch_block_c<float, false, 2>(ctx, G, H, K, n);
      return launch_block_c<float, false, 4>(ctx, G, H, K, n);
    }
    case EL_F64: {
      const HamArgs<double> H = ham_args<double>(h, h->d_diagV64);
      if (nv == 1) return launch_block_c<double, false, 1>(ctx, G, H, K, n);
      return launch_block_c<double, false, 2>(ctx, G, H, K, n);
    }
    case EL_C64: {
      const HamArgs<float> H = ham_args<float>(h, h->d_diagV32);
      if (nv == 1) return launch_block_c<float, true, 2>(ctx, G, H, K, n);
      return launch_block_c<float, true, 4>(ctx, G, H, K, n);
    }
    case EL_C128:
      return launch_block_c<double, true, 2>(ctx, G, ham_args<double>(h, h->d_diagV64), K, n);
    default:
      return fail(ctx, EL_EINVAL, "unknown dtype %d", A.dtype);
  }
}

}  // namespace el
