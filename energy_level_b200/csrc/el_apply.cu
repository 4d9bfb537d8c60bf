// Generic fused H-apply kernel, the row kernel of small bases and the vector
// helpers used by the drivers (large chain, ring and full bases: el_chain.cu,
// el_full.cu).
//
// Generic: one thread handles one (row, vector) element of a block [dim][nvec]; the
// nvec lanes of a row are adjacent, so every flip gather of a row block is a
// contiguous nvec-element segment.  For each row the kernel
//   - recovers the configuration code (arithmetic unranking or code table),
//   - accumulates the delta part of the diagonal bit by bit,
//   - gathers x[target] for every sigma^x flip whose target is in the basis
//     (flip targets computed arithmetically or from the class tables),
// and fuses the caller's recurrence  y = a*Hx + b*x + c*z,  acc += w*y  and
// the FP64 dot products the drivers need (moments, alpha, beta, norms).
// Channel semantics: channels.py:58-132 (diagonal delta n + V n n, sigma^x
// amplitude Omega/2 into |r>, conj(Omega)/2 into |g>).
#include "el_apply.cuh"

#include <algorithm>

namespace {

using namespace el;

// Amplitude <row|H|row ^ (bit bi | bit bj)> of exchange pair e for a row whose
// bits at bi, bj are (si, sj): J channel (channels.py:121-125) when the bits
// differ -- J into (r, g), conj(J) into (g, r) -- and A channel
// (channels.py:126-130) when they agree -- A into (r, r), conj(A) into (g, g).
__device__ __forceinline__ void exchange_amp(const ExPair &e, bool si, bool sj,
                                             double &re, double &im) {
  if (si != sj) { re = e.jre; im = si ? e.jim : -e.jim; }
  else { re = e.are; im = si ? e.aim : -e.aim; }
}

template <typename S, bool C> struct Val;
template <typename S> struct Val<S, false> {
  S v;
  __device__ static Val load(const void *p, int64_t i) { Val r; r.v = ((const S *)p)[i]; return r; }
  __device__ void store(void *p, int64_t i) const { ((S *)p)[i] = v; }
};
template <typename S> struct Val<S, true> {
  S re, im;
  __device__ static Val load(const void *p, int64_t i) {
    Val r; r.re = ((const S *)p)[2 * i]; r.im = ((const S *)p)[2 * i + 1]; return r;
  }
  __device__ void store(void *p, int64_t i) const { ((S *)p)[2 * i] = re; ((S *)p)[2 * i + 1] = im; }
};

// Block reduction of 4 doubles per thread into per-(vector, quantity) sums
// (thread t holds vector t mod nvec; nvec divides 256), then a deterministic
// cross-block sum by the last block to finish.  Lanes that hold the same
// vector meet in a butterfly of shuffles, warps through shared memory; the
// last block gives every output 256 / nout threads, each adding every
// (256 / nout)-th block in order.  Both tails are latency chains: with four
// threads adding 256 values of the block and then one per block in turn, an
// FP64 product with dots on 65,536 rows took 34.1 us of which the product is
// 9 us; this form takes 10.2 us.
__device__ void reduce4(const KArgs &K, double q0, double q1, double q2, double q3) {
  __shared__ double red[256][4];
  __shared__ bool last;
  const int tid = threadIdx.x;
  const int nv = (int)K.nvec;
  const int nout = nv * 4;
  for (int o = 16; o >= nv; o >>= 1) {
    q0 += __shfl_xor_sync(0xffffffffu, q0, o);
    q1 += __shfl_xor_sync(0xffffffffu, q1, o);
    q2 += __shfl_xor_sync(0xffffffffu, q2, o);
    q3 += __shfl_xor_sync(0xffffffffu, q3, o);
  }
  red[tid][0] = q0; red[tid][1] = q1; red[tid][2] = q2; red[tid][3] = q3;
  __syncthreads();
  const int step = nv < 32 ? 32 : nv;    // one value per warp below 32 vectors
  for (int o = tid; o < nout; o += 256) {
    const int v = o >> 2, q = o & 3;
    double s = 0.0;
    for (int j = v; j < 256; j += step) s += red[j][q];
    K.partials[(size_t)blockIdx.x * nout + o] = s;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = (atomicAdd(K.counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (nout <= 128) {
    // tid = share * nout + output: neighbours read neighbouring outputs
    const int per = 256 / nout, o = tid & (nout - 1), sh = tid / nout;
    double s = 0.0;
    for (unsigned b = sh; b < gridDim.x; b += per) s += __ldcg(&K.partials[(size_t)b * nout + o]);
    double *flat = &red[0][0];
    flat[tid] = s;
    __syncthreads();
    for (int w = per >> 1; w > 0; w >>= 1) {
      if (sh < w) flat[tid] += flat[tid + w * nout];
      __syncthreads();
    }
    if (sh == 0) K.dots[o] = flat[tid];
  } else {
    for (int o = tid; o < nout; o += 256) {
      double s = 0.0;
      for (unsigned b = 0; b < gridDim.x; ++b) s += __ldcg(&K.partials[(size_t)b * nout + o]);
      K.dots[o] = s;
    }
  }
  if (tid == 0) *K.counter = 0u;
}

template <typename S, bool C>
__global__ void __launch_bounds__(256) k_apply(BasisDev B, HamArgs<S> H, KArgs K) {
  typedef Val<S, C> V;
  const int64_t total = B.dim * K.nvec;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  double q0 = 0, q1 = 0, q2 = 0, q3 = 0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
    const int64_t row = t >> K.lognv;
    const int64_t v = t & (K.nvec - 1);
    const uint64_t code = el::unrank_row(B, row);
    const V xr = V::load(K.x, t);
    S hre = 0, him = 0, dsum = 0, dimg = 0;
    for (int k = 0; k < B.n; ++k) {
      const bool set = (code >> k) & 1ULL;
      if (set) {
        dsum += H.delta[k];
        if constexpr (C) dimg += H.loss[k];
      }
      const S are = H.up_re[k];
      const S aim = C ? (set ? H.up_im[k] : -H.up_im[k]) : S(0);
      if (are == S(0) && aim == S(0)) continue;
      const int64_t tg = el::flip_target(B, code, row, k);
      if (tg < 0) continue;
      const V xs = V::load(K.x, (tg << K.lognv) + v);
      if constexpr (C) {
        hre += are * xs.re - aim * xs.im;
        him += are * xs.im + aim * xs.re;
      } else {
        hre += are * xs.v;
      }
    }
    for (int p = 0; p < H.npx; ++p) {
      const ExPair e = H.px[p];
      double pre, pim;
      exchange_amp(e, (code >> e.bi) & 1ULL, (code >> e.bj) & 1ULL, pre, pim);
      if (pre == 0.0 && pim == 0.0) continue;
      const int64_t tg = el::rank_any(B, code ^ ((1ULL << e.bi) | (1ULL << e.bj)));
      if (tg < 0) continue;
      const V xs = V::load(K.x, (tg << K.lognv) + v);
      const S are = (S)pre, aim = (S)pim;
      if constexpr (C) {
        hre += are * xs.re - aim * xs.im;
        him += are * xs.im + aim * xs.re;
      } else {
        hre += are * xs.v;
      }
    }
    if (!K.skip_diag) {
      dsum += H.diagV[row];
      if constexpr (C) {
        hre += dsum * xr.re - dimg * xr.im;
        him += dsum * xr.im + dimg * xr.re;
      } else {
        hre += dsum * xr.v;
      }
    }
    V yv;
    if constexpr (C) {
      yv.re = (S)K.a * hre + (S)K.b * xr.re;
      yv.im = (S)K.a * him + (S)K.b * xr.im;
      if (K.z) { const V zv = V::load(K.z, t); yv.re += (S)coef_c(K) * zv.re; yv.im += (S)coef_c(K) * zv.im; }
      if (K.acc) {
        V av = V::load(K.acc, t);
        av.re += (S)K.w_re * yv.re - (S)K.w_im * yv.im;
        av.im += (S)K.w_re * yv.im + (S)K.w_im * yv.re;
        av.store(K.acc, t);
      }
    } else {
      yv.v = (S)K.a * hre + (S)K.b * xr.v;
      if (K.z) { const V zv = V::load(K.z, t); yv.v += (S)coef_c(K) * zv.v; }
      if (K.acc) { V av = V::load(K.acc, t); av.v += (S)K.w_re * yv.v; av.store(K.acc, t); }
    }
    if (K.y) yv.store(K.y, t);
    if (K.want) {
      // FP32 values are widened before multiplying: the products are exact in
      // FP64, so only the FP64 summation rounds.
      if constexpr (C) {
        const double xre = xr.re, xim = xr.im, yre = yv.re, yim = yv.im;
        q0 += xre * xre + xim * xim;
        q1 += xre * yre + xim * yim;
        q2 += xre * yim - xim * yre;
        q3 += yre * yre + yim * yim;
      } else {
        const double xd = xr.v, yd = yv.v;
        q0 += xd * xd;
        q1 += xd * yd;
        q3 += yd * yd;
        if (K.probe) q2 += yd * (double)V::load(K.probe, t).v;
      }
    }
  }
  if (K.want) reduce4(K, q0, q1, q2, q3);
}

// --------------------------------------------- hop kernel (exchange channels)
// H with exchange channels on a FULL or TABLE (fixed-excitation, general
// restricted) basis of at most 32 sites: the generic kernel's per-element
// work, but the J channels are visited as hops -- every (set bit a, clear bit
// b) pair of the row, k (n - k) of them, with the amplitude from a table in
// shared memory -- instead of testing every site pair, codes and table ranks
// are 32-bit, and only the pairs with a nonzero A are scanned.
__device__ __forceinline__ int rank32(const BasisDev &B, uint32_t c) {
  if (B.layout == EL_LAYOUT_FULL) return (int)c;
  // no branch between the reads, so that several ranks can be in flight
  // (a prefix that is not allowed has offset -1 and a class of its own reads 0)
  const int2 pk = B.pre_pack[c >> B.L];
  const int32_t rr = B.suf_rank[((uint32_t)pk.y << B.L) + (c & ((1u << B.L) - 1u))];
  return (pk.x | rr) < 0 ? -1 : pk.x + rr;
}

// Hops go four at a time (ranks, gathers, additions) with no branch between
// their reads: a rank is two dependent reads and a gather the third, and a row
// has k (n - k) of them.  16 sites, k = 8 (12,870 rows, 64 hops a row), float64:
// 30.9 us one hop after the other, 26 four at a time with the rank's early
// returns, 14.5 without; 20 sites, k = 10 (184,756 rows) 59.5 -> 51.6.  Lanes
// sharing a row (8 or 4) measured 20.6 and 16.5 at k = 8 of 16.
template <typename S, bool C>
__global__ void __launch_bounds__(256) k_apply_hop(BasisDev B, HamArgs<S> H, KArgs K, const double *hop,
                                                   const ExPair *pxA, int npxA) {
  typedef Val<S, C> V;
  extern __shared__ __align__(16) unsigned char hop_smem[];
  const int n = B.n;
  S *hre_t = reinterpret_cast<S *>(hop_smem);
  S *him_t = hre_t + n * n;
  // per-bit constants by the row's own bits: shared memory (a constant read
  // with a different index in every lane is one read per index)
  __shared__ S s_de[32], s_lo[32], s_re[32], s_im[32];
  if (threadIdx.x < 32) {
    s_de[threadIdx.x] = H.delta[threadIdx.x];
    s_lo[threadIdx.x] = H.loss[threadIdx.x];
    s_re[threadIdx.x] = H.up_re[threadIdx.x];
    s_im[threadIdx.x] = H.up_im[threadIdx.x];
  }
  for (int i = threadIdx.x; i < n * n; i += blockDim.x) {
    hre_t[i] = (S)hop[i];
    if constexpr (C) him_t[i] = (S)hop[n * n + i];
  }
  __syncthreads();
  const uint32_t full = (n >= 32) ? 0xffffffffu : ((1u << n) - 1u);
  const int64_t total = B.dim * K.nvec;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  double q0 = 0, q1 = 0, q2 = 0, q3 = 0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
    const int64_t row = t >> K.lognv;
    const int64_t v = t & (K.nvec - 1);
    const uint32_t code = (B.layout == EL_LAYOUT_FULL) ? (uint32_t)row : (uint32_t)B.codes[row];
    const V xr = V::load(K.x, t);
    S hre = 0, him = 0, dsum = 0, dimg = 0;
    for (uint32_t m = code; m; m &= m - 1) {
      const int k = __ffs(m) - 1;
      dsum += s_de[k];
      if constexpr (C) dimg += s_lo[k];
    }
    // sigma^x channels (bits with a nonzero Omega)
    for (int k = 0; k < n; ++k) {
      const bool set = (code >> k) & 1u;
      const S are = s_re[k];
      const S aim = C ? (set ? s_im[k] : -s_im[k]) : S(0);
      if (are == S(0) && aim == S(0)) continue;
      const int tg = rank32(B, code ^ (1u << k));
      if (tg < 0) continue;
      const V xs = V::load(K.x, ((int64_t)tg << K.lognv) + v);
      if constexpr (C) { hre += are * xs.re - aim * xs.im; him += are * xs.im + aim * xs.re; }
      else { hre += are * xs.v; }
    }
    // J channels: move one excitation from a set bit a to a clear bit b
    for (uint32_t ma = code; ma; ma &= ma - 1) {
      const int o = __ffs(ma) - 1;
      const S *const hr = hre_t + o * n;
      const S *const hi = him_t + o * n;
      uint32_t mi = ~code & full;
      while (mi) {
        constexpr int U = 4;
        int tg[U];
        S are[U], aim[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          // past the last bit: the row itself, with no amplitude
          const bool on = mi != 0;
          const int i = on ? __ffs(mi) - 1 : o;
          mi &= mi - 1;
          are[u] = on ? hr[i] : S(0);
          aim[u] = (C && on) ? hi[i] : S(0);
          tg[u] = rank32(B, on ? code ^ (1u << o) ^ (1u << i) : code);
        }
        V xs[U];
#pragma unroll
        for (int u = 0; u < U; ++u) xs[u] = V::load(K.x, ((int64_t)max(tg[u], 0) << K.lognv) + v);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (tg[u] < 0 || (are[u] == S(0) && aim[u] == S(0))) continue;
          if constexpr (C) { hre += are[u] * xs[u].re - aim[u] * xs[u].im; him += are[u] * xs[u].im + aim[u] * xs[u].re; }
          else { hre += are[u] * xs[u].v; }
        }
      }
    }
    // A channels: create or remove both excitations
    for (int p = 0; p < npxA; ++p) {
      const ExPair e = pxA[p];
      const bool si = (code >> e.bi) & 1u, sj = (code >> e.bj) & 1u;
      if (si != sj) continue;
      const S are = (S)e.are;
      const S aim = C ? (S)(si ? e.aim : -e.aim) : S(0);
      const int tg = rank32(B, code ^ (1u << e.bi) ^ (1u << e.bj));
      if (tg < 0) continue;
      const V xs = V::load(K.x, ((int64_t)tg << K.lognv) + v);
      if constexpr (C) { hre += are * xs.re - aim * xs.im; him += are * xs.im + aim * xs.re; }
      else { hre += are * xs.v; }
    }
    if (!K.skip_diag) {
      dsum += H.diagV[row];
      if constexpr (C) {
        hre += dsum * xr.re - dimg * xr.im;
        him += dsum * xr.im + dimg * xr.re;
      } else {
        hre += dsum * xr.v;
      }
    }
    V yv;
    if constexpr (C) {
      yv.re = (S)K.a * hre + (S)K.b * xr.re;
      yv.im = (S)K.a * him + (S)K.b * xr.im;
      if (K.z) { const V zv = V::load(K.z, t); yv.re += (S)coef_c(K) * zv.re; yv.im += (S)coef_c(K) * zv.im; }
      if (K.acc) {
        V av = V::load(K.acc, t);
        av.re += (S)K.w_re * yv.re - (S)K.w_im * yv.im;
        av.im += (S)K.w_re * yv.im + (S)K.w_im * yv.re;
        av.store(K.acc, t);
      }
    } else {
      yv.v = (S)K.a * hre + (S)K.b * xr.v;
      if (K.z) { const V zv = V::load(K.z, t); yv.v += (S)coef_c(K) * zv.v; }
      if (K.acc) { V av = V::load(K.acc, t); av.v += (S)K.w_re * yv.v; av.store(K.acc, t); }
    }
    if (K.y) yv.store(K.y, t);
    if (K.want) {
      if constexpr (C) {
        const double xre = xr.re, xim = xr.im, yre = yv.re, yim = yv.im;
        q0 += xre * xre + xim * xim;
        q1 += xre * yre + xim * yim;
        q2 += xre * yim - xim * yre;
        q3 += yre * yre + yim * yim;
      } else {
        const double xd = xr.v, yd = yv.v;
        q0 += xd * xd;
        q1 += xd * yd;
        q3 += yd * yd;
        if (K.probe) q2 += yd * (double)V::load(K.probe, t).v;
      }
    }
  }
  if (K.want) reduce4(K, q0, q1, q2, q3);
}

// ------------------------------------------------- row kernel (FULL/CHAIN/RING)
// One vector on a small basis: G adjacent lanes of a warp share one row and
// take the bits k = lane, lane + G, ...; eight bits per round (a lane issues
// their gathers before it adds any of them), codes, ranks and targets in 32
// bits.  The lanes' flip sums and detunings meet in a butterfly of shuffles
// and the row's first lane runs the epilogue.  The row loop is uniform over
// the block so that every lane reaches the shuffles; lanes past the last row
// work on row 0 and store nothing.

// A row's value in one access: W = 2 for a complex one (aligned to both parts).
template <typename S, int W>
struct alignas(W * sizeof(S)) RowValue { S s[W]; };
template <typename S, int W>
__device__ __forceinline__ void ld_row(const S *p, S (&v)[W]) {
  const RowValue<S, W> t = *reinterpret_cast<const RowValue<S, W> *>(p);
#pragma unroll
  for (int i = 0; i < W; ++i) v[i] = t.s[i];
}
template <typename S, int W>
__device__ __forceinline__ void st_row(S *p, const S (&v)[W]) {
  RowValue<S, W> t;
#pragma unroll
  for (int i = 0; i < W; ++i) t.s[i] = v[i];
  *reinterpret_cast<RowValue<S, W> *>(p) = t;
}

// Code of `row` (FULL / CHAIN / RING) in CT arithmetic.
template <int LAY, typename CT, typename RT>
__device__ __forceinline__ CT unrank_fib(const BasisDev &B, RT row) {
  if constexpr (LAY == EL_LAYOUT_FULL) {
    return (CT)row;
  } else {
    const int n = B.n;
    RT r = row;
    CT c = 0;
    if constexpr (LAY == EL_LAYOUT_CHAIN) {
      for (int k = n - 1; k >= 0; --k) {
        const RT w = (RT)B.fib[k + 2];
        if (r >= w) { c |= (CT)1 << k; r -= w; }
      }
      return c;
    } else {
      const RT split = (RT)B.fib[n + 1];
      if (r < split) {
        for (int k = n - 2; k >= 0; --k) {
          const RT w = (RT)B.fib[k + 2];
          if (r >= w) { c |= (CT)1 << k; r -= w; }
        }
        return c;
      }
      r -= split;
      c = (CT)1 << (n - 1);
      for (int k = n - 3; k >= 1; --k) {
        const RT w = (RT)B.fib[k + 1];
        if (r >= w) { c |= (CT)1 << k; r -= w; }
      }
      return c;
    }
  }
}

// Rank of an allowed ring code.
template <typename CT, typename RT>
__device__ __forceinline__ RT ring_rank_t(const BasisDev &B, CT c, int n) {
  RT r = 0;
  if ((c >> (n - 1)) & 1) {
    r = (RT)B.fib[n + 1];
    for (int k = 0; k < n - 1; ++k)
      if ((c >> k) & 1) r += (RT)B.fib[k + 1];
  } else {
    for (int k = 0; k < n; ++k)
      if ((c >> k) & 1) r += (RT)B.fib[k + 2];
  }
  return r;
}

template <typename S, bool C, int LAY, bool WANT, int G>
__global__ void __launch_bounds__(256) k_apply_row(BasisDev B, HamArgs<S> H, KArgs K) {
  static_assert(32 % G == 0, "lanes per row: G divides 32");
  typedef uint32_t CT;
  typedef int32_t RT;
  constexpr int W = C ? 2 : 1;
  constexpr int U = 8;   // one round covers 8 G sites
  const int n = B.n;
  const CT full = (n >= (int)(8 * sizeof(CT))) ? ~(CT)0 : (((CT)1 << n) - 1);
  const S *__restrict__ xp = (const S *)K.x;
  double q0 = 0, q1 = 0, q2 = 0, q3 = 0;
  const RT dim = (RT)B.dim;
  const int lane = (int)threadIdx.x & (G - 1);
  const RT rpb = (RT)(blockDim.x / G);
  const RT stride = (RT)gridDim.x * rpb;
  for (RT base = (RT)blockIdx.x * rpb; base < dim; base += stride) {
    const RT mine = base + (RT)(threadIdx.x / G);
    const bool active = mine < dim;       // the same for the G lanes of a row
    const RT row = active ? mine : (RT)0;
    const CT code = unrank_fib<LAY, CT, RT>(B, row);
    CT allowed = full;
    if constexpr (LAY != EL_LAYOUT_FULL) {
      CT occ = (code << 1) | (code >> 1);
      if constexpr (LAY == EL_LAYOUT_RING) occ |= ((code >> (n - 1)) & 1) | ((code & 1) << (n - 1));
      allowed = code | (~occ & full);
    }
    const bool top = (LAY == EL_LAYOUT_RING) && ((code >> (n - 1)) & 1);
    S h[W];
#pragma unroll
    for (int i = 0; i < W; ++i) h[i] = S(0);
    S dsum = S(0);
    for (int j0 = 0; j0 * G < n; j0 += U) {
      S xv[U][W];
      S ar[U], ai[U];
      bool ok[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = (j0 + u) * G + lane;
        ok[u] = false;
        ar[u] = S(0);
        ai[u] = S(0);
        if (k < n) {
          const bool set = (code >> k) & 1;
          if (set) dsum += H.delta[k];
          ar[u] = H.up_re[k];
          if constexpr (C) ai[u] = set ? H.up_im[k] : -H.up_im[k];
          ok[u] = ((allowed >> k) & 1) && (ar[u] != S(0) || ai[u] != S(0));
          if (ok[u]) {
            RT tg;
            if constexpr (LAY == EL_LAYOUT_FULL) {
              tg = row ^ ((RT)1 << k);
            } else if constexpr (LAY == EL_LAYOUT_CHAIN) {
              const RT w = (RT)B.fib[k + 2];
              tg = set ? row - w : row + w;
            } else {
              if (k == n - 1) {
                tg = ring_rank_t<CT, RT>(B, code ^ ((CT)1 << k), n);
              } else {
                const RT w = (RT)(top ? B.fib[k + 1] : B.fib[k + 2]);
                tg = set ? row - w : row + w;
              }
            }
            ld_row<S, W>(xp + (size_t)tg * W, xv[u]);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!ok[u]) continue;
        if constexpr (C) {
          if (H.real_amp) {   // uniform: a real drive needs two FMAs per complex entry
            h[0] += ar[u] * xv[u][0];
            h[1] += ar[u] * xv[u][1];
          } else {
            h[0] += ar[u] * xv[u][0] - ai[u] * xv[u][1];
            h[1] += ar[u] * xv[u][1] + ai[u] * xv[u][0];
          }
        } else {
          h[0] += ar[u] * xv[u][0];
        }
      }
    }
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) {
#pragma unroll
      for (int i = 0; i < W; ++i) h[i] += __shfl_xor_sync(0xffffffffu, h[i], off);
      dsum += __shfl_xor_sync(0xffffffffu, dsum, off);
    }
    if (lane != 0 || !active) continue;
    S xr[W];
    ld_row<S, W>(xp + (size_t)row * W, xr);
    if (!K.skip_diag) {
      dsum += H.diagV[row];
#pragma unroll
      for (int i = 0; i < W; ++i) h[i] += dsum * xr[i];
    }
    S yv[W];
    const S a = (S)K.a, b = (S)K.b;
#pragma unroll
    for (int i = 0; i < W; ++i) yv[i] = a * h[i] + b * xr[i];
    if (K.z) {
      S zv[W];
      ld_row<S, W>((const S *)K.z + (size_t)row * W, zv);
      const S c = (S)coef_c(K);
#pragma unroll
      for (int i = 0; i < W; ++i) yv[i] += c * zv[i];
    }
    if (K.acc) {
      S av[W];
      S *ap = (S *)K.acc + (size_t)row * W;
      ld_row<S, W>(ap, av);
      const S wr = (S)K.w_re, wi = (S)K.w_im;
      if constexpr (C) {
        av[0] += wr * yv[0] - wi * yv[1];
        av[1] += wr * yv[1] + wi * yv[0];
      } else {
        av[0] += wr * yv[0];
      }
      st_row<S, W>(ap, av);
    }
    if (K.y) st_row<S, W>((S *)K.y + (size_t)row * W, yv);
    if constexpr (WANT) {
      if constexpr (C) {
        const double xre = xr[0], xim = xr[1], yre = yv[0], yim = yv[1];
        q0 += xre * xre + xim * xim;
        q1 += xre * yre + xim * yim;
        q2 += xre * yim - xim * yre;
        q3 += yre * yre + yim * yim;
      } else {
        const double xd = xr[0], yd = yv[0];
        q0 += xd * xd;
        q1 += xd * yd;
        q3 += yd * yd;
        if (K.probe) q2 += yd * (double)((const S *)K.probe)[row];
      }
    }
  }
  if constexpr (WANT) reduce4(K, q0, q1, q2, q3);
}

int ilog2(int64_t v) {
  int l = 0;
  while ((1LL << l) < v) ++l;
  return l;
}

// ---------------------------------------------------------------- diagonal

__global__ void k_diag_v(BasisDev B, int n, const double *__restrict__ Vg,
                         double *out64, float *out32) {
  extern __shared__ double Vs[];
  for (int i = threadIdx.x; i < n * n; i += blockDim.x) Vs[i] = Vg[i];
  __syncthreads();
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < B.dim;
       r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t code = el::unrank_row(B, r);
    double s = 0.0;
    uint64_t m = code;
    while (m) {
      const int k = __ffsll((long long)m) - 1;
      m &= m - 1;
      uint64_t m2 = m;
      while (m2) {
        const int k2 = __ffsll((long long)m2) - 1;
        m2 &= m2 - 1;
        s += Vs[k * n + k2];
      }
    }
    if (out64) out64[r] = s;
    if (out32) out32[r] = (float)s;
  }
}

template <typename S>
__global__ void k_full_diag(BasisDev B, HamArgs<double> H, S *out) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < B.dim;
       r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t code = el::unrank_row(B, r);
    double d = H.diagV[r];
    for (int k = 0; k < B.n; ++k) if ((code >> k) & 1ULL) d += H.delta[k];
    out[r] = (S)d;
  }
}

// Minimum, maximum, maximum over the launch (256 threads per block): warps
// by shuffles, blocks by the last one to finish with all its threads.
__device__ void gersh_tail(double lo, double hi, double nm, double *partials, unsigned int *counter, double *out) {
  __shared__ double red[8][3];
  __shared__ bool last;
  auto block = [&]() {          // totals in thread 0
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      nm = fmax(nm, __shfl_xor_sync(0xffffffffu, nm, o));
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
      red[threadIdx.x >> 5][0] = lo; red[threadIdx.x >> 5][1] = hi; red[threadIdx.x >> 5][2] = nm;
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 1; w < 8; ++w) { lo = fmin(lo, red[w][0]); hi = fmax(hi, red[w][1]); nm = fmax(nm, red[w][2]); }
  };
  block();
  if (threadIdx.x == 0) {
    partials[3 * blockIdx.x] = lo;
    partials[3 * blockIdx.x + 1] = hi;
    partials[3 * blockIdx.x + 2] = nm;
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  lo = 1e300; hi = -1e300; nm = 0.0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += 256) {
    lo = fmin(lo, __ldcg(&partials[3 * i]));
    hi = fmax(hi, __ldcg(&partials[3 * i + 1]));
    nm = fmax(nm, __ldcg(&partials[3 * i + 2]));
  }
  block();
  if (threadIdx.x == 0) {
    out[0] = lo;
    out[1] = hi;
    out[2] = nm;
    *counter = 0u;
  }
}

// Gershgorin interval: min_r (d_r - R_r), max_r (d_r + R_r).
__global__ void __launch_bounds__(256) k_gershgorin(BasisDev B, HamArgs<double> H, double *partials,
                             unsigned int *counter, double *out) {
  double lo = 1e300, hi = -1e300, nm = 0.0;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < B.dim;
       r += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t code = el::unrank_row(B, r);
    double d = H.diagV[r], R = 0.0, di = 0.0;
    for (int k = 0; k < B.n; ++k) {
      if ((code >> k) & 1ULL) { d += H.delta[k]; di += H.loss[k]; }
      const double amp = sqrt(H.up_re[k] * H.up_re[k] + H.up_im[k] * H.up_im[k]);
      if (amp == 0.0) continue;
      if (el::flip_target(B, code, r, k) >= 0) R += amp;
    }
    for (int p = 0; p < H.npx; ++p) {
      const ExPair e = H.px[p];
      double pre, pim;
      exchange_amp(e, (code >> e.bi) & 1ULL, (code >> e.bj) & 1ULL, pre, pim);
      if (pre == 0.0 && pim == 0.0) continue;
      if (el::rank_any(B, code ^ ((1ULL << e.bi) | (1ULL << e.bj))) >= 0) R += sqrt(pre * pre + pim * pim);
    }
    lo = fmin(lo, d - R);
    hi = fmax(hi, d + R);
    nm = fmax(nm, sqrt(d * d + di * di) + R);
  }
  gersh_tail(lo, hi, nm, partials, counter, out);
}

// The same for sigma^x channels on bases of at most 32 sites: a row's flips
// are a mask (set bits, and clear ones without a set neighbour), and sums
// over a mask come from tables of the sums over each byte of it: 8 to 12
// shared-memory reads per row instead of a target, a square root and two
// additions per bit.  31-site chain: 521 -> 72 us.
template <int LAY>
__global__ void __launch_bounds__(256) k_gersh_masks(BasisDev B, HamArgs<double> H, int charge, double *partials,
                                                     unsigned int *counter, double *out) {
  __shared__ double td[4][256], tr[4][256], tl[4][256];
  __shared__ uint32_t tn[4][256];
  const int n = B.n;
  for (int e = threadIdx.x; e < 1024; e += 256) {
    const int byte = e >> 8, v = e & 255;
    double d = 0.0, r = 0.0, l = 0.0;
    uint32_t nb = 0;
    for (int q = 0; q < 8; ++q) {
      const int k = byte * 8 + q;
      if (k >= n || !((v >> q) & 1)) continue;
      d += H.delta[k];
      l += H.loss[k];
      r += sqrt(H.up_re[k] * H.up_re[k] + H.up_im[k] * H.up_im[k]);
      nb |= (uint32_t)B.adj[k];
    }
    td[byte][v] = d; tr[byte][v] = r; tl[byte][v] = l; tn[byte][v] = nb;
  }
  __syncthreads();
  const uint32_t full = n >= 32 ? 0xffffffffu : (1u << n) - 1u;
  double lo = 1e300, hi = -1e300, nm = 0.0;
  for (int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x; r < B.dim; r += (int64_t)gridDim.x * 256) {
    uint32_t code;
    if constexpr (LAY == EL_LAYOUT_TABLE) code = (uint32_t)B.codes[r];
    else code = unrank_fib<LAY, uint32_t, uint32_t>(B, (uint32_t)r);
    double d = H.diagV[r], R = 0.0, di = 0.0;
    uint32_t nb = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int v = (code >> (8 * b)) & 255;
      d += td[b][v];
      if (LAY != EL_LAYOUT_FULL) nb |= tn[b][v];
      if (H.lossy) di += tl[b][v];
    }
    // a set bit's own neighbours are clear, so nb never covers a set bit
    const uint32_t flips = charge ? 0u : (full & ~nb);
#pragma unroll
    for (int b = 0; b < 4; ++b) R += tr[b][(flips >> (8 * b)) & 255];
    lo = fmin(lo, d - R);
    hi = fmax(hi, d + R);
    nm = fmax(nm, (H.lossy ? sqrt(d * d + di * di) : fabs(d)) + R);
  }
  gersh_tail(lo, hi, nm, partials, counter, out);
}

// ------------------------------------------------------------ BLAS-like ops

// Scalars of launch_lanczos_update (dots null: a plain axpby).
struct LanczosScalars {
  const double *dots, *k2;
  double *rec;
};

// y = alpha x + beta y in FP64 arithmetic and, if asked, |y|^2.  HBM-bound on
// long vectors: 16-byte accesses (ALN: both pointers on 16-byte boundaries)
// move 2^25 FP64 values of x, y and the result at 6.1 TB/s (4.0 with 8-byte
// ones); on short vectors the norm's tail counts, so warps meet by shuffles
// and the last block adds the block sums with all its threads.
template <typename S, bool C, bool ALN>
__global__ void __launch_bounds__(256) k_axpby(int64_t len, double a_re, double a_im, const S *x,
                        double b_re, double b_im, S *y, double *partials,
                        unsigned int *counter, double *norm2, LanczosScalars U) {
  __shared__ double red[8];
  __shared__ bool last;
  constexpr int E = ALN ? 16 / (int)sizeof(S) : (C ? 2 : 1);   // values per step
  struct alignas(ALN ? 16 : sizeof(S)) Chunk { S v[E]; };
  double acc = 0.0, alpha = 0.0, bpred = 1.0, k2 = 1.0;
  if (U.dots) {
    k2 = U.k2 ? *U.k2 : 1.0;
    alpha = U.dots[1] / k2;
    double sc = 1.0;
    if (U.k2) {
      // |w - alpha v|^2 from <y, y>; where that cancels, the norm is formed directly
      const double bp2 = U.dots[3] / k2 - alpha * alpha, s1 = fmax(1.0, fabs(alpha));
      bpred = bp2 > 1e-6 * s1 * s1 ? sqrt(bp2) : 1.0;
      sc = 1.0 / (sqrt(k2) * bpred);
    }
    a_re = -alpha * sc;
    b_re = sc;
  }
  const int64_t values = C ? 2 * len : len;
  // beta == 0 must not read y: workspace may hold stale bits (NaN)
  const bool ry = (b_re != 0.0 || b_im != 0.0);
  auto combine = [&](const S *xv, S *yv, int cnt) {
    if constexpr (C) {
#pragma unroll
      for (int i = 0; i < E; i += 2) {
        if (i >= cnt) break;
        const double xr = xv[i], xi = xv[i + 1], yr = yv[i], yi = yv[i + 1];
        const S rs = (S)(a_re * xr - a_im * xi + b_re * yr - b_im * yi);
        const S is = (S)(a_re * xi + a_im * xr + b_re * yi + b_im * yr);
        yv[i] = rs;
        yv[i + 1] = is;
        acc += (double)rs * (double)rs + (double)is * (double)is;
      }
    } else {
#pragma unroll
      for (int i = 0; i < E; ++i) {
        if (i >= cnt) break;
        const S r = (S)(a_re * (double)xv[i] + b_re * (double)yv[i]);
        yv[i] = r;
        acc += (double)r * (double)r;
      }
    }
  };
  const int64_t chunks = values / E;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < chunks; c += stride) {
    Chunk xc{}, yc{};
    if (x) xc = reinterpret_cast<const Chunk *>(x)[c];
    if (ry) yc = reinterpret_cast<const Chunk *>(y)[c];
    combine(xc.v, yc.v, E);
    reinterpret_cast<Chunk *>(y)[c] = yc;
  }
  const int tail = (int)(values - chunks * E);   // fewer than E values after the last chunk
  if (tail > 0 && blockIdx.x == 0 && threadIdx.x == 0) {
    Chunk xc{}, yc{};
    for (int i = 0; i < tail; ++i) {
      if (x) xc.v[i] = x[chunks * E + i];
      if (ry) yc.v[i] = y[chunks * E + i];
    }
    combine(xc.v, yc.v, tail);
    for (int i = 0; i < tail; ++i) y[chunks * E + i] = yc.v[i];
  }
  if (!norm2 && !U.dots) return;
  auto block_total = [&](double v) -> double {   // in thread 0
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
      for (int w = 0; w < 8; ++w) s += red[w];
    return s;
  };
  const double mine = block_total(acc);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = mine;
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double part = 0.0;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += 256) part += __ldcg(&partials[i]);
  const double all = block_total(part);
  if (threadIdx.x == 0) {
    if (U.dots) {
      U.rec[0] = alpha;
      U.rec[1] = all;
      U.rec[2] = -sqrt(all) * bpred * sqrt(all) / sqrt(k2);
      if (!U.k2) U.rec[2] = -sqrt(all);
      U.rec[3] = bpred;
    } else {
      *norm2 = all;
    }
    *counter = 0u;
  }
}

// partials[bx][j] (re, im) of <V_j, w> over the block's rows.
constexpr int GJ = 16;
// dots_j = <V_j, w> for a group of GJ columns per blockIdx.y (200 FP64 columns
// of 65,536 rows, L2-resident: 55 us with 8-byte loads, 14.3 with 16-byte
// ones): every thread accumulates its rows in FP64 registers, warps reduce by shuffles (fixed
// tree), then the block's warps in order; per-block partials are summed by
// k_sum_partials in block order (deterministic).
template <typename S, bool C, bool ALN>
__global__ void __launch_bounds__(256, 2) k_gemv_t(int64_t len, int k, const S *V, int64_t ld, const S *w,
                                                double *partials) {
  __shared__ double red[8][2 * GJ];
  const int j0 = blockIdx.y * GJ;
  const int nq = min(GJ, k - j0);
  double accr[GJ], acci[GJ];
#pragma unroll
  for (int q = 0; q < GJ; ++q) { accr[q] = 0.0; acci[q] = 0.0; }
  // E values per step: one 16-byte piece where every column starts on such a
  // boundary (ALN), else one (complex) value
  constexpr int E = ALN ? 16 / (int)sizeof(S) : (C ? 2 : 1);
  struct alignas(ALN ? 16 : sizeof(S)) Chunk { S v[E]; };
  const int64_t values = C ? 2 * len : len, cols = C ? 2 * ld : ld;
  const int64_t chunks = values / E;
  const S *const V0 = V + (size_t)j0 * cols;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < chunks; i += (int64_t)gridDim.x * blockDim.x) {
    const Chunk wc = reinterpret_cast<const Chunk *>(w)[i];
    Chunk vc[GJ];
#pragma unroll
    for (int q = 0; q < GJ; ++q)
      if (q < nq) vc[q] = reinterpret_cast<const Chunk *>(V0 + (size_t)q * cols)[i];
#pragma unroll
    for (int q = 0; q < GJ; ++q) {
      if (q >= nq) continue;
      if constexpr (C) {
#pragma unroll
        for (int e = 0; e < E; e += 2) {
          const double wr = wc.v[e], wi = wc.v[e + 1], vr = vc[q].v[e], vi = vc[q].v[e + 1];
          accr[q] += vr * wr + vi * wi;
          acci[q] += vr * wi - vi * wr;
        }
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e) accr[q] += (double)vc[q].v[e] * (double)wc.v[e];
      }
    }
  }
  // values after the last piece (columns of a 16-byte pitch have fewer than E)
  const int64_t tail0 = chunks * E;
  if (tail0 < values && blockIdx.x == 0 && threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < GJ; ++q) {
      if (q >= nq) continue;
      const S *const vj = V0 + (size_t)q * cols;
      for (int64_t t = tail0; t < values; t += C ? 2 : 1) {
        if constexpr (C) {
          const double wr = w[t], wi = w[t + 1], vr = vj[t], vi = vj[t + 1];
          accr[q] += vr * wr + vi * wi;
          acci[q] += vr * wi - vi * wr;
        } else {
          accr[q] += (double)vj[t] * (double)w[t];
        }
      }
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < GJ; ++q) {
    double a = accr[q], b = acci[q];
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      if (C) b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) { red[warp][2 * q] = a; red[warp][2 * q + 1] = b; }
  }
  __syncthreads();
  if (threadIdx.x < 2 * GJ) {
    const int q = threadIdx.x >> 1;
    double sum = 0.0;
    for (int wp = 0; wp < (int)(blockDim.x >> 5); ++wp) sum += red[wp][threadIdx.x];
    if (q < nq) partials[((size_t)blockIdx.x * k + j0 + q) * 2 + (threadIdx.x & 1)] = sum;
  }
}

// out[o] = sum over blocks, 32 outputs per block with 8 threads each (fixed order).
__global__ void __launch_bounds__(256) k_sum_partials(int nparts, int k, const double *partials, double *out) {
  __shared__ double red[8][32];
  const int o = blockIdx.x * 32 + (threadIdx.x & 31), sh = threadIdx.x >> 5;
  double s = 0.0;
  if (o < 2 * k) {
#pragma unroll 4
    for (int b = sh; b < nparts; b += 8) s += partials[(size_t)b * 2 * k + o];
  }
  red[sh][threadIdx.x & 31] = s;
  __syncthreads();
  if (sh == 0 && o < 2 * k) {
    for (int w = 1; w < 8; ++w) s += red[w][threadIdx.x];
    out[o] = s;
  }
}

// w -= sum_j coef_j V_j  (sub = true) or w = sum_j coef_j V_j (sub = false).
// The coefficients are staged in shared memory (k <= GN_MAX, else read from
// global memory); eight columns are read at a time and added to four partial sums.
// Each thread has one 16-byte piece of w (ALN: every column starts on such a
// boundary), else one value.
constexpr int GN_MAX = 1024;
template <typename S, bool C, bool ALN>
__global__ void __launch_bounds__(256) k_gemv_n(int64_t len, int k, const S *V, int64_t ld,
                                                const double *coef, S *w, bool sub) {
  __shared__ double cs[2 * GN_MAX];
  const bool staged = k <= GN_MAX;
  if (staged)
    for (int t = threadIdx.x; t < 2 * k; t += blockDim.x) cs[t] = coef[t];
  __syncthreads();
  const double *cf = staged ? cs : coef;
  constexpr int E = ALN ? 16 / (int)sizeof(S) : (C ? 2 : 1);
  struct alignas(ALN ? 16 : sizeof(S)) Chunk { S v[E]; };
  const int64_t values = C ? 2 * len : len, cols = C ? 2 * ld : ld;
  // the piece at value index at, of cnt values
  auto piece = [&](int64_t at, int cnt, auto load, auto store) {
    double s[4][E];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int e = 0; e < E; ++e) s[u][e] = 0.0;
    auto add = [&](const Chunk &v, int j, double (&t)[E]) {
      const double cr = cf[2 * j], ci = cf[2 * j + 1];
      if constexpr (C) {
#pragma unroll
        for (int e = 0; e < E; e += 2) {
          t[e] += cr * (double)v.v[e] - ci * (double)v.v[e + 1];
          t[e + 1] += cr * (double)v.v[e + 1] + ci * (double)v.v[e];
        }
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e) t[e] += cr * (double)v.v[e];
      }
    };
    int j = 0;
    for (; j + 8 <= k; j += 8) {
      Chunk v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = load(V + (size_t)(j + u) * cols + at, cnt);
#pragma unroll
      for (int u = 0; u < 8; ++u) add(v[u], j + u, s[u & 3]);
    }
    for (; j + 4 <= k; j += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) add(load(V + (size_t)(j + u) * cols + at, cnt), j + u, s[u]);
    }
    for (; j < k; ++j) add(load(V + (size_t)j * cols + at, cnt), j, s[0]);
    Chunk o = sub ? load(w + at, cnt) : Chunk{};
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const double t = (s[0][e] + s[1][e]) + (s[2][e] + s[3][e]);
      o.v[e] = sub ? (S)((double)o.v[e] - t) : (S)t;
    }
    store(w + at, o, cnt);
  };
  const int64_t chunks = values / E;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < chunks; i += (int64_t)gridDim.x * blockDim.x)
    piece(i * E, E, [](const S *p, int) { return *reinterpret_cast<const Chunk *>(p); },
          [](S *p, const Chunk &c, int) { *reinterpret_cast<Chunk *>(p) = c; });
  if (chunks * E < values && blockIdx.x == 0 && threadIdx.x == 0)
    piece(chunks * E, (int)(values - chunks * E),
          [](const S *p, int cnt) { Chunk c{}; for (int e = 0; e < cnt; ++e) c.v[e] = p[e]; return c; },
          [](S *p, const Chunk &c, int cnt) { for (int e = 0; e < cnt; ++e) p[e] = c.v[e]; });
}

// Gaussian start vector from a counter-based hash (Box-Muller).
template <typename S>
__global__ void k_fill_gauss(int64_t len, uint64_t seed, S *out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t h1 = el::counter_hash(seed, 0x5151, (uint64_t)i);
    const uint64_t h2 = el::counter_hash(seed, 0xA7A7, (uint64_t)i);
    const double u1 = ((h1 >> 11) + 1.0) * (1.0 / 9007199254740993.0);
    const double u2 = (h2 >> 11) * (1.0 / 9007199254740992.0);
    out[i] = (S)(sqrt(-2.0 * log(u1)) * cospi(2.0 * u2));
  }
}

// Probe block [dim][nvec]; probes v >= nvalid are zero vectors.
template <typename S>
__global__ void k_fill_rademacher(int64_t dim, int nvec, uint64_t seed,
                                  int64_t probe0, int nvalid, S *out) {
  const int64_t total = dim * nvec;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t / nvec, v = t % nvec;
    out[t] = v < nvalid ? (S)el::rademacher(seed, (uint64_t)(probe0 + v), (uint64_t)r) : (S)0;
  }
}

// probes_dev is [nvec][dim] int8; out is [dim][nvec]
template <typename S>
__global__ void k_probe_copy(int64_t dim, int nvec, const int8_t *probes, S *out) {
  const int64_t total = dim * nvec;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t / nvec, v = t % nvec;
    out[t] = (S)probes[v * dim + r];
  }
}

template <typename S>
__global__ void k_scale(int64_t len, const double *scale, int invert_sqrt, S *x) {
  const double s = invert_sqrt ? 1.0 / sqrt(*scale) : *scale;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len;
       i += (int64_t)gridDim.x * blockDim.x)
    x[i] = (S)((double)x[i] * s);
}

// out[k] = sum |psi_r|^2 bit_k(r) (k < n), out[n] = sum |psi_r|^2
template <typename S, bool C>
__global__ void k_observables(BasisDev B, const S *psi, double *partials,
                              unsigned int *counter, double *out) {
  __shared__ double ws[8][EL_MAX_SITES + 1];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = B.n;
  for (int k = threadIdx.x; k < 8 * (EL_MAX_SITES + 1); k += blockDim.x) (&ws[0][0])[k] = 0.0;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < B.dim; base += stride) {
    const int64_t r = base + threadIdx.x;
    double p = 0.0;
    uint64_t code = 0;
    if (r < B.dim) {
      code = el::unrank_row(B, r);
      if constexpr (C) { const double a = psi[2 * r], b = psi[2 * r + 1]; p = a * a + b * b; }
      else { const double a = psi[r]; p = a * a; }
    }
    for (int k = 0; k <= n; ++k) {
      double v = (k == n) ? p : (((code >> k) & 1ULL) ? p : 0.0);
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) ws[warp][k] += v;
    }
  }
  __syncthreads();
  const int nout = n + 1;
  for (int k = threadIdx.x; k < nout; k += blockDim.x) {
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += ws[w][k];
    partials[(size_t)blockIdx.x * nout + k] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int k = threadIdx.x; k < nout; k += blockDim.x) {
    double s = 0.0;
    for (unsigned b = 0; b < gridDim.x; ++b) s += __ldcg(&partials[(size_t)b * nout + k]);
    out[k] = s;
  }
  if (threadIdx.x == 0) *counter = 0u;
}

bool is_complex(int dtype) { return dtype == EL_C64 || dtype == EL_C128; }

}  // namespace

namespace {

// Rows below which one vector goes to the row kernel: a launch is then all
// latency, and the row kernel's chain (its gathers) is shorter than the tiled
// kernels' (tile, barrier, gathers).  Full basis, row against tiled kernel
// alone (torch profiler): n = 15 3.1 against 4.8 us in float32, 3.4 and 5.0
// float64, 3.8 and 5.0 complex64, 4.9 and 5.4 complex128; n = 16 4.3 and 5.1,
// 5.3 and 5.3, 5.7 and 5.3, 8.4 and 5.8; n = 17 7.2 and 5.4, 15.0 and 6.2.
// Chains, float64: n = 18 4.7 against 8.3 us, 22 8.3 against 10.3, 23 (75,025
// rows) 10.3 both.
constexpr int64_t ROW_FULL = 1 << 16, ROW_SECTOR = 75776;
constexpr int ROW_LANES = 4;

bool row_kernel_ok(const el_ham *h, const ApplyArgs &A) {
  if (!h->px.empty() || h->lossy) return false;   // exchange channels or loss: generic kernel
  const int lay = h->basis->layout;
  if (lay != EL_LAYOUT_FULL && lay != EL_LAYOUT_CHAIN && lay != EL_LAYOUT_RING) return false;
  if (A.nvec != 1 || h->n > 32 || h->basis->dim >= (lay == EL_LAYOUT_FULL ? ROW_FULL : ROW_SECTOR)) return false;
  const size_t align = dtype_size(A.dtype);
  for (const void *p : {A.x, (const void *)A.z, (const void *)A.y, (const void *)A.acc, A.probe})
    if (p && ((uintptr_t)p % align) != 0) return false;
  return true;
}

template <typename S, bool C, bool WANT>
void launch_row_lay(el_ctx *ctx, int lay, int grid, const BasisDev &B, const HamArgs<S> &H, const KArgs &K) {
  if (lay == EL_LAYOUT_FULL)
    k_apply_row<S, C, EL_LAYOUT_FULL, WANT, ROW_LANES><<<grid, 256, 0, ctx->stream>>>(B, H, K);
  else if (lay == EL_LAYOUT_CHAIN)
    k_apply_row<S, C, EL_LAYOUT_CHAIN, WANT, ROW_LANES><<<grid, 256, 0, ctx->stream>>>(B, H, K);
  else
    k_apply_row<S, C, EL_LAYOUT_RING, WANT, ROW_LANES><<<grid, 256, 0, ctx->stream>>>(B, H, K);
}

template <typename S, bool C>
void launch_row_t(el_ctx *ctx, int lay, bool want, int grid, const BasisDev &B, const HamArgs<S> &H,
                  const KArgs &K) {
  if (want) launch_row_lay<S, C, true>(ctx, lay, grid, B, H, K);
  else launch_row_lay<S, C, false>(ctx, lay, grid, B, H, K);
}

int launch_apply_row(el_ctx *ctx, el_ham *h, const ApplyArgs &A, const BasisDev &B, KArgs K) {
  const int lay = h->basis->layout;
  const int grid = el::grid_for(h->basis->dim * ROW_LANES, 256);
  const bool want = K.want != 0;
  if (want) {
    K.nvec = 1;
    K.lognv = 0;
    int rc = el::ensure_partials(ctx, (size_t)grid * 4);
    if (rc) return rc;
    K.partials = ctx->d_partials;
  }
  switch (A.dtype) {
    case EL_F32: launch_row_t<float, false>(ctx, lay, want, grid, B, ham_args<float>(h, h->d_diagV32), K); break;
    case EL_F64: launch_row_t<double, false>(ctx, lay, want, grid, B, ham_args<double>(h, h->d_diagV64), K); break;
    case EL_C64: launch_row_t<float, true>(ctx, lay, want, grid, B, ham_args<float>(h, h->d_diagV32), K); break;
    case EL_C128: launch_row_t<double, true>(ctx, lay, want, grid, B, ham_args<double>(h, h->d_diagV64), K); break;
    default: return el::fail(ctx, EL_EINVAL, "unknown dtype %d", A.dtype);
  }
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

}  // namespace

namespace el {

int launch_apply(el_ctx *ctx, el_ham *h, const ApplyArgs &A) {
  const int64_t nvec = A.nvec;
  if (nvec < 1 || nvec > 256 || (nvec & (nvec - 1)))
    return fail(ctx, EL_EINVAL, "nvec must be a power of two in [1, 256], got %lld", (long long)nvec);
  if (!is_complex(A.dtype) && (h->complex_drive))
    return fail(ctx, EL_EINVAL, "complex Omega, J or A needs a complex vector dtype");
  BasisDev B = basis_dev(h->basis);
  KArgs K;
  K.nvec = nvec;
  K.lognv = ilog2(nvec);
  K.x = A.x; K.z = A.z; K.y = A.y; K.acc = A.acc;
  K.a = A.a; K.b = A.b; K.c = A.c; K.c_dev = A.c_dev; K.w_re = A.w_re; K.w_im = A.w_im;
  K.dots = A.dots;
  K.want = A.dots ? (A.want_dots ? A.want_dots : 7) : 0;
  K.skip_diag = A.skip_diag;
  K.probe = A.probe;
  K.counter = ctx->d_counter;
  const int64_t total = h->basis->dim * nvec;
  const int grid = grid_for(total, 256);
  if (K.want) {
    int rc = ensure_partials(ctx, (size_t)grid * nvec * 4);
    if (rc) return rc;
  }
  K.partials = ctx->d_partials;
  const bool single = (A.dtype == EL_F32 || A.dtype == EL_C64);
  if (single) {
    int rc = ham_diag32(ctx, h);
    if (rc) return rc;
  }
  if (row_kernel_ok(h, A)) return launch_apply_row(ctx, h, A, B, K);
  if (chain_block_ok(ctx, h, A)) return launch_chain_block(ctx, h, A, B, K);
  if (full_block_ok(h, A)) return launch_full_block(ctx, h, A, K);
  if (table_block_ok(h, A)) return launch_table_block(ctx, h, A, B, K);
  if (!h->px.empty() && (B.layout == EL_LAYOUT_FULL || B.layout == EL_LAYOUT_TABLE) && B.n <= 32 &&
      B.dim < ((int64_t)1 << 31)) {
    const size_t sm = (size_t)B.n * B.n * (single ? sizeof(float) : sizeof(double)) * 2;
    switch (A.dtype) {
      case EL_F32: k_apply_hop<float, false><<<grid, 256, sm, ctx->stream>>>(B, ham_args<float>(h, h->d_diagV32), K, h->d_hop, h->d_pxA, h->npxA); break;
      case EL_F64: k_apply_hop<double, false><<<grid, 256, sm, ctx->stream>>>(B, ham_args<double>(h, h->d_diagV64), K, h->d_hop, h->d_pxA, h->npxA); break;
      case EL_C64: k_apply_hop<float, true><<<grid, 256, sm, ctx->stream>>>(B, ham_args<float>(h, h->d_diagV32), K, h->d_hop, h->d_pxA, h->npxA); break;
      case EL_C128: k_apply_hop<double, true><<<grid, 256, sm, ctx->stream>>>(B, ham_args<double>(h, h->d_diagV64), K, h->d_hop, h->d_pxA, h->npxA); break;
      default: return fail(ctx, EL_EINVAL, "unknown dtype %d", A.dtype);
    }
    EL_LAUNCH_CHECK(ctx);
    return EL_OK;
  }
  switch (A.dtype) {
    case EL_F32:
      k_apply<float, false><<<grid, 256, 0, ctx->stream>>>(B, ham_args<float>(h, h->d_diagV32), K);
      break;
    case EL_F64:
      k_apply<double, false><<<grid, 256, 0, ctx->stream>>>(B, ham_args<double>(h, h->d_diagV64), K);
      break;
    case EL_C64:
      k_apply<float, true><<<grid, 256, 0, ctx->stream>>>(B, ham_args<float>(h, h->d_diagV32), K);
      break;
    case EL_C128:
      k_apply<double, true><<<grid, 256, 0, ctx->stream>>>(B, ham_args<double>(h, h->d_diagV64), K);
      break;
    default:
      return fail(ctx, EL_EINVAL, "unknown dtype %d", A.dtype);
  }
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

int launch_diag_v(el_ctx *ctx, el_ham *h) {
  BasisDev B = basis_dev(h->basis);
  const int n = h->n;
  double *d_V = nullptr;
  EL_CUDA_TRY(ctx, cudaMalloc(&d_V, (size_t)n * n * sizeof(double)));
  cudaError_t e = el::copy(ctx, d_V, h->Vbits.data(), (size_t)n * n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_diag_v<<<grid_for(B.dim, 256), 256, (size_t)n * n * sizeof(double), ctx->stream>>>(
        B, n, d_V, h->d_diagV64, nullptr);
    ctx->launches++;
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  cudaFree(d_V);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "diag_v");
  return EL_OK;
}

__global__ void k_to_f32(int64_t len, const double *a, float *b) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len;
       i += (int64_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}

int ham_diag32(el_ctx *ctx, el_ham *h) {
  if (h->d_diagV32) return EL_OK;
  const int64_t dim = h->basis->dim;
  EL_CUDA_TRY(ctx, cudaMalloc(&h->d_diagV32, (size_t)dim * sizeof(float)));
  k_to_f32<<<grid_for(dim, 256), 256, 0, ctx->stream>>>(dim, h->d_diagV64, h->d_diagV32);
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

int launch_full_diag(el_ctx *ctx, el_ham *h, int dtype, void *out) {
  BasisDev B = basis_dev(h->basis);
  HamArgs<double> H = ham_args<double>(h, h->d_diagV64);
  if (dtype == EL_F64)
    k_full_diag<double><<<grid_for(B.dim, 256), 256, 0, ctx->stream>>>(B, H, (double *)out);
  else if (dtype == EL_F32)
    k_full_diag<float><<<grid_for(B.dim, 256), 256, 0, ctx->stream>>>(B, H, (float *)out);
  else
    return fail(ctx, EL_EINVAL, "diagonal dtype must be EL_F32 or EL_F64");
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

int gershgorin(el_ctx *ctx, el_ham *h, double *lo, double *hi, double *norm1) {
  BasisDev B = basis_dev(h->basis);
  HamArgs<double> H = ham_args<double>(h, h->d_diagV64);
  const int grid = std::min(grid_for(B.dim, 256), 8 * sm_count(ctx));
  int rc = ensure_partials(ctx, (size_t)grid * 3);
  if (rc) return rc;
  const int charge = h->basis->kind == EL_BASIS_CHARGE;
#define EL_GERSH(LAY) k_gersh_masks<LAY><<<grid, 256, 0, ctx->stream>>>(B, H, charge, ctx->d_partials, ctx->d_counter, ctx->d_scalars)
  if (!h->px.empty() || B.n > 32 || B.dim >= ((int64_t)1 << 32))
    k_gershgorin<<<grid, 256, 0, ctx->stream>>>(B, H, ctx->d_partials, ctx->d_counter, ctx->d_scalars);
  else if (B.layout == EL_LAYOUT_FULL) EL_GERSH(EL_LAYOUT_FULL);
  else if (B.layout == EL_LAYOUT_CHAIN) EL_GERSH(EL_LAYOUT_CHAIN);
  else if (B.layout == EL_LAYOUT_RING) EL_GERSH(EL_LAYOUT_RING);
  else EL_GERSH(EL_LAYOUT_TABLE);
#undef EL_GERSH
  EL_LAUNCH_CHECK(ctx);
  EL_CUDA_TRY(ctx, el::copy(ctx, ctx->h_scalars, ctx->d_scalars, 3 * sizeof(double), cudaMemcpyDeviceToHost));
  EL_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  *lo = ctx->h_scalars[0];
  *hi = ctx->h_scalars[1];
  if (norm1) *norm1 = ctx->h_scalars[2];
  return EL_OK;
}

static int axpby(el_ctx *ctx, int dtype, int64_t len, double a_re, double a_im, const void *x, double b_re,
                 double b_im, void *y, double *norm2_out, const LanczosScalars &U) {
  const bool aln = (((uintptr_t)x | (uintptr_t)y) & 15) == 0;
  const int es = dtype_size(dtype);
  if (!es) return fail(ctx, EL_EINVAL, "unknown dtype %d", dtype);
  const int grid = grid_for(aln ? (len * es + 15) / 16 : len, 256);
  if (norm2_out || U.dots) {
    int rc = ensure_partials(ctx, (size_t)grid);
    if (rc) return rc;
  }
#define EL_AXPBY(S, C)                                                                                 \
  do {                                                                                                 \
    if (aln)                                                                                           \
      k_axpby<S, C, true><<<grid, 256, 0, ctx->stream>>>(len, a_re, a_im, (const S *)x, b_re, b_im,    \
                                                         (S *)y, ctx->d_partials, ctx->d_counter,      \
                                                         norm2_out, U);                                \
    else                                                                                               \
      k_axpby<S, C, false><<<grid, 256, 0, ctx->stream>>>(len, a_re, a_im, (const S *)x, b_re, b_im,   \
                                                          (S *)y, ctx->d_partials, ctx->d_counter,     \
                                                          norm2_out, U);                               \
  } while (0)
  switch (dtype) {
    case EL_F32: EL_AXPBY(float, false); break;
    case EL_F64: EL_AXPBY(double, false); break;
    case EL_C64: EL_AXPBY(float, true); break;
    default: EL_AXPBY(double, true); break;
  }
#undef EL_AXPBY
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

int launch_axpby(el_ctx *ctx, int dtype, int64_t len, double a_re, double a_im,
                 const void *x, double b_re, double b_im, void *y, double *norm2_out) {
  return axpby(ctx, dtype, len, a_re, a_im, x, b_re, b_im, y, norm2_out, LanczosScalars{nullptr, nullptr, nullptr});
}

int launch_lanczos_update(el_ctx *ctx, int dtype, int64_t len, const void *x, void *y, const double *dots,
                          const double *k2, double *rec) {
  return axpby(ctx, dtype, len, 0, 0, x, 1, 0, y, nullptr, LanczosScalars{dots, k2, rec});
}

int launch_gemv_t(el_ctx *ctx, int dtype, int64_t len, int k, const void *V,
                  int64_t ld, const void *w, double *dots_out) {
  if (k <= 0) return EL_OK;
  // one CTA per SM and column group: each thread walks many rows, so the
  // block reduction is paid once per many rows
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  int gx = grid_for(len, 256);
  const int ngroups = (k + GJ - 1) / GJ;
  const int gcap = std::max(1, (2 * sms + ngroups - 1) / ngroups);   // about two CTAs per SM in total
  if (gx > gcap) gx = gcap;
  dim3 grid(gx, ngroups);
  const bool aln = (((uintptr_t)V | (uintptr_t)w | ((size_t)ld * dtype_size(dtype))) & 15) == 0;
  int rc = ensure_partials(ctx, (size_t)gx * k * 2);
  if (rc) return rc;
  switch (dtype) {
#define EL_GEMVT(S, C)                                                                                            \
  do {                                                                                                            \
    if (aln) k_gemv_t<S, C, true><<<grid, 256, 0, ctx->stream>>>(len, k, (const S *)V, ld, (const S *)w, ctx->d_partials); \
    else k_gemv_t<S, C, false><<<grid, 256, 0, ctx->stream>>>(len, k, (const S *)V, ld, (const S *)w, ctx->d_partials);    \
  } while (0)
    case EL_F32: EL_GEMVT(float, false); break;
    case EL_F64: EL_GEMVT(double, false); break;
    case EL_C64: EL_GEMVT(float, true); break;
    case EL_C128: EL_GEMVT(double, true); break;
#undef EL_GEMVT
    default: return fail(ctx, EL_EINVAL, "unknown dtype %d", dtype);
  }
  EL_LAUNCH_CHECK(ctx);
  k_sum_partials<<<(2 * k + 31) / 32, 256, 0, ctx->stream>>>(gx, k, ctx->d_partials, dots_out);
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

static int gemv_n(el_ctx *ctx, int dtype, int64_t len, int k, const void *V, int64_t ld, const double *coef,
                  void *w, bool sub) {
  if (k <= 0) return EL_OK;
  const int es = dtype_size(dtype);
  if (!es) return fail(ctx, EL_EINVAL, "unknown dtype %d", dtype);
  // pieces where they still fill the GPU: a thread's columns are a chain of reads
  const bool aln = (((uintptr_t)V | (uintptr_t)w | ((size_t)ld * es)) & 15) == 0 &&
                   len * es / 16 >= (int64_t)sm_count(ctx) * 1024;
  const int grid = grid_for(aln ? (len * es + 15) / 16 : len, 256);
#define EL_GEMVN(S, C)                                                                                         \
  do {                                                                                                         \
    if (aln) k_gemv_n<S, C, true><<<grid, 256, 0, ctx->stream>>>(len, k, (const S *)V, ld, coef, (S *)w, sub); \
    else k_gemv_n<S, C, false><<<grid, 256, 0, ctx->stream>>>(len, k, (const S *)V, ld, coef, (S *)w, sub);    \
  } while (0)
  switch (dtype) {
    case EL_F32: EL_GEMVN(float, false); break;
    case EL_F64: EL_GEMVN(double, false); break;
    case EL_C64: EL_GEMVN(float, true); break;
    default: EL_GEMVN(double, true); break;
  }
#undef EL_GEMVN
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

int launch_gemv_n_sub(el_ctx *ctx, int dtype, int64_t len, int k, const void *V,
                      int64_t ld, const double *coef, void *w) {
  return gemv_n(ctx, dtype, len, k, V, ld, coef, w, true);
}

int launch_gemv_n(el_ctx *ctx, int dtype, int64_t len, int k, const void *V,
                  int64_t ld, const double *coef_dev, void *out) {
  return gemv_n(ctx, dtype, len, k, V, ld, coef_dev, out, false);
}

int launch_fill_gauss(el_ctx *ctx, int dtype, int64_t len, uint64_t seed, void *out) {
  const int grid = grid_for(len, 256);
  switch (dtype) {
    case EL_F32: k_fill_gauss<float><<<grid, 256, 0, ctx->stream>>>(len, seed, (float *)out); break;
    case EL_F64: k_fill_gauss<double><<<grid, 256, 0, ctx->stream>>>(len, seed, (double *)out); break;
    case EL_C64: k_fill_gauss<float><<<grid_for(2 * len, 256), 256, 0, ctx->stream>>>(2 * len, seed, (float *)out); break;
    case EL_C128: k_fill_gauss<double><<<grid_for(2 * len, 256), 256, 0, ctx->stream>>>(2 * len, seed, (double *)out); break;
    default: return fail(ctx, EL_EINVAL, "unknown dtype %d", dtype);
  }
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

int launch_fill_rademacher(el_ctx *ctx, int dtype, int64_t dim, int nvec,
                           uint64_t seed, int64_t probe0, int nvalid, void *out) {
  const int grid = grid_for(dim * nvec, 256);
  if (dtype == EL_F32)
    k_fill_rademacher<float><<<grid, 256, 0, ctx->stream>>>(dim, nvec, seed, probe0, nvalid, (float *)out);
  else if (dtype == EL_F64)
    k_fill_rademacher<double><<<grid, 256, 0, ctx->stream>>>(dim, nvec, seed, probe0, nvalid, (double *)out);
  else
    return fail(ctx, EL_EINVAL, "probes need a real dtype");
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

int launch_probe_copy(el_ctx *ctx, int dtype, int64_t dim, int nvec,
                      const int8_t *probes_dev, void *out) {
  const int grid = grid_for(dim * nvec, 256);
  if (dtype == EL_F32)
    k_probe_copy<float><<<grid, 256, 0, ctx->stream>>>(dim, nvec, probes_dev, (float *)out);
  else if (dtype == EL_F64)
    k_probe_copy<double><<<grid, 256, 0, ctx->stream>>>(dim, nvec, probes_dev, (double *)out);
  else
    return fail(ctx, EL_EINVAL, "probes need a real dtype");
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

int launch_scale(el_ctx *ctx, int dtype, int64_t len, const double *scale_dev,
                 int invert_sqrt, void *x) {
  const int64_t n = is_complex(dtype) ? 2 * len : len;
  const int grid = grid_for(n, 256);
  if (dtype == EL_F32 || dtype == EL_C64)
    k_scale<float><<<grid, 256, 0, ctx->stream>>>(n, scale_dev, invert_sqrt, (float *)x);
  else
    k_scale<double><<<grid, 256, 0, ctx->stream>>>(n, scale_dev, invert_sqrt, (double *)x);
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

int launch_observables(el_ctx *ctx, el_ham *h, int dtype, const void *psi, double *out_dev) {
  BasisDev B = basis_dev(h->basis);
  const int grid = grid_for(B.dim, 256);
  int rc = ensure_partials(ctx, (size_t)grid * (B.n + 1));
  if (rc) return rc;
  switch (dtype) {
    case EL_F32: k_observables<float, false><<<grid, 256, 0, ctx->stream>>>(B, (const float *)psi, ctx->d_partials, ctx->d_counter, out_dev); break;
    case EL_F64: k_observables<double, false><<<grid, 256, 0, ctx->stream>>>(B, (const double *)psi, ctx->d_partials, ctx->d_counter, out_dev); break;
    case EL_C64: k_observables<float, true><<<grid, 256, 0, ctx->stream>>>(B, (const float *)psi, ctx->d_partials, ctx->d_counter, out_dev); break;
    case EL_C128: k_observables<double, true><<<grid, 256, 0, ctx->stream>>>(B, (const double *)psi, ctx->d_partials, ctx->d_counter, out_dev); break;
    default: return fail(ctx, EL_EINVAL, "unknown dtype %d", dtype);
  }
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

}  // namespace el

// ------------------------------------------------------------------ C ABI

extern "C" {

int el_ham_create(el_ctx *ctx, el_basis *basis, const double *omega_re,
                  const double *omega_im, const double *delta, int n_pairs,
                  const int32_t *pi, const int32_t *pj, const double *V, el_ham **out) {
  if (!ctx || !basis || !out || !omega_re || !delta) return EL_EINVAL;
  *out = nullptr;
  if (n_pairs < 0 || (n_pairs > 0 && (!pi || !pj || !V))) return fail(ctx, EL_EINVAL, "bad pair list");
  EL_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int n = basis->n;
  el_ham *h = new el_ham();
  h->basis = basis;
  h->n = n;
  memset(h->om_re, 0, sizeof h->om_re);
  memset(h->om_im, 0, sizeof h->om_im);
  memset(h->delta, 0, sizeof h->delta);
  memset(h->loss, 0, sizeof h->loss);
  h->Vbits.assign((size_t)n * n, 0.0);
  for (int p = 0; p < n_pairs; ++p) {
    const int i = pi[p], j = pj[p];
    if (i < 0 || j < 0 || i >= n || j >= n || i == j || !std::isfinite(V[p])) {
      delete h;
      return fail(ctx, EL_EINVAL, "pair %d: bad sites (%d, %d) or non-finite V", p, i, j);
    }
    const int qi = n - 1 - i, qj = n - 1 - j;
    h->Vbits[(size_t)qi * n + qj] += V[p];
    if (qi != qj) h->Vbits[(size_t)qj * n + qi] += V[p];
  }
  int rc = el_ham_set_drive(ctx, h, omega_re, omega_im, delta);
  if (rc) { delete h; return rc; }
  cudaError_t e = cudaMalloc(&h->d_diagV64, (size_t)basis->dim * sizeof(double));
  if (e != cudaSuccess) { delete h; return el::fail(ctx, EL_ENOMEM, "cannot allocate diagonal (%s)", cudaGetErrorString(e)); }
  rc = el::launch_diag_v(ctx, h);
  if (rc) { el_ham_destroy(h); return rc; }
  *out = h;
  return EL_OK;
}

int el_ham_set_drive(el_ctx *ctx, el_ham *h, const double *omega_re,
                     const double *omega_im, const double *delta) {
  if (!ctx || !h || !omega_re || !delta) return EL_EINVAL;
  const int n = h->n;
  bool cplx = false;
  for (int i = 0; i < n; ++i) {
    const double ore = omega_re[i], oim = omega_im ? omega_im[i] : 0.0, d = delta[i];
    if (!std::isfinite(ore) || !std::isfinite(oim) || !std::isfinite(d))
      return fail(ctx, EL_EINVAL, "Om/delta must be finite");
    const int q = n - 1 - i;
    h->om_re[q] = ore;
    h->om_im[q] = oim;
    h->delta[q] = d;
    if (oim != 0.0) cplx = true;
  }
  h->drive_complex = cplx;
  h->complex_drive = h->drive_complex || h->px_complex || h->lossy;
  return EL_OK;
}

int el_ham_set_loss(el_ctx *ctx, el_ham *h, const double *gamma) {
  if (!ctx || !h) return EL_EINVAL;
  const int n = h->n;
  // channels.py:69-76: diagonal (delta_i - 0.5 i gamma_i 1e-3 / CONV) n_i
  const double conv = 2.0 * 3.14159265358979323846 * 1e-3;
  bool any = false;
  double loss[EL_MAX_SITES] = {0.0};
  for (int i = 0; gamma && i < n; ++i) {
    if (!std::isfinite(gamma[i])) return fail(ctx, EL_EINVAL, "gamma must be finite");
    loss[n - 1 - i] = -0.5 * gamma[i] * 1e-3 / conv;
    if (gamma[i] != 0.0) any = true;
  }
  memcpy(h->loss, loss, sizeof loss);
  h->lossy = any;
  h->complex_drive = h->drive_complex || h->px_complex || h->lossy;
  return EL_OK;
}

int el_ham_set_exchange(el_ctx *ctx, el_ham *h, int n_pairs, const int32_t *pi,
                        const int32_t *pj, const double *J_re, const double *J_im,
                        const double *A_re, const double *A_im) {
  if (!ctx || !h) return EL_EINVAL;
  if (n_pairs < 0 || (n_pairs > 0 && (!pi || !pj))) return fail(ctx, EL_EINVAL, "bad exchange pair list");
  EL_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int n = h->n;
  std::vector<ExPair> px;
  bool cplx = false;
  for (int p = 0; p < n_pairs; ++p) {
    const int i = pi[p], j = pj[p];
    ExPair e;
    e.jre = J_re ? J_re[p] : 0.0;
    e.jim = J_im ? J_im[p] : 0.0;
    e.are = A_re ? A_re[p] : 0.0;
    e.aim = A_im ? A_im[p] : 0.0;
    if (i < 0 || j < 0 || i >= n || j >= n || i == j)
      return fail(ctx, EL_EINVAL, "exchange pair %d: bad sites (%d, %d)", p, i, j);
    if (!std::isfinite(e.jre) || !std::isfinite(e.jim) || !std::isfinite(e.are) || !std::isfinite(e.aim))
      return fail(ctx, EL_EINVAL, "exchange pair %d: non-finite J or A", p);
    if (e.jre == 0.0 && e.jim == 0.0 && e.are == 0.0 && e.aim == 0.0) continue;
    e.bi = n - 1 - i;
    e.bj = n - 1 - j;
    if (e.jim != 0.0 || e.aim != 0.0) cplx = true;
    px.push_back(e);
  }
  // hop table of the J channels and the list of A pairs
  std::vector<double> hop(2 * (size_t)n * n, 0.0);
  std::vector<ExPair> pxA;
  for (const ExPair &e : px) {
    // row (i, j) = (r, g): bit bi set, bj clear -> J; row (g, r) -> conj(J)
    hop[(size_t)e.bi * n + e.bj] += e.jre;
    hop[(size_t)n * n + (size_t)e.bi * n + e.bj] += e.jim;
    hop[(size_t)e.bj * n + e.bi] += e.jre;
    hop[(size_t)n * n + (size_t)e.bj * n + e.bi] -= e.jim;
    if (e.are != 0.0 || e.aim != 0.0) pxA.push_back(e);
  }
  ExPair *d = nullptr, *dA = nullptr;
  double *dh = nullptr;
  auto upload = [&](void **dst, const void *src, size_t bytes) -> cudaError_t {
    cudaError_t e = cudaMalloc(dst, bytes);
    if (e != cudaSuccess) return e;
    e = el::copy(ctx, *dst, src, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    return e;
  };
  if (!px.empty()) {
    cudaError_t e = upload((void **)&d, px.data(), px.size() * sizeof(ExPair));
    if (e == cudaSuccess) e = upload((void **)&dh, hop.data(), hop.size() * sizeof(double));
    if (e == cudaSuccess && !pxA.empty()) e = upload((void **)&dA, pxA.data(), pxA.size() * sizeof(ExPair));
    if (e != cudaSuccess) {
      cudaFree(d); cudaFree(dh); cudaFree(dA);
      cudaGetLastError();
      return el::fail(ctx, EL_ENOMEM, "cannot store exchange channels (%s)", cudaGetErrorString(e));
    }
  }
  // the previous lists may still be read by work queued on the stream
  if (h->d_px || h->d_hop || h->d_pxA) {
    EL_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    cudaFree(h->d_px);
    cudaFree(h->d_hop);
    cudaFree(h->d_pxA);
  }
  h->d_px = d;
  h->d_hop = dh;
  h->d_pxA = dA;
  h->npxA = (int)pxA.size();
  h->px.swap(px);
  h->px_complex = cplx;
  h->complex_drive = h->drive_complex || h->px_complex || h->lossy;
  return EL_OK;
}

int el_ham_diag(el_ctx *ctx, el_ham *h, int dtype, void *out) {
  if (!ctx || !h || !out) return EL_EINVAL;
  EL_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  return el::launch_full_diag(ctx, h, dtype, out);
}

int el_ham_destroy(el_ham *h) {
  if (!h) return EL_OK;
  if (h->basis) cudaSetDevice(h->basis->device);
  if (h->d_diagV64) cudaFree(h->d_diagV64);
  if (h->d_diagV32) cudaFree(h->d_diagV32);
  if (h->d_px) cudaFree(h->d_px);
  if (h->d_hop) cudaFree(h->d_hop);
  if (h->d_pxA) cudaFree(h->d_pxA);
  delete h;
  return EL_OK;
}

int el_hv(el_ctx *ctx, el_ham *h, int dtype, int nvec, const void *x, void *y) {
  if (!ctx || !h || !x || !y) return EL_EINVAL;
  if (x == y) return el::fail(ctx, EL_EINVAL, "el_hv: x and y must not alias");
  EL_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  ApplyArgs A;
  memset(&A, 0, sizeof A);
  A.dtype = dtype;
  A.nvec = nvec;
  A.x = x;
  A.y = y;
  A.a = 1.0;
  return el::launch_apply(ctx, h, A);
}

int el_hv_host(el_ctx *ctx, el_ham *h, int dtype, int nvec, const void *x_host, void *y_host) {
  if (!ctx || !h || !x_host || !y_host) return EL_EINVAL;
  const int es = el::dtype_size(dtype);
  if (!es) return el::fail(ctx, EL_EINVAL, "unknown dtype %d", dtype);
  EL_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const size_t bytes = (size_t)h->basis->dim * nvec * es;
  // device copies in the context's cached workspace (kept between calls)
  char *buf = (char *)el::workspace(ctx, 14, 2 * bytes);
  if (!buf) return EL_ENOMEM;
  void *dx = buf, *dy = buf + bytes;
  cudaError_t e = el::copy(ctx, dx, x_host, bytes, cudaMemcpyHostToDevice);
  int rc = EL_OK;
  if (e == cudaSuccess) {
    rc = el_hv(ctx, h, dtype, nvec, dx, dy);
    if (rc == EL_OK) {
      e = el::copy(ctx, y_host, dy, bytes, cudaMemcpyDeviceToHost);
      if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    }
  }
  if (rc) return rc;
  if (e != cudaSuccess) return el::cuda_fail(ctx, e, "el_hv_host");
  return EL_OK;
}

int el_observables(el_ctx *ctx, el_ham *h, int dtype, const void *psi,
                   double *n_site_host, double *norm_host) {
  if (!ctx || !h || !psi) return EL_EINVAL;
  EL_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int n = h->n;
  int rc = el::launch_observables(ctx, h, dtype, psi, ctx->d_scalars);
  if (rc) return rc;
  EL_CUDA_TRY(ctx, el::copy(ctx, ctx->h_scalars, ctx->d_scalars, (n + 1) * sizeof(double), cudaMemcpyDeviceToHost));
  EL_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  if (n_site_host)
    for (int i = 0; i < n; ++i) n_site_host[i] = ctx->h_scalars[n - 1 - i];
  if (norm_host) *norm_host = ctx->h_scalars[n];
  return EL_OK;
}

}  // extern "C"
