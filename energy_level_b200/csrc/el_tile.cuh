// Device helpers of the tiled H-apply kernels (el_chain.cu, el_full.cu): a
// row's vectors in chunks of at most 16 bytes, the flip's multiply-add, the
// fused recurrence on a chunk and the sums of its dot products.
#pragma once

#include "el_apply.cuh"

namespace el {

template <typename S, int CW>
struct alignas(CW * sizeof(S)) Chunk {
  S v[CW];
};

// h += a x for two FP32 values in one instruction.
__device__ __forceinline__ void fma2(float &h0, float &h1, float a, float x0, float x1) {
  asm("{\n\t.reg .b64 x, a, h;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 a, {%4, %4};\n\tmov.b64 h, {%0, %1};\n\t"
      "fma.rn.f32x2 h, a, x, h;\n\tmov.b64 {%0, %1}, h;\n\t}"
      : "+f"(h0), "+f"(h1)
      : "f"(x0), "f"(x1), "f"(a));
}

// RA: the amplitudes are real (real Omega) although the vectors are complex.
template <typename S, bool C, int CW, bool RA>
__device__ __forceinline__ void add_flip(Chunk<S, CW> &h, S are, S aim, const Chunk<S, CW> &x) {
  if constexpr (sizeof(S) == 4 && CW % 2 == 0 && (!C || RA)) {
#pragma unroll
    for (int i = 0; i < CW; i += 2) fma2(h.v[i], h.v[i + 1], are, x.v[i], x.v[i + 1]);
  } else if constexpr (C && !RA) {
#pragma unroll
    for (int i = 0; i < CW; i += 2) {
      h.v[i] += are * x.v[i] - aim * x.v[i + 1];
      h.v[i + 1] += are * x.v[i + 1] + aim * x.v[i];
    }
  } else {
#pragma unroll
    for (int i = 0; i < CW; ++i) h.v[i] += are * x.v[i];
  }
}

// Streaming (evict-first) accesses for the vectors that a launch touches
// once (y, z, acc), so that L2 keeps x, whose rows other tiles read again.
template <typename S, int CW>
__device__ __forceinline__ Chunk<S, CW> load_cs(const Chunk<S, CW> *p) {
  union { Chunk<S, CW> c; uint4 q; uint2 d; unsigned w; } u;
  if constexpr (sizeof(Chunk<S, CW>) == 16) u.q = __ldcs(reinterpret_cast<const uint4 *>(p));
  else if constexpr (sizeof(Chunk<S, CW>) == 8) u.d = __ldcs(reinterpret_cast<const uint2 *>(p));
  else u.w = __ldcs(reinterpret_cast<const unsigned *>(p));
  return u.c;
}
template <typename S, int CW>
__device__ __forceinline__ void store_cs(Chunk<S, CW> *p, const Chunk<S, CW> &c) {
  union { Chunk<S, CW> c; uint4 q; uint2 d; unsigned w; } u;
  u.c = c;
  if constexpr (sizeof(Chunk<S, CW>) == 16) __stcs(reinterpret_cast<uint4 *>(p), u.q);
  else if constexpr (sizeof(Chunk<S, CW>) == 8) __stcs(reinterpret_cast<uint2 *>(p), u.d);
  else __stcs(reinterpret_cast<unsigned *>(p), u.w);
}

// The caller's recurrence on one chunk of a row (index e): y = a h + b x + c z,
// acc += w y and the dot products, h = H x.
template <typename S, bool C, int CW, int ND>
__device__ __forceinline__ void finish_chunk(const KArgs &K, int64_t e, const Chunk<S, CW> &h, const Chunk<S, CW> &x,
                                             double (&dots)[C ? CW / 2 : CW][ND ? ND : 1]) {
  typedef Chunk<S, CW> V;
  constexpr int CV = C ? CW / 2 : CW;     // vectors of a chunk
  const S a = (S)K.a, b = (S)K.b;
  V y;
#pragma unroll
  for (int w = 0; w < CW; ++w) y.v[w] = a * h.v[w] + b * x.v[w];
  if (K.z) {
    const V z = load_cs<S, CW>(reinterpret_cast<const V *>(K.z) + e);
    const S c = (S)coef_c(K);
#pragma unroll
    for (int w = 0; w < CW; ++w) y.v[w] += c * z.v[w];
  }
  if (K.acc) {
    V *ap = reinterpret_cast<V *>(K.acc) + e;
    V av = load_cs<S, CW>(ap);
    const S wr = (S)K.w_re, wi = (S)K.w_im;
    if constexpr (C) {
#pragma unroll
      for (int w = 0; w < CW; w += 2) {
        av.v[w] += wr * y.v[w] - wi * y.v[w + 1];
        av.v[w + 1] += wr * y.v[w + 1] + wi * y.v[w];
      }
    } else {
#pragma unroll
      for (int w = 0; w < CW; ++w) av.v[w] += wr * y.v[w];
    }
    store_cs<S, CW>(ap, av);
  }
  if (K.y) store_cs<S, CW>(reinterpret_cast<V *>(K.y) + e, y);
  if constexpr (ND > 0) {
    // FP32 values are widened first: their products are exact in FP64
#pragma unroll
    for (int v = 0; v < CV; ++v) {
      if constexpr (C) {
        const double xr = x.v[2 * v], xi = x.v[2 * v + 1], yr = y.v[2 * v], yi = y.v[2 * v + 1];
        dots[v][0] += xr * xr + xi * xi;
        dots[v][1] += xr * yr + xi * yi;
        if constexpr (ND == 4) {
          dots[v][2] += xr * yi - xi * yr;
          dots[v][3] += yr * yr + yi * yi;
        }
      } else {
        const double xd = x.v[v], yd = y.v[v];
        dots[v][0] += xd * xd;
        dots[v][1] += xd * yd;
        if constexpr (ND == 4) {
          dots[v][3] += yd * yd;
          if (K.probe) dots[v][2] += yd * (double)reinterpret_cast<const V *>(K.probe)[e].v[v];
        }
      }
    }
  }
}

// out[o] = sum of rows[b][o] over b < nrows, in a fixed order, by the whole
// block: output o by nt / nout threads, each adding every (nt / nout)-th row.
__device__ __forceinline__ void sum_rows(const double *rows, int nrows, int nout, double *sm, double *out,
                                         int odst, int osrc) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int per = nout <= nt ? nt / nout : 1;
  for (int o0 = 0; o0 < nout; o0 += nt) {
    const int o = o0 + (per > 1 ? tid % nout : tid), sh = per > 1 ? tid / nout : 0;
    const bool on = o < nout && sh < per;
    double s = 0.0;
    if (on) {
#pragma unroll 8
      for (int b = sh; b < nrows; b += per) s += __ldcg(&rows[(size_t)b * nout + o]);
    }
    __syncthreads();
    if (per > 1) {
      if (on) sm[sh * nout + o] = s;
      __syncthreads();
      if (on && sh == 0) {
        s = 0.0;
        for (int w = 0; w < per; ++w) s += sm[w * nout + o];
      }
    }
    if (on && sh == 0) out[(o / osrc) * odst + o % osrc] = s;
  }
}

// Sums of the dot products over the launch: lanes of a warp that hold the
// same chunk of a row meet by shuffles, warps in shared memory, and blocks in
// global memory in two levels: the last block of each group of `group` to
// finish adds its group's sums, the last group's the groups' (all in fixed
// orders).  One level, the very last block adding 592 rows of 128 sums,
// took 130 of the 160 us of a step with 32 vectors on 24 sites.
// q: ND values (xx, Re xy, then Im xy or <y, probe>, yy) per vector of the chunk.
constexpr int DOT_GROUPS = 48;      // counters 1 .. DOT_GROUPS of the context
template <int CV, int ND>
__device__ void block_dots(const KArgs &K, int nch, double (&q)[CV][ND], double *sm) {
  __shared__ bool last;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
#pragma unroll
  for (int v = 0; v < CV; ++v)
#pragma unroll
    for (int c = 0; c < ND; ++c)
      for (int o = 16; o >= nch; o >>= 1) q[v][c] += __shfl_xor_sync(0xffffffffu, q[v][c], o);
  __syncthreads();                    // the tile in shared memory is done with
  const int nout = nch * CV * ND;
  if (lane < nch) {
#pragma unroll
    for (int v = 0; v < CV; ++v)
#pragma unroll
      for (int c = 0; c < ND; ++c) sm[warp * nout + (lane * CV + v) * ND + c] = q[v][c];
  }
  __syncthreads();
  for (int o = tid; o < nout; o += nt) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += sm[w * nout + o];
    K.partials[(size_t)blockIdx.x * nout + o] = s;
  }
  const int nb = (int)gridDim.x;
  const int group = max(16, (nb + DOT_GROUPS - 1) / DOT_GROUPS);
  const int ngroups = (nb + group - 1) / group, g = (int)blockIdx.x / group;
  const int first = g * group, size = min(group, nb - first);
  double *gsum = K.partials + (size_t)nb * nout;
  __threadfence();
  __syncthreads();
  if (tid == 0) last = (atomicAdd(&K.counter[1 + g], 1u) == (unsigned)size - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  sum_rows(K.partials + (size_t)first * nout, size, nout, sm, gsum + (size_t)g * nout, 1, 1);
  if (tid == 0) K.counter[1 + g] = 0u;
  __threadfence();
  __syncthreads();
  if (tid == 0) last = (atomicAdd(&K.counter[0], 1u) == (unsigned)ngroups - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  sum_rows(gsum, ngroups, nout, sm, K.dots, 4, ND);
  if (tid == 0) K.counter[0] = 0u;
}

// Chunks of at most 16 bytes per row.
inline int chunks_per_row(const ApplyArgs &A) {
  const int rb = (int)A.nvec * dtype_size(A.dtype);
  return rb <= 16 ? 1 : rb / 16;
}

// Every vector of A can be read in those chunks.
inline bool chunks_aligned(const ApplyArgs &A) {
  const size_t rb = (size_t)A.nvec * dtype_size(A.dtype);
  const size_t align = rb >= 16 ? 16 : rb;
  for (const void *p : {A.x, A.z, (const void *)A.y, (const void *)A.acc, A.probe})
    if (p && ((uintptr_t)p % align) != 0) return false;
  return true;
}

}  // namespace el
