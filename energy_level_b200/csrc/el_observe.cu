// Spin observables of a state on the device: the per-site and pair
// expectations that the evolution reports at every output time.
//
// For a state v on the basis of `ham` one launch computes, per requested
// item, three FP64 sums over the rows s of the basis (p = |v_s|^2):
//   norm item         sum p
//   site item i       <n_i>      = sum_{s_i = r} p
//                     <sigma-_i> = sum_{s_i = g} conj(v_s) v_{s + i}   (flip target in the basis)
//   pair item (i, j)  <n_i n_j>  = sum_{s_i = s_j = r} p
//                     <sigma+_i sigma-_j> = sum_{s_i = g, s_j = r} conj(v_t) v_s,
//                                           t = s with i -> r, j -> g (in the basis)
//   Pauli item        <P> = sum_s conj(v_t) c(s) v_s for P = prod of sigma^x/y/z
//                     on distinct sites, t = s ^ (x and y sites), c(s) = i^e with
//                     e = #(y on g) + 3 #(y on r) + 2 #(z on r)  (mod 4), since
//                     sigma^y|g> = i|r>, sigma^y|r> = -i|g>, sigma^z|r> = -|r>
// which are observables.py:117-159 spin_observables (full basis) and
// observables.py:162-205 spin_observables_basis (restricted basis: targets
// outside the basis drop out), the <n_i n_j> of observables.py:40-47
// corr_matrix and PauliPlan.expect (observables.py:486-622) for the Pauli
// strings.  Items come in groups of six, one group per blockIdx.y; a
// thread keeps the 18 sums of its group in registers over a grid-stride
// loop of rows, so v is read once per group and every flip target once per
// item.  Block sums go to per-block partials and a second kernel adds them
// in a fixed order (deterministic results).
#include "el_internal.cuh"

#include <algorithm>
#include <vector>

namespace {

using el::fail;

constexpr int kGroup = 6;   // items per launch column: 6 x 3 FP64 sums fit the registers of 2 CTAs per SM
enum { kNoItem = 0, kNormItem, kSiteItem, kPairItem, kPauliItem };

struct ObsItem {
  int kind;
  int bi, bj;         // bit positions of sites i (site and pair items) and j (pair items)
  int pad_;
  uint64_t fm, ym, zm;  // Pauli item: flipped bits (x and y), y bits, z bits
};

template <typename S, bool C>
__device__ __forceinline__ void load_amp(const S *__restrict__ psi, int64_t r, double &re, double &im) {
  if constexpr (C) { re = (double)psi[2 * r]; im = (double)psi[2 * r + 1]; }
  else { re = (double)psi[r]; im = 0.0; }
}

template <typename S, bool C>
__global__ void __launch_bounds__(256, 2) k_obs_items(BasisDev B, const S *__restrict__ psi,
                                                   const ObsItem *__restrict__ items,
                                                   double *__restrict__ partials, int K) {
  __shared__ double red[8][kGroup * 3];
  __shared__ ObsItem it[kGroup];
  const int g = blockIdx.y;
  if (threadIdx.x < kGroup) it[threadIdx.x] = items[g * kGroup + threadIdx.x];
  __syncthreads();
  double acc[kGroup][3];
#pragma unroll
  for (int q = 0; q < kGroup; ++q) acc[q][0] = acc[q][1] = acc[q][2] = 0.0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < B.dim; r += stride) {
    const uint64_t code = el::unrank_row(B, r);
    double re, im;
    load_amp<S, C>(psi, r, re, im);
    const double p = re * re + im * im;
#pragma unroll
    for (int q = 0; q < kGroup; ++q) {
      const int kind = it[q].kind;
      if (kind == kNoItem) continue;
      if (kind == kNormItem) { acc[q][0] += p; continue; }
      if (kind == kPauliItem) {
        const uint64_t ym = it[q].ym;
        const int64_t t = it[q].fm ? el::rank_any(B, code ^ it[q].fm) : r;
        if (t >= 0) {
          const int e = (__popcll(ym & ~code) + 3 * __popcll(ym & code) + 2 * __popcll(it[q].zm & code)) & 3;
          double wr, wi;
          load_amp<S, C>(psi, t, wr, wi);
          // conj(v_t) v_s, then times i^e
          const double ar = wr * re + wi * im, ai = wr * im - wi * re;
          const double cr = (e == 0) ? ar : (e == 1) ? -ai : (e == 2) ? -ar : ai;
          const double ci = (e == 0) ? ai : (e == 1) ? ar : (e == 2) ? -ai : -ar;
          acc[q][1] += cr;
          acc[q][2] += ci;
        }
        continue;
      }
      const int bi = it[q].bi, bj = it[q].bj;
      const bool si = (code >> bi) & 1ULL;
      if (kind == kSiteItem) {
        if (si) { acc[q][0] += p; continue; }
        const int64_t t = el::flip_target(B, code, r, bi);
        if (t >= 0) {
          double wr, wi;
          load_amp<S, C>(psi, t, wr, wi);
          acc[q][1] += re * wr + im * wi;   // conj(v_s) v_t
          acc[q][2] += re * wi - im * wr;
        }
        continue;
      }
      const bool sj = (code >> bj) & 1ULL;
      if (si && sj) acc[q][0] += p;
      if (!si && sj) {
        // on chain / ring sectors: clear bit j (which keeps the state in the
        // sector), then set bit i -- two O(1) single flips instead of a
        // re-rank; other layouts rank the target directly (on a
        // fixed-excitation sector the intermediate state is outside it)
        int64_t t;
        if (B.layout == EL_LAYOUT_CHAIN || B.layout == EL_LAYOUT_RING) {
          const int64_t t1 = el::flip_target(B, code, r, bj);
          t = (t1 >= 0) ? el::flip_target(B, code ^ (1ULL << bj), t1, bi) : -1;
        } else {
          t = el::rank_any(B, code ^ ((1ULL << bi) | (1ULL << bj)));
        }
        if (t >= 0) {
          double wr, wi;
          load_amp<S, C>(psi, t, wr, wi);
          acc[q][1] += wr * re + wi * im;   // conj(v_t) v_s
          acc[q][2] += wr * im - wi * re;
        }
      }
    }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < kGroup; ++q) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double v = acc[q][c];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[warp][q * 3 + c] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < kGroup * 3) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w][threadIdx.x];
    partials[(size_t)blockIdx.x * K + (size_t)g * kGroup * 3 + threadIdx.x] = s;
  }
}

// out[k] = sum over the blocks' partials: 32 outputs per block, 8 threads
// each (a fixed order).
__global__ void __launch_bounds__(256) k_obs_sum(int nparts, int K, const double *__restrict__ partials,
                                                 double *__restrict__ out) {
  __shared__ double red[8][32];
  const int k = blockIdx.x * 32 + (threadIdx.x & 31), sh = threadIdx.x >> 5;
  double s = 0.0;
  if (k < K) {
#pragma unroll 8
    for (int b = sh; b < nparts; b += 8) s += partials[(size_t)b * K + k];
  }
  red[sh][threadIdx.x & 31] = s;
  __syncthreads();
  if (sh == 0 && k < K) {
    for (int w = 1; w < 8; ++w) s += red[w][threadIdx.x];
    out[k] = s;
  }
}

// ------------------------------------------- sites and all pairs at once
// Norm, <n_i> and <sigma-_i> of every site or, with PAIRS, <n_i n_j> and
// <sigma+_i sigma-_j> of every pair i < j, on bases of at most 32 sites (two
// launches: both sets of sums together do not fit the registers).  For
// a row u let a_k = v_{u + k} where site k can be excited from u, else 0; then
//     <sigma-_k> = sum_u conj(v_u) a_k,  <sigma+_i sigma-_j> = sum_u conj(a_i) a_j,
// so the flip targets of a row are found once for all pairs (an item per pair
// finds two per row): the pair sums are a Gram matrix of the a_k.  A CTA
// stages 256 rows (128 with PAIRS): codes and amplitudes, then the a_k (a
// thread has every 64th row and a group of 8 sites; site sums in registers,
// a_k of pairs in shared memory), then 36
// blocks of 4 x 4 sites (i-block <= j-block), each shared by 7 threads with
// their share of the rows, add their 16 pairs in FP64 registers.  Bound: instruction
// issue, most of it the FP64 multiply-adds (4 per pair and row), at 16 warps
// per SM (24-site chain: issue 46 %, FP64 pipe 35 %).  31-site chain (dim 3,524,578,
// complex64), 465 pairs: 13.7 ms with an item per pair, 2.1 here; sites
// alone 0.83 -> 0.52 ms.
constexpr int obs_rows(bool pairs) { return pairs ? 128 : 256; }   // rows per stage
constexpr int OB = 8;             // blocks of 4 sites
constexpr int OT = OB * (OB + 1) / 2;   // site-block pairs
constexpr int OSL = 256 / OT;     // threads (row shares) of a site-block pair

template <typename S, bool C, bool PAIRS>
__global__ void __launch_bounds__(256, 2) k_obs_all(BasisDev B, const S *__restrict__ psi,
                                                    double *__restrict__ partials, int K) {
  constexpr int SITES = 32, OR = obs_rows(PAIRS);
  __shared__ uint32_t code_s[OR];
  __shared__ double p_s[OR];
  __shared__ S vr_s[OR], vi_s[C ? OR : 1];
  extern __shared__ __align__(16) unsigned char obs_smem[];
  // a_k: [site][row] (re, then im), one row of padding against bank conflicts
  S *const ar = reinterpret_cast<S *>(obs_smem);
  S *const ai = ar + SITES * (OR + 1);
  const int tid = threadIdx.x, n = B.n;
  const int g = tid / 64;                              // gather role: rows tid % 64 + 64 i, sites 8 g .. 8 g + 7
  const int ti = tid / OSL, sl = tid - ti * OSL;       // Gram role: block pair, row share
  int bi = 0, bj = 0;
  if (PAIRS) {
    int q = ti;
    for (bi = 0; bi < OB && q >= OB - bi; ++bi) q -= OB - bi;
    bj = bi + q;
  }
  const bool gram = PAIRS && ti < OT;
  double sn[PAIRS ? 1 : 8], sr[PAIRS ? 1 : 8], si[PAIRS ? 1 : 8], norm = 0.0;
#pragma unroll
  for (int q = 0; q < (PAIRS ? 1 : 8); ++q) sn[q] = sr[q] = si[q] = 0.0;
  double xr[PAIRS ? 16 : 1], xi[PAIRS ? 16 : 1], nn[PAIRS ? 16 : 1];
#pragma unroll
  for (int q = 0; q < (PAIRS ? 16 : 1); ++q) xr[q] = xi[q] = nn[q] = 0.0;
  for (int64_t base = (int64_t)blockIdx.x * OR; base < B.dim; base += (int64_t)gridDim.x * OR) {
    if (tid < OR) {
      const int64_t row = base + tid;
      uint32_t c = 0;
      double re = 0.0, im = 0.0;
      if (row < B.dim) {
        c = (uint32_t)el::unrank_row(B, row);
        load_amp<S, C>(psi, row, re, im);
      }
      code_s[tid] = c;
      p_s[tid] = re * re + im * im;
      vr_s[tid] = (S)re;
      if constexpr (C) vi_s[tid] = (S)im;
    }
    __syncthreads();
#pragma unroll 1
    for (int r = tid & 63; r < OR; r += 64) {
      const uint32_t code = code_s[r];
      const int64_t row = base + r;
      const double p = p_s[r], vr = vr_s[r], vi = C ? (double)vi_s[C ? r : 0] : 0.0;
      if (g == 0) norm += p;
      S wr[8], wi[8];
      bool ok[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int k = g * 8 + q;
        wr[q] = S(0);
        wi[q] = S(0);
        ok[q] = false;
        if (k < n && row < B.dim && !((code >> k) & 1u)) {
          const int64_t t = el::flip_target(B, code, row, k);
          if (t >= 0) {
            ok[q] = true;
            if constexpr (C) { wr[q] = psi[2 * t]; wi[q] = psi[2 * t + 1]; }
            else { wr[q] = psi[t]; }
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int k = g * 8 + q;
        if constexpr (PAIRS) {
          ar[k * (OR + 1) + r] = wr[q];
          if constexpr (C) ai[k * (OR + 1) + r] = wi[q];
        } else {
          if ((code >> k) & 1u) sn[q] += p;
          if (ok[q]) {
            const double dr = wr[q], di = wi[q];
            sr[q] += vr * dr + vi * di;      // conj(v_u) a_k
            si[q] += vr * di - vi * dr;
          }
        }
      }
    }
    __syncthreads();
    if (gram) {
      for (int u = sl; u < OR; u += OSL) {
        const uint32_t code = code_s[u];
        const double p = p_s[u];
        double ir[4], ii[4], jr[4], ji[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          ir[q] = ar[(bi * 4 + q) * (OR + 1) + u];
          jr[q] = ar[(bj * 4 + q) * (OR + 1) + u];
          ii[q] = C ? (double)ai[(bi * 4 + q) * (OR + 1) + u] : 0.0;
          ji[q] = C ? (double)ai[(bj * 4 + q) * (OR + 1) + u] : 0.0;
        }
        const uint32_t mi = code >> (bi * 4), mj = code >> (bj * 4);
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) {
            xr[x * 4 + y] += ir[x] * jr[y] + ii[x] * ji[y];    // conj(a_i) a_j
            if constexpr (C) xi[x * 4 + y] += ir[x] * ji[y] - ii[x] * jr[y];
            if ((mi >> x) & (mj >> y) & 1u) nn[x * 4 + y] += p;
          }
      }
    }
    __syncthreads();
  }
  // block sums in fixed orders, through shared memory
  double *const red = reinterpret_cast<double *>(obs_smem);
  double *const out = partials + (size_t)blockIdx.x * K;
  if constexpr (!PAIRS) {
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sn[q] += __shfl_xor_sync(0xffffffffu, sn[q], o);
        sr[q] += __shfl_xor_sync(0xffffffffu, sr[q], o);
        si[q] += __shfl_xor_sync(0xffffffffu, si[q], o);
      }
    for (int o = 16; o > 0; o >>= 1) norm += __shfl_xor_sync(0xffffffffu, norm, o);
    const int warp = tid >> 5;               // warps 2 g and 2 g + 1 hold group g
    if ((tid & 31) == 0) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        red[(warp * 8 + q) * 3] = sn[q];
        red[(warp * 8 + q) * 3 + 1] = sr[q];
        red[(warp * 8 + q) * 3 + 2] = si[q];
      }
      red[192 + warp] = norm;
    }
    __syncthreads();
    if (tid == 0) out[0] = red[192] + red[193];
    for (int o = tid; o < 3 * n; o += 256) {
      const int k = o / 3, c = o - 3 * k, w = 2 * (k / 8);
      out[1 + o] = red[(w * 8 + k % 8) * 3 + c] + red[((w + 1) * 8 + k % 8) * 3 + c];
    }
  }
  if constexpr (PAIRS) {
    // [bit i][bit j] of (nn, re, im), one quantity at a time
    for (int c = 0; c < 3; ++c) {
      __syncthreads();
      if (gram) {
#pragma unroll
        for (int q = 0; q < 16; ++q) red[(size_t)tid * 16 + q] = c == 0 ? nn[q] : c == 1 ? xr[q] : xi[q];
      }
      __syncthreads();
      for (int o = tid; o < OT * 16; o += 256) {
        const int b = o / 16, q = o - 16 * b;
        double sum = 0.0;
        for (int w = 0; w < OSL; ++w) sum += red[(size_t)(b * OSL + w) * 16 + q];
        out[o * 3 + c] = sum;
      }
    }
  }
}

ObsItem item(int kind, int bi, int bj) {
  ObsItem it;
  memset(&it, 0, sizeof it);
  it.kind = kind;
  it.bi = bi;
  it.bj = bj;
  return it;
}

// Evaluate `items` (padded here to whole groups) on psi; out[3 q .. 3 q + 2]
// receives the three sums of item q.
int run_items(el_ctx *ctx, el_ham *h, int dtype, const void *psi, std::vector<ObsItem> &items,
              std::vector<double> &out) {
  while (items.size() % kGroup) items.push_back(item(kNoItem, 0, 0));
  const int ngroups = (int)(items.size() / kGroup);
  if (ngroups > 65535) return fail(ctx, EL_EINVAL, "too many observables (%zu)", items.size());
  const int K = ngroups * kGroup * 3;
  BasisDev B = el::basis_dev(h->basis);
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  int gx = el::grid_for(B.dim, 256);
  if (gx > 2 * sms) gx = 2 * sms;
  ObsItem *d_items = (ObsItem *)el::workspace(ctx, 9, items.size() * sizeof(ObsItem));
  double *d_out = (double *)el::workspace(ctx, 10, (size_t)K * sizeof(double));
  if (!d_items || !d_out) return EL_ENOMEM;
  int rc = el::ensure_partials(ctx, (size_t)gx * K);
  if (rc) return rc;
  EL_CUDA_TRY(ctx, el::copy(ctx, d_items, items.data(), items.size() * sizeof(ObsItem), cudaMemcpyHostToDevice));
  const dim3 grid(gx, ngroups);
  switch (dtype) {
    case EL_F32: k_obs_items<float, false><<<grid, 256, 0, ctx->stream>>>(B, (const float *)psi, d_items, ctx->d_partials, K); break;
    case EL_F64: k_obs_items<double, false><<<grid, 256, 0, ctx->stream>>>(B, (const double *)psi, d_items, ctx->d_partials, K); break;
    case EL_C64: k_obs_items<float, true><<<grid, 256, 0, ctx->stream>>>(B, (const float *)psi, d_items, ctx->d_partials, K); break;
    case EL_C128: k_obs_items<double, true><<<grid, 256, 0, ctx->stream>>>(B, (const double *)psi, d_items, ctx->d_partials, K); break;
    default: return fail(ctx, EL_EINVAL, "unknown dtype %d", dtype);
  }
  EL_LAUNCH_CHECK(ctx);
  k_obs_sum<<<(K + 31) / 32, 256, 0, ctx->stream>>>(gx, K, ctx->d_partials, d_out);
  EL_LAUNCH_CHECK(ctx);
  out.assign(K, 0.0);
  EL_CUDA_TRY(ctx, el::copy(ctx, out.data(), d_out, (size_t)K * sizeof(double), cudaMemcpyDeviceToHost));
  EL_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return EL_OK;
}

// Position of pair (bit i < bit j) in k_obs_all's pair sums.
int gram_slot(int i, int j) {
  const int bi = i / 4, bj = j / 4;
  int b = 0;
  for (int q = 0; q < bi; ++q) b += OB - q;
  return (b + bj - bi) * 16 + (i % 4) * 4 + j % 4;
}

template <typename S, bool C, bool PAIRS>
int launch_obs_all(el_ctx *ctx, const BasisDev &B, const void *psi, int gx, int K) {
  size_t smem = 256 * sizeof(double);      // block sums of the sites
  if (PAIRS) smem = std::max((size_t)32 * (obs_rows(true) + 1) * sizeof(S) * (C ? 2 : 1), (size_t)256 * 16 * sizeof(double));
  auto *fn = k_obs_all<S, C, PAIRS>;
  if (smem > 48 * 1024)
    EL_CUDA_TRY(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  fn<<<gx, 256, smem, ctx->stream>>>(B, (const S *)psi, ctx->d_partials, K);
  EL_LAUNCH_CHECK(ctx);
  return EL_OK;
}

template <bool PAIRS>
int launch_obs_dtype(el_ctx *ctx, const BasisDev &B, int dtype, const void *psi, int gx, int K) {
  switch (dtype) {
    case EL_F32: return launch_obs_all<float, false, PAIRS>(ctx, B, psi, gx, K);
    case EL_F64: return launch_obs_all<double, false, PAIRS>(ctx, B, psi, gx, K);
    case EL_C64: return launch_obs_all<float, true, PAIRS>(ctx, B, psi, gx, K);
    case EL_C128: return launch_obs_all<double, true, PAIRS>(ctx, B, psi, gx, K);
    default: return fail(ctx, EL_EINVAL, "unknown dtype %d", dtype);
  }
}

// out: norm, then (n, Re sm, Im sm) per bit position; or with pairs the
// (nn, Re, Im) sums of k_obs_all.
int run_all(el_ctx *ctx, el_ham *h, int dtype, const void *psi, bool pairs, std::vector<double> &out) {
  const BasisDev B = el::basis_dev(h->basis);
  const int K = pairs ? OT * 16 * 3 : 1 + 3 * B.n;
  const int64_t stages = (B.dim + obs_rows(pairs) - 1) / obs_rows(pairs);
  const int gx = (int)std::min<int64_t>(stages, 2 * (int64_t)el::sm_count(ctx));
  double *d_out = (double *)el::workspace(ctx, 10, (size_t)K * sizeof(double));
  if (!d_out) return EL_ENOMEM;
  int rc = el::ensure_partials(ctx, (size_t)gx * K);
  if (rc) return rc;
  rc = pairs ? launch_obs_dtype<true>(ctx, B, dtype, psi, gx, K) : launch_obs_dtype<false>(ctx, B, dtype, psi, gx, K);
  if (rc) return rc;
  k_obs_sum<<<(K + 31) / 32, 256, 0, ctx->stream>>>(gx, K, ctx->d_partials, d_out);
  EL_LAUNCH_CHECK(ctx);
  out.assign(K, 0.0);
  EL_CUDA_TRY(ctx, el::copy(ctx, out.data(), d_out, (size_t)K * sizeof(double), cudaMemcpyDeviceToHost));
  EL_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return EL_OK;
}

}  // namespace

extern "C" int el_spin_observables(el_ctx *ctx, el_ham *h, int dtype, const void *psi,
                                   int n_pairs, const int32_t *pi, const int32_t *pj,
                                   double *n_site, double *norm, double *sigma_minus,
                                   double *nn, double *xy) {
  if (!ctx || !h || !psi) return EL_EINVAL;
  const int n = h->n;
  if (n_pairs < 0 || (n_pairs > 0 && (!pi || !pj))) return fail(ctx, EL_EINVAL, "bad pair list");
  EL_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  // every site, and every pair when about as many are wanted as one Gram pass
  // costs (it takes the time of 36 pair items: 31-site chain, 6 groups)
  // (not the pairs of a fixed-excitation sector: the row with both sites
  // clear, from which the Gram matrix starts, is outside it)
  if (n <= 32 && (n_pairs == 0 || (n_pairs >= 36 && h->basis->kind != EL_BASIS_CHARGE))) {
    for (int p = 0; p < n_pairs; ++p)
      if (pi[p] < 0 || pj[p] < 0 || pi[p] >= n || pj[p] >= n || pi[p] == pj[p])
        return fail(ctx, EL_EINVAL, "pair %d: bad sites (%d, %d)", p, pi[p], pj[p]);
    std::vector<double> out;
    int rc = run_all(ctx, h, dtype, psi, false, out);
    if (rc) return rc;
    if (norm) *norm = out[0];
    for (int i = 0; i < n; ++i) {
      const double *o = &out[1 + 3 * (n - 1 - i)];
      if (n_site) n_site[i] = o[0];
      if (sigma_minus) { sigma_minus[2 * i] = o[1]; sigma_minus[2 * i + 1] = o[2]; }
    }
    if (n_pairs > 0) {
      rc = run_all(ctx, h, dtype, psi, true, out);
      if (rc) return rc;
    }
    for (int p = 0; p < n_pairs; ++p) {
      const int bi = n - 1 - pi[p], bj = n - 1 - pj[p];
      const double *o = &out[3 * (size_t)gram_slot(std::min(bi, bj), std::max(bi, bj))];
      if (nn) nn[p] = o[0];
      if (xy) { xy[2 * p] = o[1]; xy[2 * p + 1] = bi < bj ? o[2] : -o[2]; }   // conj(a_i) a_j
    }
    return EL_OK;
  }
  std::vector<ObsItem> items;
  items.push_back(item(kNormItem, 0, 0));
  for (int i = 0; i < n; ++i) items.push_back(item(kSiteItem, n - 1 - i, 0));
  for (int p = 0; p < n_pairs; ++p) {
    const int i = pi[p], j = pj[p];
    if (i < 0 || j < 0 || i >= n || j >= n || i == j)
      return fail(ctx, EL_EINVAL, "pair %d: bad sites (%d, %d)", p, i, j);
    items.push_back(item(kPairItem, n - 1 - i, n - 1 - j));
  }
  std::vector<double> out;
  int rc = run_items(ctx, h, dtype, psi, items, out);
  if (rc) return rc;
  if (norm) *norm = out[0];
  for (int i = 0; i < n; ++i) {
    const double *o = &out[3 * (1 + i)];
    if (n_site) n_site[i] = o[0];
    if (sigma_minus) { sigma_minus[2 * i] = o[1]; sigma_minus[2 * i + 1] = o[2]; }
  }
  for (int p = 0; p < n_pairs; ++p) {
    const double *o = &out[3 * (1 + n + p)];
    if (nn) nn[p] = o[0];
    if (xy) { xy[2 * p] = o[1]; xy[2 * p + 1] = o[2]; }
  }
  return EL_OK;
}

extern "C" int el_pauli_expect(el_ctx *ctx, el_ham *h, int dtype, const void *psi, int n_strings,
                               const int32_t *offsets, const int32_t *sites, const char *axes,
                               double *out_host) {
  if (!ctx || !h || !psi || (n_strings > 0 && (!offsets || !sites || !axes || !out_host))) return EL_EINVAL;
  if (n_strings < 0) return fail(ctx, EL_EINVAL, "n_strings must be >= 0");
  if (n_strings == 0) return EL_OK;
  EL_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int n = h->n;
  std::vector<ObsItem> items;
  for (int q = 0; q < n_strings; ++q) {
    ObsItem it = item(kPauliItem, 0, 0);
    uint64_t used = 0;
    if (offsets[q + 1] <= offsets[q]) return fail(ctx, EL_EINVAL, "Pauli string %d is empty", q);
    for (int k = offsets[q]; k < offsets[q + 1]; ++k) {
      const int site = sites[k];
      if (site < 0 || site >= n) return fail(ctx, EL_EINVAL, "Pauli string %d: site %d out of range", q, site);
      const uint64_t bit = 1ULL << (n - 1 - site);
      if (used & bit) return fail(ctx, EL_EINVAL, "Pauli string %d: site %d appears twice", q, site);
      used |= bit;
      switch (axes[k]) {
        case 'x': it.fm |= bit; break;
        case 'y': it.fm |= bit; it.ym |= bit; break;
        case 'z': it.zm |= bit; break;
        default: return fail(ctx, EL_EINVAL, "Pauli string %d: axis must be x, y or z", q);
      }
    }
    items.push_back(it);
  }
  std::vector<double> out;
  int rc = run_items(ctx, h, dtype, psi, items, out);
  if (rc) return rc;
  for (int q = 0; q < n_strings; ++q) {
    out_host[2 * q] = out[3 * q + 1];
    out_host[2 * q + 1] = out[3 * q + 2];
  }
  return EL_OK;
}
