// Declarations shared by the H-apply kernels (el_apply.cu, el_chain.cu).
#pragma once

#include "el_internal.cuh"

namespace el {

template <typename S>
struct HamArgs {
  const S *diagV;
  S delta[EL_MAX_SITES];
  S up_re[EL_MAX_SITES];  // amplitude into a row whose bit k is 1: Omega/2
  S up_im[EL_MAX_SITES];  // (into a row whose bit k is 0: conj(Omega)/2)
  const ExPair *px;       // exchange channels (generic and hop kernels)
  int npx;
  int lossy;              // loss diagonal present (generic and hop kernels)
  int real_amp;           // every sigma^x amplitude is real: cheaper complex multiply-adds
  S loss[EL_MAX_SITES];   // imaginary diagonal per set bit: -gamma/2 (evolution units)
};

struct KArgs {
  int64_t nvec;
  int lognv;
  const void *x;
  const void *z;
  void *y;
  void *acc;
  double a, b, c, w_re, w_im;
  const double *c_dev;    // if not null: c from the device (written by an earlier launch)
  double *dots;
  int want;
  int skip_diag;
  const void *probe;
  double *partials;
  unsigned int *counter;
};

__device__ __forceinline__ double coef_c(const KArgs &K) { return K.c_dev ? *K.c_dev : K.c; }

template <typename S>
inline HamArgs<S> ham_args(const el_ham *h, const S *diagV) {
  HamArgs<S> A;
  memset(&A, 0, sizeof A);
  A.diagV = diagV;
  A.px = h->d_px;
  A.npx = (int)h->px.size();
  A.lossy = h->lossy ? 1 : 0;
  A.real_amp = h->drive_complex ? 0 : 1;
  for (int k = 0; k < h->n; ++k) {
    A.delta[k] = (S)h->delta[k];
    A.up_re[k] = (S)(0.5 * h->om_re[k]);
    A.up_im[k] = (S)(0.5 * h->om_im[k]);
    A.loss[k] = (S)h->loss[k];
  }
  return A;
}

// y = a H x + b x + c z (+ acc, dots) on CHAIN and RING sectors (el_chain.cu).
bool chain_block_ok(const el_ctx *ctx, const el_ham *h, const ApplyArgs &A);
int launch_chain_block(el_ctx *ctx, el_ham *h, const ApplyArgs &A, const BasisDev &B, const KArgs &K);

// The same on the full 2^n basis (el_full.cu).
bool full_block_ok(const el_ham *h, const ApplyArgs &A);
int launch_full_block(el_ctx *ctx, el_ham *h, const ApplyArgs &A, const KArgs &K);
// The same on blockade sectors of a graph (el_table.cu).
bool table_block_ok(const el_ham *h, const ApplyArgs &A);
int launch_table_block(el_ctx *ctx, el_ham *h, const ApplyArgs &A, const BasisDev &B, const KArgs &K);

}  // namespace el
