// Index groups of a strided contraction on the device, shared by the FP64
// kernels (zcontract.cu) and the tensor-core ones (zcontract_tc.cu).
#pragma once
#include "ptn_common.cuh"

struct ModeDev {
  int n;
  int64_t dim[PTN_MAX_MODES];
  int64_t s0[PTN_MAX_MODES];
  int64_t s1[PTN_MAX_MODES];
};

struct ContractArgs {
  const double2* A;
  const double2* B;
  double2* C;
  double2 alpha, beta;
  int conj_a, conj_b;
  int beta_zero;
  int64_t M, N, K;
  int64_t tiles_n;
  int64_t k_chunk;  // K indices per split (the whole K when not split)
  int split;        // accumulate with atomics into a pre-scaled C
  ModeDev m, n, k;  // m: (A, C) strides; n: (B, C); k: (A, B)
};

// Offsets of a group index in both operands. Indices below 2^31 (all but the
// largest tensors) divide in 32 bits: a 64-bit division is a call of ~70
// instructions, and several of them in a row were most of a small kernel's
// time. The slowest mode needs no division.
__device__ __forceinline__ void decode(const ModeDev& md, int64_t idx, int64_t& o0, int64_t& o1) {
  o0 = 0;
  o1 = 0;
  if (idx < 0x7fffffffll) {
    uint32_t i = (uint32_t)idx;
    for (int d = md.n - 1; d > 0; --d) {
      const int64_t dd = md.dim[d];
      const uint32_t w = dd < 0x80000000ll ? (uint32_t)dd : 0x80000000u;
      const uint32_t q = i / w, r = i - q * w;
      o0 += r * md.s0[d];
      o1 += r * md.s1[d];
      i = q;
    }
    if (md.n > 0) {
      o0 += i * md.s0[0];
      o1 += i * md.s1[0];
    }
    return;
  }
  for (int d = md.n - 1; d >= 0; --d) {
    int64_t dd = md.dim[d];
    int64_t q = idx / dd;
    int64_t r = idx - q * dd;
    o0 += r * md.s0[d];
    o1 += r * md.s1[d];
    idx = q;
  }
}

static inline int fill_modes(const ptn_modes& src, ModeDev& dst, int which, int64_t& total) {
  // which: 0 -> (a, c) strides, 1 -> (b, c), 2 -> (a, b)
  if (src.n < 0 || src.n > PTN_MAX_MODES) return PTN_ERR_ARG;
  dst.n = src.n;
  total = 1;
  for (int i = 0; i < src.n; ++i) {
    if (src.dim[i] <= 0) return PTN_ERR_ARG;
    dst.dim[i] = src.dim[i];
    total *= src.dim[i];
    switch (which) {
      case 0: dst.s0[i] = src.stride_a[i]; dst.s1[i] = src.stride_c[i]; break;
      case 1: dst.s0[i] = src.stride_b[i]; dst.s1[i] = src.stride_c[i]; break;
      default: dst.s0[i] = src.stride_a[i]; dst.s1[i] = src.stride_b[i]; break;
    }
  }
  return PTN_OK;
}

// The arguments of a descriptor in device form (modes, pointers, factors);
// tiles_n, k_chunk and split are the launcher's.
static inline int zcontract_args(const ptn_contract_desc& d, ContractArgs& a) {
  if (fill_modes(d.m, a.m, 0, a.M) || fill_modes(d.n, a.n, 1, a.N) || fill_modes(d.k, a.k, 2, a.K))
    return PTN_ERR_ARG;
  a.A = static_cast<const double2*>(d.A);
  a.B = static_cast<const double2*>(d.B);
  a.C = static_cast<double2*>(d.C);
  a.alpha = make_double2(d.alpha_re, d.alpha_im);
  a.beta = make_double2(d.beta_re, d.beta_im);
  a.beta_zero = (d.beta_re == 0.0 && d.beta_im == 0.0);
  a.conj_a = d.conj_a;
  a.conj_b = d.conj_b;
  return PTN_OK;
}
