// Native executor for contraction chains and Krylov steps.
//
// A plan (a chain of strided contractions, or of tensor-core GEMMs with their
// operand conversions) is a fixed list of descriptors whose operand pointers
// are only known when the plan runs (the Krylov vector in and out, workspace
// slots that may have moved). ptn_exec_ops patches those pointers from a small
// table and issues every launch from C++, so a host language pays one foreign
// call per matvec instead of one per kernel. ptn_krylov_gs_step does the same
// for the vector work of one Lanczos/Arnoldi step, and ptn_krylov_batch for a
// whole batch of steps with the host's decisions where they are little work, which
// took longer in the host language than the GPU's work on vectors of a few thousand
// entries (an eigendecomposition of the m x m projection per step).
#include <algorithm>
#include <cmath>
#include <complex>

#include "ptn_common.cuh"

extern "C" int ptn_exec_ops(const ptn_exec_op* ops, int32_t nops, void* const* ptrs, int32_t nptrs,
                            void* stream) {
  if (!ops || nops < 0 || (nops > 0 && (!ptrs || nptrs < 1))) return PTN_ERR_ARG;
  for (int32_t i = 0; i < nops; ++i) {
    const ptn_exec_op& op = ops[i];
    if (!op.desc || op.a < 0 || op.a >= nptrs || op.b < -1 || op.b >= nptrs || op.c < 0 || op.c >= nptrs ||
        op.d < -1 || op.d >= nptrs)
      return PTN_ERR_ARG;
    int st;
    switch (op.kind) {
      case PTN_OP_ZCONTRACT: {
        ptn_contract_desc d = *static_cast<const ptn_contract_desc*>(op.desc);
        d.A = ptrs[op.a];
        d.B = op.b >= 0 ? ptrs[op.b] : nullptr;
        d.C = ptrs[op.c];
        st = ptn_zcontract(&d, stream);
        break;
      }
      case PTN_OP_ZCONTRACT_WS: {
        ptn_contract_desc d = *static_cast<const ptn_contract_desc*>(op.desc);
        d.A = ptrs[op.a];
        d.B = op.b >= 0 ? ptrs[op.b] : nullptr;
        d.C = ptrs[op.c];
        void* work = op.d >= 0 ? ptrs[op.d] : nullptr;
        st = ptn_zcontract_ws(&d, work, work ? ptn_zcontract_work_bytes(&d) : 0, stream);
        break;
      }
      case PTN_OP_CGEMM: {
        ptn_cgemm_desc d = *static_cast<const ptn_cgemm_desc*>(op.desc);
        d.A = ptrs[op.a];
        d.Bx = op.b >= 0 ? ptrs[op.b] : nullptr;
        d.C = ptrs[op.c];
        if (op.d >= 0) d.partial = ptrs[op.d];
        st = ptn_cgemm_bf16x3(&d, stream);
        break;
      }
      case PTN_OP_TO_PLANES:
      case PTN_OP_EXPAND_B: {
        ptn_convert_desc d = *static_cast<const ptn_convert_desc*>(op.desc);
        d.src = ptrs[op.a];
        d.dst = ptrs[op.c];
        st = op.kind == PTN_OP_TO_PLANES ? ptn_to_planes(&d, stream) : ptn_expand_b(&d, stream);
        break;
      }
      default:
        return PTN_ERR_ARG;
    }
    if (st != PTN_OK) return st;
  }
  return PTN_OK;
}

int ptn_gs_step_passes(const void* Q, int64_t ldq, int32_t nq, void* w, int64_t n, void* h, void* partial,
                       double* norms, void* qnext, void* stream);

extern "C" int ptn_krylov_gs_step(const void* Q, int64_t ldq, int32_t nq, void* w, int64_t n, void* h,
                                  void* partial, double* norms, void* qnext, void* stream) {
  if (!Q || !w || !h || !partial || !norms || nq < 1 || n < 1 || ldq < n) return PTN_ERR_ARG;
  int st = ptn_gs_step_passes(Q, ldq, nq, w, n, h, partial, norms, qnext, stream);
  if (st != PTN_ERR_UNSUPPORTED) return st;
  st = ptn_dznrm2(w, n, norms, partial, stream);
  if (st != PTN_OK) return st;
  double2* h1 = static_cast<double2*>(h);
  double2* h2 = h1 + nq;
  for (double2* hp : {h1, h2}) {
    st = ptn_zdot_multi(Q, ldq, nq, w, n, hp, 0, partial, stream);
    if (st != PTN_OK) return st;
    st = ptn_zaxpy_multi(Q, ldq, nq, hp, w, n, stream);
    if (st != PTN_OK) return st;
  }
  st = ptn_dznrm2(w, n, norms + 1, partial, stream);
  if (st != PTN_OK) return st;
  if (qnext) st = ptn_zscal_inv(w, norms + 1, qnext, n, stream);
  return st;
}

namespace {

using cd = std::complex<double>;

// exp(z H) e_1 for the Hermitian m x m projection H (the symmetrised T, or its real
// tridiagonal part) where that is little work: a Taylor series over steps with
// |z H|_1 <= 1 each, whose terms fall below 1e-18 after about 20. False, and nothing
// written, for more than TAYLOR_WORK steps times m^2, where an eigendecomposition, which
// does not depend on the norm, is the better one: the caller has it. (All columns of a
// solve on a CPU: 25 vectors at |z H| = 10 1.9 ms of series and 1.2 of eigendecompositions,
// 64 at 50 121 and 11 ms, 64 at 500 1.2 s and 11 ms; a site update of a time step has 5 to
// 9 vectors at 1 and below.) Also for a norm that is not a number.
constexpr int TAYLOR_MAX_M = 32;
constexpr double TAYLOR_WORK = 1024.0;
bool projected_column(const cd* T, int64_t ldt, int m, bool tridiagonal, cd z, cd* col) {
  if (m > TAYLOR_MAX_M) return false;
  cd H[TAYLOR_MAX_M * TAYLOR_MAX_M], term[TAYLOR_MAX_M], next[TAYLOR_MAX_M];
  for (int i = 0; i < m; ++i)
    for (int j = 0; j < m; ++j) {
      if (!tridiagonal)
        H[i * m + j] = 0.5 * (T[i * ldt + j] + std::conj(T[j * ldt + i]));
      else if (i == j)
        H[i * m + j] = T[i * ldt + i].real();
      else if (i == j + 1)
        H[i * m + j] = T[i * ldt + j].real();
      else if (j == i + 1)
        H[i * m + j] = T[j * ldt + i].real();
      else
        H[i * m + j] = cd(0.0, 0.0);
    }
  double norm = 0.0;
  for (int j = 0; j < m; ++j) {
    double c = 0.0;
    for (int i = 0; i < m; ++i) c += std::abs(H[i * m + j]);
    if (!(c <= norm)) norm = c;
  }
  double steps = std::ceil(norm * std::abs(z));
  if (steps < 1.0) steps = 1.0;
  if (!(steps * m * m <= TAYLOR_WORK)) return false;
  const cd zs = z / steps;
  std::fill(col, col + m, cd(0.0, 0.0));
  col[0] = 1.0;
  for (int s = 0; s < (int)steps; ++s) {
    std::copy(col, col + m, term);
    for (int k = 1; k < 200; ++k) {
      double size = 0.0, total = 0.0;
      const cd f = zs / (double)k;
      for (int i = 0; i < m; ++i) {
        double re = 0.0, im = 0.0;
        for (int j = 0; j < m; ++j) {
          const cd a = H[i * m + j], b = term[j];
          re += a.real() * b.real() - a.imag() * b.imag();
          im += a.real() * b.imag() + a.imag() * b.real();
        }
        next[i] = cd(re * f.real() - im * f.imag(), re * f.imag() + im * f.real());
        col[i] += next[i];
        size = std::max(size, std::max(std::fabs(next[i].real()), std::fabs(next[i].imag())));
        total = std::max(total, std::max(std::fabs(col[i].real()), std::fabs(col[i].imag())));
      }
      std::copy(next, next + m, term);
      if (!(size > 1e-18 * total)) break;
    }
  }
  return true;
}

struct Coefficients {
  double2 c[64];
};

__global__ void __launch_bounds__(256) zcombine_arg_kernel(const double2* __restrict__ Q, int64_t n, int m,
                                                           const Coefficients k, double2* __restrict__ out, int add) {
  for (int64_t x = blockIdx.x * 256ll + threadIdx.x; x < n; x += gridDim.x * 256ll) {
    double2 v = add ? out[x] : make_double2(0.0, 0.0);
    for (int i = 0; i < m; ++i) v = cfma(k.c[i], Q[(int64_t)i * n + x], v);
    out[x] = v;
  }
}

}  // namespace

extern "C" int ptn_krylov_batch(ptn_krylov_desc* d, void* stream) {
  if (!d || !d->ops || !d->ptrs || d->nptrs < 2 || !d->Q || !d->w || !d->h || !d->norms || !d->partial ||
      !d->h_host || !d->norms_host || !d->T || !d->coef || d->n < 1 || d->j0 < 0 || d->batch < 1 ||
      d->j0 + d->batch > d->qcap || d->ldt < (int64_t)d->j0 + d->batch + 1 || (d->j0 == 0 && !d->x) ||
      (d->status && !d->status_host))
    return PTN_ERR_ARG;
  cudaStream_t s = ptn_stream(stream);
  const int64_t n = d->n;
  const int J = d->j0 + d->batch;
  double2* Q = static_cast<double2*>(d->Q);
  double2* h = static_cast<double2*>(d->h);
  double* nr = static_cast<double*>(d->norms);
  int st;
  if (d->j0 == 0) {
    if ((st = ptn_dznrm2(d->x, n, nr, d->partial, stream)) != PTN_OK) return st;
    if ((st = ptn_zscal_inv(d->x, nr, Q, n, stream)) != PTN_OK) return st;
  }
  for (int j = d->j0; j < J; ++j) {
    d->ptrs[0] = Q + (int64_t)j * n;
    d->ptrs[1] = d->w;
    if ((st = ptn_exec_ops(d->ops, d->nops, d->ptrs, d->nptrs, stream)) != PTN_OK) return st;
    // step j's coefficients start at entry j (j + 1): those before it have 2 (i + 1) each
    void* qnext = j + 1 < d->qcap ? Q + (int64_t)(j + 1) * n : nullptr;
    if ((st = ptn_krylov_gs_step(Q, n, j + 1, d->w, n, h + (int64_t)j * (j + 1), d->partial, nr + 1 + 2 * j, qnext,
                                 stream)) != PTN_OK)
      return st;
  }
  const int64_t h0 = (int64_t)d->j0 * (d->j0 + 1), h1 = (int64_t)J * (J + 1);
  const int64_t n0 = d->j0 == 0 ? 0 : 1 + 2 * d->j0;
  cd* hh = static_cast<cd*>(d->h_host);
  if (cudaMemcpyAsync(hh + h0, h + h0, (size_t)(h1 - h0) * sizeof(double2), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaMemcpyAsync(d->norms_host + n0, nr + n0, (size_t)(1 + 2 * J - n0) * sizeof(double), cudaMemcpyDeviceToHost,
                      s) != cudaSuccess ||
      (d->status && cudaMemcpyAsync(d->status_host, d->status, sizeof(int32_t), cudaMemcpyDeviceToHost, s) !=
                        cudaSuccess) ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return PTN_ERR_LAUNCH;
  d->done = d->have = 0;
  d->open = -1;
  d->m = d->j0;
  if (d->status && *d->status_host != 0) return PTN_OK;      // the caller reports it
  if (d->j0 == 0) d->beta0 = d->norms_host[0];
  const double beta0 = d->beta0;
  if (beta0 == 0.0) {
    d->m = 0;
    d->done = 1;
    return PTN_OK;
  }
  cd* T = static_cast<cd*>(d->T);
  cd* coef = static_cast<cd*>(d->coef);
  const cd z(d->z_re, d->z_im);
  const double floor_abs = 2.220446049250313e-16 * (double)n;
  for (int j = d->j0; j < J && !d->done; ++j) {
    const cd* c = hh + (int64_t)j * (j + 1);
    const double w0 = d->norms_host[1 + 2 * j], beta = d->norms_host[2 + 2 * j];
    for (int i = 0; i <= j; ++i) T[i * d->ldt + j] = c[i] + c[j + 1 + i];
    T[(j + 1) * d->ldt + j] = beta;
    if (d->open >= 0) continue;                      // the caller decides from there on
    d->m = j + 1;
    d->have = 0;
    if (!std::isfinite(beta) || std::isnan(w0)) return PTN_ERR_NONFINITE;
    if (beta <= std::max(floor_abs, 1e-12 * w0)) {
      d->done = 1;
    } else if (d->tol > 0.0) {
      d->have = projected_column(T, d->ldt, d->m, d->tridiagonal != 0, z, coef);
      if (!d->have) {
        d->open = j;
        continue;
      }
      if (beta0 * beta * std::abs(coef[d->m - 1]) < d->tol) d->done = 1;
    }
    if (j + 1 >= d->qcap) d->done = 1;
  }
  if (d->open < 0 && d->done && !d->have) d->have = projected_column(T, d->ldt, d->m, d->tridiagonal != 0, z, coef);
  if (d->have)
    for (int i = 0; i < d->m; ++i) coef[i] *= beta0;
  return PTN_OK;
}

extern "C" int ptn_krylov_combine(const void* Q, int64_t n, int32_t m, const void* coef_host, void* out,
                                  void* stream) {
  if (!Q || !coef_host || !out || n < 1 || m < 1) return PTN_ERR_ARG;
  const double2* c = static_cast<const double2*>(coef_host);
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  // the coefficients travel as a kernel argument: no copy to the device
  for (int i0 = 0; i0 < m; i0 += 64) {
    const int cnt = m - i0 < 64 ? m - i0 : 64;
    Coefficients k;
    for (int i = 0; i < 64; ++i) k.c[i] = i < cnt ? c[i0 + i] : make_double2(0.0, 0.0);
    PTN_COUNT(1);
    zcombine_arg_kernel<<<(unsigned)blocks, 256, 0, ptn_stream(stream)>>>(
        static_cast<const double2*>(Q) + (int64_t)i0 * n, n, cnt, k, static_cast<double2*>(out), i0 > 0);
  }
  return ptn_launch_status();
}
