// Householder QR in complex128 with LAPACK's zgeqr2/zung2r conventions.
//
// PyTreeNet splits a site with np.linalg.qr (LAPACK zgeqrf + zungqr) inside
// tensor_qr_decomposition(mode=KEEP) (util/tensor_splitting.py:60-107). On the
// zero-padded, rank-deficient tensors that one-site TDVP starts from, the
// orthonormal complement that Householder QR produces decides the TDVP result,
// so this follows the same published reflector convention (zlarfg: beta real,
// beta = -sign(Re alpha) * ||(alpha, x)||, tau = (beta - alpha) / beta,
// v = x / (alpha - beta); H = I - tau v v^H applied as H^H during the
// factorisation and as H when Q is formed). Exact zeros stay exact zeros, so
// the complement is reproduced exactly.
//
// The matrix is addressed in place inside the site tensor: element (i, c) at
// A[rowoff[i] + c * colstride], where the row-offset table carries the
// reference's (logical) row order. Where the columns fit the chip's shared memory
// the whole QR is one cooperative launch; a matrix of at most 2048 rows past that
// takes one launch per reflector, a taller one a short sequence of launches (column
// norm, reflector, column dots, dot reduction, trailing update).
#include <type_traits>

#include "ptn_common.cuh"

namespace {

constexpr int QT = 256;          // threads per CTA
constexpr int RB = 1024;         // rows per row-chunk
constexpr int CB = 8;            // columns per column-chunk (one warp each)

struct QRWork {
  // device layout of the work buffer
  double2* tau;       // [k]
  double2* scal;      // [k]
  double2* w;         // [k]
  double* npart;      // [nrb]
  double2* dpart;     // [nrb * k]
};

inline int64_t nrb_for(int64_t m) { return (m + RB - 1) / RB; }

inline QRWork carve(void* work, int64_t m, int64_t k) {
  QRWork q;
  char* p = static_cast<char*>(work);
  q.tau = reinterpret_cast<double2*>(p);
  p += 16 * k;
  q.scal = reinterpret_cast<double2*>(p);
  p += 16 * k;
  q.w = reinterpret_cast<double2*>(p);
  p += 16 * k;
  q.npart = reinterpret_cast<double*>(p);
  p += 16 * ((nrb_for(m) + 1) / 2 + 1);
  q.dpart = reinterpret_cast<double2*>(p);
  return q;
}

__device__ __forceinline__ double2 ld(const double2* A, const int64_t* rowoff, int64_t cs,
                                      int64_t i, int64_t c) {
  return A[rowoff[i] + c * cs];
}

// partial[b] = sum_{i in chunk b, i > j} |A[i, j]|^2
__global__ void __launch_bounds__(QT) colnorm_kernel(const double2* __restrict__ A,
                                                     const int64_t* __restrict__ rowoff, int64_t cs,
                                                     int64_t m, int64_t j, double* __restrict__ part) {
  const int64_t r0 = (j + 1) + (int64_t)blockIdx.x * RB;
  double acc = 0.0;
  for (int64_t i = r0 + threadIdx.x; i < m && i < r0 + RB; i += QT) acc += cabs2(ld(A, rowoff, cs, i, j));
  __shared__ double red[QT / 32];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < QT / 32; ++i) s += red[i];
    part[blockIdx.x] = s;
  }
}

// One thread: zlarfg on (A[j, j], A[j+1:, j]).
__global__ void reflector_kernel(double2* __restrict__ A, const int64_t* __restrict__ rowoff, int64_t cs,
                                 int64_t j, const double* __restrict__ part, int nparts,
                                 double2* __restrict__ tau, double2* __restrict__ scal) {
  if (threadIdx.x != 0) return;
  double s = 0.0;
  for (int b = 0; b < nparts; ++b) s += part[b];
  const double xnorm = sqrt(s);
  double2* pa = A + rowoff[j] + j * cs;
  const double2 alpha = *pa;
  if (xnorm == 0.0 && alpha.y == 0.0) {
    tau[j] = make_double2(0.0, 0.0);
    scal[j] = make_double2(0.0, 0.0);
    return;
  }
  double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm * xnorm);
  const double beta = (alpha.x >= 0.0) ? -nrm : nrm;
  tau[j] = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
  // scal = 1 / (alpha - beta)
  double2 d = make_double2(alpha.x - beta, alpha.y);
  double den = d.x * d.x + d.y * d.y;
  scal[j] = make_double2(d.x / den, -d.y / den);
  *pa = make_double2(beta, 0.0);
}

// Reflector component v_i (v_j = 1).
__device__ __forceinline__ double2 vcomp(const double2* A, const int64_t* rowoff, int64_t cs, int64_t i,
                                         int64_t j, double2 sc, bool stored) {
  if (i == j) return make_double2(1.0, 0.0);
  double2 a = ld(A, rowoff, cs, i, j);
  return stored ? a : cmul(a, sc);
}

// dpart[rb * k + c] = sum_{i in chunk rb, i >= j} conj(v_i) X[i, c], for c in [c_lo, k)
// grid: (row chunks, column chunks of CB); one warp per column.
// stored != 0: column j already holds v (Q formation); else v = scal * A[:, j].
__global__ void __launch_bounds__(QT) dots_kernel(const double2* __restrict__ A,
                                                  const int64_t* __restrict__ rowoff, int64_t cs,
                                                  int64_t m, int64_t k, int64_t j, int64_t c_lo,
                                                  const double2* __restrict__ scal, int stored,
                                                  double2* __restrict__ dpart) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t c = c_lo + (int64_t)blockIdx.y * CB + warp;
  const int64_t r0 = j + (int64_t)blockIdx.x * RB;
  const double2 sc = scal[j];
  __shared__ double2 vs[RB];
  for (int64_t t = threadIdx.x; t < RB; t += QT) {
    int64_t i = r0 + t;
    vs[t] = (i < m) ? vcomp(A, rowoff, cs, i, j, sc, stored != 0) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  if (c >= k) return;
  double2 acc = make_double2(0.0, 0.0);
  for (int64_t t = lane; t < RB; t += 32) {
    int64_t i = r0 + t;
    if (i >= m) break;
    acc = cfmac(vs[t], ld(A, rowoff, cs, i, c), acc);
  }
  acc = warp_sum2(acc);
  if (lane == 0) dpart[(int64_t)blockIdx.x * k + c] = acc;
}

__global__ void dots_finish_kernel(const double2* __restrict__ dpart, int nrb, int64_t k, int64_t c_lo,
                                   double2* __restrict__ w) {
  const int64_t c = c_lo + blockIdx.x;
  double2 s = make_double2(0.0, 0.0);
  for (int b = threadIdx.x; b < nrb; b += 32) s = cadd(s, dpart[(int64_t)b * k + c]);
  s = warp_sum2(s);
  if (threadIdx.x == 0) w[c] = s;
}

// X[i, c] -= f * v_i * w_c for i >= j, c in [c_lo, k); f = conj(tau) (factorisation)
// or tau (Q formation).
__global__ void __launch_bounds__(QT) update_kernel(double2* __restrict__ A,
                                                    const int64_t* __restrict__ rowoff, int64_t cs,
                                                    int64_t m, int64_t k, int64_t j, int64_t c_lo,
                                                    const double2* __restrict__ tau,
                                                    const double2* __restrict__ scal,
                                                    const double2* __restrict__ w, int stored,
                                                    int conj_tau) {
  const int64_t r0 = j + (int64_t)blockIdx.x * RB;
  const int64_t cbase = c_lo + (int64_t)blockIdx.y * CB;
  double2 f = tau[j];
  if (conj_tau) f.y = -f.y;
  const double2 sc = scal[j];
  for (int64_t t = threadIdx.x; t < RB; t += QT) {
    int64_t i = r0 + t;
    if (i >= m) break;
    double2 v = vcomp(A, rowoff, cs, i, j, sc, stored != 0);
    double2 fv = cmul(f, v);
    const int64_t ro = rowoff[i];
    for (int cc = 0; cc < CB; ++cc) {
      int64_t c = cbase + cc;
      if (c >= k) break;
      double2* p = A + ro + c * cs;
      *p = csub(*p, cmul(fv, w[c]));
    }
  }
}

// After the trailing update of step j: A[i, j] <- scal * A[i, j] (the stored v_i), i > j.
__global__ void __launch_bounds__(QT) store_v_kernel(double2* __restrict__ A, const int64_t* __restrict__ rowoff,
                                                     int64_t cs, int64_t m, int64_t j,
                                                     const double2* __restrict__ scal) {
  const double2 sc = scal[j];
  for (int64_t i = j + 1 + blockIdx.x * (int64_t)QT + threadIdx.x; i < m; i += (int64_t)gridDim.x * QT) {
    double2* p = A + rowoff[i] + j * cs;
    *p = cmul(*p, sc);
  }
}

// Copy the upper triangle of rows < p into R (k x k row-major), zero elsewhere.
__global__ void extract_r_kernel(const double2* __restrict__ A, const int64_t* __restrict__ rowoff,
                                 int64_t cs, int64_t k, int64_t p, double2* __restrict__ R) {
  for (int64_t e = blockIdx.x * (int64_t)QT + threadIdx.x; e < k * k; e += (int64_t)gridDim.x * QT) {
    int64_t r = e / k, c = e - r * k;
    R[e] = (r < p && c >= r) ? ld(A, rowoff, cs, r, c) : make_double2(0.0, 0.0);
  }
}

// Column j of Q: Q[j, j] = 1 - tau, Q[i > j, j] = -tau v_i, Q[i < j, j] = 0.
__global__ void __launch_bounds__(QT) qcol_kernel(double2* __restrict__ A, const int64_t* __restrict__ rowoff,
                                                  int64_t cs, int64_t m, int64_t j,
                                                  const double2* __restrict__ tau) {
  const double2 t = tau[j];
  for (int64_t i = blockIdx.x * (int64_t)QT + threadIdx.x; i < m; i += (int64_t)gridDim.x * QT) {
    double2* p = A + rowoff[i] + j * cs;
    if (i < j) *p = make_double2(0.0, 0.0);
    else if (i == j) *p = make_double2(1.0 - t.x, -t.y);
    else *p = make_double2(-(t.x * p->x - t.y * p->y), -(t.x * p->y + t.y * p->x));
  }
}

// KEEP padding: zero the columns p..k-1 of Q.
__global__ void zero_cols_kernel(double2* __restrict__ A, const int64_t* __restrict__ rowoff, int64_t cs,
                                 int64_t m, int64_t k, int64_t p) {
  const int64_t nc = k - p;
  for (int64_t e = blockIdx.x * (int64_t)QT + threadIdx.x; e < m * nc; e += (int64_t)gridDim.x * QT) {
    int64_t i = e / nc, c = p + (e - (e / nc) * nc);
    A[rowoff[i] + c * cs] = make_double2(0.0, 0.0);
  }
}

// ---- small m (at most QR_SMALL_M rows) --------------------------------------------------
// Two forms of the same arithmetic: a launch sequence (one kernel per Householder
// step) and, below, one cooperative launch. Both give the same bits: rows r, r +
// HT, ... belong to thread r mod HT, a thread adds its rows in ascending order, the
// lanes of a warp and then the four warps are added by a butterfly, and all
// scalars come from the functions here. A reflector is kept unscaled: x = the
// column below row j, s = 1 / (alpha - beta), v = (1, s x), so that
//   v^H c = conj(s) x^H c + c_j,   H c = c - tau (v^H c) (1, s x),
// which takes the scaling of v off the chain of dependent steps.
//
// What bounds a step on GB300 is the FP64 pipe and its latency: a warp
// instruction holds a scheduler's FP64 unit for 64 cycles whatever the active
// lanes. Hence four warps (one per scheduler) with several rows per thread, FMA
// forms (4 per row of a dot product, 6 per row of an update), and sums of both parts of
// all of a CTA's columns reduced together.
constexpr int64_t QR_SMALL_M = 2048;
constexpr int ST = 256;
constexpr int HT = 128;                  // threads of the small-m kernels
constexpr int HW = HT / 32;

// c - x g, rounded once at the size of c: an entry goes through k of these, and a
// second rounding (two FMAs onto c, an instruction less per part) shows in the
// factors' error, |Q R - A| / |A| of 512 x 256 1.04e-15 in place of 7.8e-16. Costs 9 %
// there (1.75 and 1.91 ms).
__device__ __forceinline__ double2 csub_mul(double2 c, double2 x, double2 g) {
  const double px = fma(x.x, g.x, -x.y * g.y), py = fma(x.x, g.y, x.y * g.x);
  c.x -= px;
  c.y -= py;
  return c;
}

// zlarfg on (alpha, x) with |x|^2 = xn2: tau, s = 1 / (alpha - beta), beta and
// nb = -1 / beta.
struct Reflector {
  double2 tau, s, beta;
  double nb;
};
// Squared norms whose reciprocal may leave the range, and those that are not numbers.
__device__ __noinline__ Reflector make_reflector_far(double2 alpha, double n2) {
  Reflector h;
  const double nrm = sqrt(n2), beta = alpha.x >= 0.0 ? -nrm : nrm;
  h.beta = make_double2(beta, 0.0);
  h.nb = -1.0 / beta;
  h.tau = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
  const double dx = alpha.x - beta, den = dx * dx + alpha.y * alpha.y;
  h.s = make_double2(dx / den, -alpha.y / den);
  return h;
}
__device__ __forceinline__ Reflector make_reflector(double2 alpha, double xn2) {
  Reflector h;
  if (xn2 == 0.0 && alpha.y == 0.0) {
    h.tau = make_double2(0.0, 0.0);
    h.s = make_double2(0.0, 0.0);
    h.beta = alpha;
    h.nb = 0.0;
    return h;
  }
  const double a2 = fma(alpha.x, alpha.x, alpha.y * alpha.y), n2 = a2 + xn2;
  if (!(n2 > 1e-290 && n2 < 1e290)) return make_reflector_far(alpha, n2);
  const bool pos = alpha.x >= 0.0;                   // beta = -sign(Re alpha) |(alpha, x)|
  // one reciprocal square root for beta and 1 / beta, one correction for each
  const double rn = rsqrt(n2), r0 = n2 * rn;
  const double nrm = fma(fma(-r0, r0, n2), 0.5 * rn, r0);
  const double ri = fma(fma(-nrm, rn, 1.0), rn, rn);
  h.beta = make_double2(pos ? -nrm : nrm, 0.0);
  h.nb = pos ? ri : -ri;
  h.tau = make_double2(fma(alpha.x, h.nb, 1.0), alpha.y * h.nb);  // (beta - alpha) / beta
  const double dx = alpha.x - h.beta.x, rd = __drcp_rn(fma(dx, dx, alpha.y * alpha.y));
  h.s = make_double2(dx * rd, -alpha.y * rd);
  return h;
}

// f and g = s f of the update c_j - f, c_r - x_r g for a column with x^H c = d:
// f = t (conj(s) d + c_j), t = conj(tau) in the factorisation and tau when Q is
// formed. With conj(tau) conj(s) = tau s = nb one product is real. Even lanes form
// the real parts, odd lanes the imaginary ones (five FP64 instructions instead
// of twelve).
template <bool FACTOR>
__device__ __forceinline__ void reflect(double2 tau, double2 s, double nb, double2 d, double2 cj, double& f,
                                        double& g) {
  const bool im = threadIdx.x & 1;
  const double dm = im ? d.y : d.x, cm = im ? cj.y : cj.x;
  if (FACTOR) {
    f = fma(tau.x, cm, fma(tau.y, im ? -cj.x : cj.y, nb * dm));
    const double o = __shfl_xor_sync(0xffffffffu, f, 1);
    g = fma(s.x, f, s.y * (im ? o : -o));
  } else {
    const double w = fma(s.x, dm, fma(s.y, im ? -d.x : d.y, cm));
    const double o = __shfl_xor_sync(0xffffffffu, w, 1);
    f = fma(tau.x, w, tau.y * (im ? o : -o));
    g = nb * w;
  }
}
__device__ __forceinline__ double2 pair_from(double v, int lane0) {
  return make_double2(__shfl_sync(0xffffffffu, v, lane0), __shfl_sync(0xffffffffu, v, lane0 + 1));
}

// CTA sums of 2 NC values (Re, Im of NC columns): partials in red[warp][value]
// first, then, after the barrier, every lane gets value lane & (2 NC - 1)...
// NC = 1 or 2.
template <int NC>
__device__ __forceinline__ void cta_partials(const double2 (&v)[NC], double (*red)[4]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (NC == 1) {
    const bool up = lane & 16;
    double t = (up ? v[0].y : v[0].x) + __shfl_xor_sync(0xffffffffu, up ? v[0].x : v[0].y, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((lane & 15) == 0) red[warp][lane >> 4] = t;
  } else {
    const bool up = lane & 16, hi = lane & 8;
    const double2 keep = up ? v[NC - 1] : v[0], send = up ? v[0] : v[NC - 1];
    const double a = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 16);
    const double b = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 16);
    double t = (hi ? b : a) + __shfl_xor_sync(0xffffffffu, hi ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((lane & 7) == 0) red[warp][lane >> 3] = t;
  }
}
template <int NC>
__device__ __forceinline__ void cta_totals(double2 (&v)[NC], double (*red)[4]) {
  // lane = warp index (2 bits) + 4 * value
  const int lane = threadIdx.x & 31, val = (lane >> 2) & (2 * NC - 1);
  double t = red[lane & 3][val];
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    v[i].x = __shfl_sync(0xffffffffu, t, 8 * i);
    v[i].y = __shfl_sync(0xffffffffu, t, 8 * i + 4);
  }
}
// one real value, the same tree
__device__ __forceinline__ double cta_total1(double v, double (*red)[4]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][0] = v;
  __syncthreads();
  double t = red[threadIdx.x & 3][0];
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  return __shfl_sync(0xffffffffu, t, 0);
}

// First row above j of this thread.
__device__ __forceinline__ int64_t first_row(int64_t j) {
  const int64_t r = (j + 1) / HT * HT + threadIdx.x;
  return r > j ? r : r + HT;
}

// Step j of the factorisation. grid = max(1, k - j - 1); CTA b owns column j + 1 + b and
// forms the reflector from column j itself (a few KB, the same bits in every
// CTA). Reflectors go to V (unscaled) and tau / s, the diagonal of R to betas.
__global__ void __launch_bounds__(HT) hh_fact_small(double2* __restrict__ A, const int64_t* __restrict__ rowoff,
                                                    int64_t cs, int64_t m, int64_t k, int64_t j,
                                                    double2* __restrict__ tau, double2* __restrict__ scal,
                                                    double2* __restrict__ V, double2* __restrict__ R) {
  __shared__ double red[2][HW][4];
  const int tid = threadIdx.x;
  double acc = 0.0;
  for (int64_t r = first_row(j); r < m; r += HT) {
    const double2 a = A[rowoff[r] + j * cs];
    acc = fma(a.x, a.x, fma(a.y, a.y, acc));
    if (blockIdx.x == 0) V[j * m + r] = a;
  }
  const double xn2 = cta_total1(acc, red[0]);
  const double2 alpha = A[rowoff[j] + j * cs];
  const Reflector h = make_reflector(alpha, xn2);
  if (blockIdx.x == 0 && tid == 0) {
    tau[j] = h.tau;
    scal[j] = h.s;
    V[j * m + j] = make_double2(h.beta.x, h.nb);
    R[j * k + j] = h.beta;
  }
  const int64_t c = j + 1 + blockIdx.x;
  if (c >= k) return;
  double2 d[1] = {make_double2(0.0, 0.0)};
  for (int64_t r = first_row(j); r < m; r += HT) d[0] = cfmac(A[rowoff[r] + j * cs], A[rowoff[r] + c * cs], d[0]);
  cta_partials<1>(d, red[1]);
  __syncthreads();
  cta_totals<1>(d, red[1]);
  double2* pj = A + rowoff[j] + c * cs;
  const double2 cj = *pj;
  __syncthreads();                                   // everyone has read c_j
  double fl, gl;
  reflect<true>(h.tau, h.s, h.nb, d[0], cj, fl, gl);
  const double2 f = pair_from(fl, 0), g = pair_from(gl, 0);
  if (tid == j % HT) *pj = csub(cj, f);
  for (int64_t r = first_row(j); r < m; r += HT) {
    double2* q = A + rowoff[r] + c * cs;
    *q = csub_mul(*q, A[rowoff[r] + j * cs], g);
  }
}

// R[r][c]: strictly-upper part from A (rows < p), zero elsewhere; the steps have
// written the diagonal.
__global__ void extract_r_small(const double2* __restrict__ A, const int64_t* __restrict__ rowoff, int64_t cs,
                                int64_t k, int64_t p, double2* __restrict__ R) {
  for (int64_t e = blockIdx.x * (int64_t)ST + threadIdx.x; e < k * k; e += (int64_t)gridDim.x * ST) {
    const int64_t r = e / k, c = e - r * k;
    double2 v = make_double2(0.0, 0.0);
    if (r < p && c == r) continue;
    if (r < p && c > r) v = A[rowoff[r] + c * cs];
    R[e] = v;
  }
}

// Column c of H_c e_c: 1 - tau at row c, -(tau s) x = -nb x below.
__device__ __forceinline__ double2 start_entry(int64_t r, int64_t c, double2 tau, double nb, double2 x) {
  if (r < c) return make_double2(0.0, 0.0);
  if (r == c) return make_double2(1.0 - tau.x, -tau.y);
  return cscale(x, -nb);
}

// Step j of forming Q (zung2r): CTAs 0..ncols-1 apply H_j to columns j+1..p-1,
// CTA ncols writes column j itself.
__global__ void __launch_bounds__(HT) hh_form_small(double2* __restrict__ A, const int64_t* __restrict__ rowoff,
                                                    int64_t cs, int64_t m, int64_t p, int64_t j,
                                                    const double2* __restrict__ tau,
                                                    const double2* __restrict__ scal,
                                                    const double2* __restrict__ V) {
  __shared__ double red[HW][4];
  const int64_t ncols = p - (j + 1);
  const double2 t_ = tau[j], s_ = scal[j];
  const double2* x = V + j * m;
  if (blockIdx.x == ncols) {
    for (int64_t r = threadIdx.x; r < m; r += HT)
      A[rowoff[r] + j * cs] = start_entry(r, j, t_, x[j].y, r > j ? x[r] : make_double2(0.0, 0.0));
    return;
  }
  const int64_t c = j + 1 + blockIdx.x;
  double2 d[1] = {make_double2(0.0, 0.0)};
  for (int64_t r = first_row(j); r < m; r += HT) d[0] = cfmac(x[r], A[rowoff[r] + c * cs], d[0]);
  cta_partials<1>(d, red);
  __syncthreads();
  cta_totals<1>(d, red);
  double2* pj = A + rowoff[j] + c * cs;
  const double2 cj = *pj;
  __syncthreads();
  double fl, gl;
  reflect<false>(t_, s_, x[j].y, d[0], cj, fl, gl);
  const double2 f = pair_from(fl, 0), g = pair_from(gl, 0);
  if (threadIdx.x == j % HT) *pj = csub(cj, f);
  for (int64_t r = first_row(j); r < m; r += HT) {
    double2* q = A + rowoff[r] + c * cs;
    *q = csub_mul(*q, x[r], g);
  }
}

inline unsigned grid1(int64_t n) {
  int64_t b = (n + QT - 1) / QT;
  if (b < 1) b = 1;
  if (b > 2048) b = 2048;
  return (unsigned)b;
}

// ---- small m, one cooperative launch ---------------------------------------------------
// CTA b owns a few columns (snake order, so the Q formation work -- column c needs
// c + 1 reflectors -- is balanced) and keeps them in shared memory, each thread
// its own rows. Reflector j is published by the owner of column j as soon as that
// column has received reflectors 0 .. j-1: first the entries of x, each thread its
// rows as it updates them, then, when the norm is known, tau and s. The buffers
// start out filled with a NaN that no result can be, and readers poll the entries
// they need: no flags and no fences, and the dot products with x run while the
// owner still forms the scalars. The owner of column j + 1 updates that column
// first. Chain per step: scalars - L2 - update - norm - scalars.
// What bounds it is that chain (the arithmetic of 512 x 256 is 0.2 ms of the FP64
// pipe): 4 us a step in the factorisation, of which norm, reflector and the two
// barriers about 1.6, and 2.7 us a reflector when Q is formed. Two columns per CTA
// rather than one: half as many readers of each x, one reduction for both.
// Measured against flags with fences, 256 threads and scaled reflectors:
// 512 x 256 3.28 -> 1.91 ms, 256 x 128 1.36 -> 0.68, 128 x 64 0.62 -> 0.30,
// 16 x 8 0.083 -> 0.047, 2048 x 128 3.38 -> 3.02.
constexpr long long HP_WAIT_CYCLES = 4000000000LL;   // ~2 s at 2 GHz
constexpr unsigned long long HP_EMPTY = ~0ull;

struct HPArgs {
  double2* A;
  const int64_t* rowoff;
  int64_t cs, m, k, p;
  double2* tau;
  double2* scal;
  double2* V;
  double2* R;
  int* status;    // nonzero: a wait ran out (every CTA stops)
  int G;          // CTAs
  int cpc;        // columns per CTA (upper bound)
};

// i-th column of CTA b (increasing in i)
__device__ __forceinline__ int64_t hp_col(int b, int i, int G) {
  return (int64_t)i * G + ((i & 1) ? (G - 1 - b) : b);
}
__device__ __forceinline__ int hp_owner(int64_t c, int G) {
  const int64_t i = c / G, r = c - i * G;
  return (int)((i & 1) ? (G - 1 - r) : r);
}

__device__ __forceinline__ void hp_put(double2* p, double2 v) {
  // an input NaN may have any payload: not the empty one
  unsigned long long a = (unsigned long long)__double_as_longlong(v.x), b = (unsigned long long)__double_as_longlong(v.y);
  if (a == HP_EMPTY) a = 0x7ff8000000000000ull;
  if (b == HP_EMPTY) b = 0x7ff8000000000000ull;
  asm volatile("st.volatile.global.v2.u64 [%0], {%1,%2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ bool hp_try(const double2* p, double2& v) {
  unsigned long long a, b;
  asm volatile("ld.volatile.global.v2.u64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
  v = make_double2(__longlong_as_double((long long)a), __longlong_as_double((long long)b));
  return a != HP_EMPTY && b != HP_EMPTY;
}

// This thread's rows below j of x_j, once published. False when the kernel must leave.
template <int PF>
__device__ __forceinline__ bool hp_wait_x(const HPArgs& a, int64_t j, double2 (&x)[PF]) {
  const double2* v = a.V + j * a.m;
  const long long t0 = clock64();
  for (unsigned it = 1;; ++it) {
    bool ok = true;
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      const int64_t r = threadIdx.x + (int64_t)q * HT;
      x[q] = make_double2(0.0, 0.0);
      if (r > j && r < a.m) ok = hp_try(v + r, x[q]) && ok;
    }
    if (__all_sync(0xffffffffu, ok)) return true;
    int stop = 0;
    if ((it & 255u) == 0u && *(volatile int*)a.status != 0) stop = 1;
    if (clock64() - t0 > HP_WAIT_CYCLES) {
      atomicExch(a.status, PTN_ERR_TIMEOUT);
      stop = 1;
    }
    if (__any_sync(0xffffffffu, stop)) return false;
  }
}
// tau, s and (beta, nb) of step j; `ready` says that they have been read already.
__device__ __forceinline__ bool hp_try_scalars(const HPArgs& a, int64_t j, double2 (&sc)[3]) {
  return hp_try(a.tau + j, sc[0]) & hp_try(a.scal + j, sc[1]) & hp_try(a.V + j * a.m + j, sc[2]);
}
__device__ __forceinline__ bool hp_wait_scalars(const HPArgs& a, int64_t j, double2 (&sc)[3], bool ready) {
  const long long t0 = clock64();
  for (unsigned it = 1;; ++it) {
    const bool ok = ready || hp_try_scalars(a, j, sc);
    if (__all_sync(0xffffffffu, ok)) return true;
    ready = false;
    int stop = 0;
    if ((it & 255u) == 0u && *(volatile int*)a.status != 0) stop = 1;
    if (clock64() - t0 > HP_WAIT_CYCLES) {
      atomicExch(a.status, PTN_ERR_TIMEOUT);
      stop = 1;
    }
    if (__any_sync(0xffffffffu, stop)) return false;
  }
}

using Yes = std::true_type;
using No = std::false_type;

// PF: rows per thread (HT PF >= m).
template <int PF>
__global__ void __launch_bounds__(HT) hh_persistent_kernel(const HPArgs a) {
  extern __shared__ double2 hsm[];           // [cpc][m] own columns
  __shared__ double red[2][HW][4];
  __shared__ double nred[HW][4];
  __shared__ double2 head[2][2];             // c_j of the two columns in work
  __shared__ int s_fail;
  const int b = blockIdx.x, tid = threadIdx.x, G = a.G;
  const int64_t m = a.m, k = a.k, p = a.p, cs = a.cs;
  int nown = 0;
  while (nown < a.cpc && hp_col(b, nown, G) < k) ++nown;
  for (int i = 0; i < nown; ++i) {
    const int64_t c = hp_col(b, i, G);
    for (int64_t r = tid; r < m; r += HT) hsm[i * m + r] = a.A[a.rowoff[r] + c * cs];
  }
  if (tid == 0) s_fail = 0;
  unsigned par = 0;                          // alternates the shared buffers of the sums
  __syncthreads();

  // norm, scalars and diagonal of column j (own slot col), whose entries are published
  auto publish_scalars = [&](int64_t j, double2* col) {
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      const int64_t r = tid + (int64_t)q * HT;
      if (r > j && r < m) acc = fma(col[r].x, col[r].x, fma(col[r].y, col[r].y, acc));
    }
    // the sum's barrier also makes alpha (thread j mod HT's row) visible
    const double xn2 = cta_total1(acc, nred);
    if (tid < 32) {
      const Reflector h = make_reflector(col[j], xn2);
      if (tid == 0) {
        hp_put(a.tau + j, h.tau);
        hp_put(a.scal + j, h.s);
        hp_put(a.V + j * m + j, make_double2(h.beta.x, h.nb));
        a.R[j * k + j] = h.beta;
      }
    }
    __syncthreads();                         // nred is free again
  };
  auto publish_x = [&](int64_t j, const double2* col) {
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      const int64_t r = tid + (int64_t)q * HT;
      if (r > j && r < m) hp_put(a.V + j * m + r, col[r]);
    }
  };

  // one reflector on one or two own columns
  auto apply = [&](auto factor, int64_t j, const double2 (&x)[PF], double2* c0, double2* c1, auto after) -> bool {
    double2 sc[3];
    const bool early = hp_try_scalars(a, j, sc);     // under way during the dot products
    double2 d[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      const int64_t r = tid + (int64_t)q * HT;
      if (r > j && r < m) {
        d[0] = cfmac(x[q], c0[r], d[0]);
        if (c1) d[1] = cfmac(x[q], c1[r], d[1]);
      }
      if (r == j) {
        head[par][0] = c0[r];
        if (c1) head[par][1] = c1[r];
      }
    }
    cta_partials<2>(d, red[par]);
    if (!hp_wait_scalars(a, j, sc, early)) s_fail = 1;
    __syncthreads();
    if (s_fail) return false;
    cta_totals<2>(d, red[par]);
    // lanes of the upper half work for the second column
    const bool second = (tid & 16) != 0;
    double f, g;
    reflect<decltype(factor)::value>(sc[0], sc[1], sc[2].y, second ? d[1] : d[0], head[par][second ? 1 : 0], f, g);
    const double2 f0 = pair_from(f, 0), g0 = pair_from(g, 0), f1 = pair_from(f, 16), g1 = pair_from(g, 16);
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      const int64_t r = tid + (int64_t)q * HT;
      if (r > j && r < m) c0[r] = csub_mul(c0[r], x[q], g0);
      if (r == j) c0[r] = csub(c0[r], f0);
    }
    after();                                 // the first column is done
    if (c1) {
#pragma unroll
      for (int q = 0; q < PF; ++q) {
        const int64_t r = tid + (int64_t)q * HT;
        if (r > j && r < m) c1[r] = csub_mul(c1[r], x[q], g1);
        if (r == j) c1[r] = csub(c1[r], f1);
      }
    }
    par ^= 1u;
    return true;
  };

  double2 x[PF];
  if (p > 0 && hp_owner(0, G) == b) {        // column 0 is this CTA's slot 0
    publish_x(0, hsm);
    publish_scalars(0, hsm);
  }
  bool ok = true;
  for (int64_t j = 0; j < p && ok; ++j) {
    int i0 = 0;                              // own columns above j: slots i0 ..
    while (i0 < nown && hp_col(b, i0, G) <= j) ++i0;
    if (i0 == nown) break;
    if (!hp_wait_x<PF>(a, j, x)) s_fail = 1; // seen by all at the next barrier
    for (int i = i0; i < nown && ok; i += 2) {
      double2* c0 = hsm + (int64_t)i * m;
      const bool next = i == i0 && hp_col(b, i, G) == j + 1 && j + 1 < p;
      ok = apply(Yes{}, j, x, c0, i + 1 < nown ? c0 + m : nullptr, [&]() {
        if (next) {
          publish_x(j + 1, c0);
          publish_scalars(j + 1, c0);
        }
      });
    }
  }
  if (!ok) {
    if (tid == 0) a.R[0] = make_double2(NAN, NAN);   // the result is not usable
    return;
  }
  __syncthreads();
  // R above the diagonal and its zeros (rows < p: the diagonal is written with the
  // scalars), then Q (zung2r: column c = H_0 ... H_c e_c), KEEP padding past p
  for (int i = 0; i < nown; ++i) {
    const int64_t c = hp_col(b, i, G);
    const double2* col = hsm + (int64_t)i * m;
    for (int64_t r = tid; r < k; r += HT)
      if (!(r == c && r < p)) a.R[r * k + c] = (r < p && c > r) ? col[r] : make_double2(0.0, 0.0);
  }
  // column c starts from its own reflector, still in its slot
  for (int i = 0; i < nown; ++i) {
    const int64_t c = hp_col(b, i, G);
    double2* col = hsm + (int64_t)i * m;
    if (c < p) {
      double2 sc[3];
      if (!hp_wait_scalars(a, c, sc, false)) s_fail = 1;
      for (int64_t r = tid; r < m; r += HT) col[r] = start_entry(r, c, sc[0], sc[2].y, col[r]);
    } else {
      for (int64_t r = tid; r < m; r += HT) col[r] = make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  ok = s_fail == 0;
  __syncthreads();
  // reflectors from the highest column down, on pairs of own columns (the later
  // column of a pair alone until the earlier one's turn comes); each x is
  // fetched while the one before it is applied
  for (int i = 0; i < nown && ok; i += 2) {
    const int64_t ca = hp_col(b, i, G), cb = i + 1 < nown ? hp_col(b, i + 1, G) : -1;
    double2* pa = hsm + (int64_t)i * m;
    double2* pb = pa + m;
    const int64_t la = ca < p ? ca : 0, lb = cb >= 0 && cb < p ? cb : 0;   // reflectors still to apply
    double2 nx[PF];
    const int64_t top = la > lb ? la : lb;
    if (top > 0 && !hp_wait_x<PF>(a, top - 1, nx)) s_fail = 1;
    for (int64_t j = top - 1; j >= 0 && ok; --j) {
#pragma unroll
      for (int q = 0; q < PF; ++q) x[q] = nx[q];
      if (j > 0) {
        const double2* v = a.V + (j - 1) * m;        // published long ago
#pragma unroll
        for (int q = 0; q < PF; ++q) {
          const int64_t r = tid + (int64_t)q * HT;
          nx[q] = (r >= j && r < m) ? __ldcg(v + r) : make_double2(0.0, 0.0);
        }
      }
      if (j < la) ok = apply(No{}, j, x, pa, j < lb ? pb : nullptr, []() {});
      else ok = apply(No{}, j, x, pb, nullptr, []() {});
    }
  }
  if (!ok) {
    if (tid == 0) a.R[0] = make_double2(NAN, NAN);
    return;
  }
  for (int i = 0; i < nown; ++i) {
    const int64_t c = hp_col(b, i, G);
    for (int64_t r = tid; r < m; r += HT) a.A[a.rowoff[r] + c * cs] = hsm[(int64_t)i * m + r];
  }
}

const void* hp_kernel(int64_t m) {
  const int64_t pf = (m + HT - 1) / HT;
  if (pf <= 1) return (const void*)hh_persistent_kernel<1>;
  if (pf <= 2) return (const void*)hh_persistent_kernel<2>;
  if (pf <= 4) return (const void*)hh_persistent_kernel<4>;
  if (pf <= 8) return (const void*)hh_persistent_kernel<8>;
  return (const void*)hh_persistent_kernel<16>;
}

}  // namespace

extern "C" int64_t ptn_zqr_work_bytes(int64_t m, int64_t k) {
  if (m <= QR_SMALL_M) {
    const int64_t p = m < k ? m : k;
    return 16 * (2 * k + m * p) + 4 * (p + 1) + 512;   // tau, s, V, status
  }
  return 16 * (3 * k + (nrb_for(m) + 1) / 2 + 1 + nrb_for(m) * k) + 256;
}

// Launch shape of the one-launch path for an m x k problem (m <= QR_SMALL_M):
// CTAs, columns per CTA and dynamic shared memory; false when it does not fit
// (columns too many for shared memory, or more CTAs than can be co-resident).
static bool hp_shape(int64_t m, int64_t k, int& G, int& cpc, size_t& smem) {
  // device properties and the kernel's shared-memory limit: once per process
  // (thread-safe static initialisation; the engine drives one device)
  struct Dev {
    int n_sm = 0;
    size_t dyn_max = 0;
  };
  static const Dev dv = []() {
    Dev d;
    int dev = 0;
    cudaDeviceProp pr;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaGetDeviceProperties(&pr, dev) != cudaSuccess ||
        !pr.cooperativeLaunch)
      return d;
    const size_t dyn = pr.sharedMemPerBlockOptin - 1024;    // room for the static shared memory
    for (int64_t rows = HT; rows <= QR_SMALL_M; rows *= 2)
      if (cudaFuncSetAttribute(hp_kernel(rows), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn) != cudaSuccess)
        return d;
    d.n_sm = pr.multiProcessorCount;
    d.dyn_max = dyn;
    return d;
  }();
  if (dv.n_sm <= 0 || m < 1 || k < 1 || m > QR_SMALL_M) return false;
  int64_t g = (k + 1) / 2;                           // two columns per CTA
  if (g > dv.n_sm) g = dv.n_sm;
  const int64_t c = (k + g - 1) / g;
  const size_t bytes = (size_t)c * (size_t)m * sizeof(double2);
  if (bytes > dv.dyn_max) return false;
  int max_per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&max_per_sm, hp_kernel(m), HT, bytes) != cudaSuccess ||
      (int64_t)max_per_sm * dv.n_sm < g)
    return false;
  G = (int)g;
  cpc = (int)c;
  smem = bytes;
  return true;
}

extern "C" int ptn_zqr_path(int64_t m, int64_t k) {
  int G, cpc;
  size_t smem;
  if (m <= QR_SMALL_M && hp_shape(m, k, G, cpc, smem)) return 1;
  return 0;
}

static int zqr_keep_persistent(double2* A, const int64_t* rowoff, int64_t m, int64_t k, int64_t cs, double2* R,
                               void* work, cudaStream_t s) {
  int G, cpc;
  size_t smem;
  if (!hp_shape(m, k, G, cpc, smem)) return PTN_ERR_UNSUPPORTED;
  const int64_t p = m < k ? m : k;
  HPArgs a;
  a.A = A;
  a.rowoff = rowoff;
  a.cs = cs;
  a.m = m;
  a.k = k;
  a.p = p;
  a.tau = static_cast<double2*>(work);
  a.scal = a.tau + k;
  a.V = a.scal + k;
  a.status = reinterpret_cast<int*>(a.V + m * p);
  a.R = R;
  a.G = G;
  a.cpc = cpc;
  // every entry empty
  if (cudaMemsetAsync(a.tau, 0xff, sizeof(double2) * (size_t)(2 * k + m * p), s) != cudaSuccess ||
      cudaMemsetAsync(a.status, 0, sizeof(int), s) != cudaSuccess)
    return PTN_ERR_LAUNCH;
  void* args[] = {&a};
  PTN_COUNT(1);
  if (cudaLaunchCooperativeKernel(hp_kernel(m), dim3((unsigned)G), dim3(HT), args, smem, s) != cudaSuccess)
    return PTN_ERR_LAUNCH;
  return ptn_launch_status();
}

static int zqr_keep_small(double2* A, const int64_t* rowoff, int64_t m, int64_t k, int64_t cs, double2* R,
                          void* work, cudaStream_t s) {
  double2* tau = static_cast<double2*>(work);
  double2* scal = tau + k;
  double2* V = scal + k;
  const int64_t p = m < k ? m : k;
  for (int64_t j = 0; j < p; ++j) {
    const int64_t ncols = k - (j + 1);
    PTN_COUNT(1);
    hh_fact_small<<<(unsigned)(ncols > 0 ? ncols : 1), HT, 0, s>>>(A, rowoff, cs, m, k, j, tau, scal, V, R);
  }
  PTN_COUNT(1);
  extract_r_small<<<grid1(k * k), ST, 0, s>>>(A, rowoff, cs, k, p, R);
  for (int64_t j = p - 1; j >= 0; --j) {
    PTN_COUNT(1);
    hh_form_small<<<(unsigned)(p - j), HT, 0, s>>>(A, rowoff, cs, m, p, j, tau, scal, V);
  }
  if (p < k) { PTN_COUNT(1); zero_cols_kernel<<<grid1(m * (k - p)), QT, 0, s>>>(A, rowoff, cs, m, k, p); }
  return ptn_launch_status();
}

// Q[j, j] = 1 for j in [lo, hi): the columns that Householder steps with an
// exactly-zero remaining column (tau = 0) leave as unit vectors.
__global__ void unit_diag_kernel(double2* __restrict__ A, const int64_t* __restrict__ rowoff, int64_t cs,
                                 int64_t lo, int64_t hi) {
  const int64_t j = lo + blockIdx.x * (int64_t)QT + threadIdx.x;
  if (j < hi) A[rowoff[j] + j * cs] = make_double2(1.0, -0.0);
}

static int zqr_keep_impl(double2* A, const int64_t* rowoff, int64_t m_path, int64_t m, int64_t k, int64_t cs,
                         double2* R, void* work, cudaStream_t s);

extern "C" int ptn_zqr_keep(void* Av, const int64_t* rowoff, int64_t m, int64_t k, int64_t cs, void* Rv,
                            void* work, void* stream) {
  if (!Av || !rowoff || !Rv || !work || m < 1 || k < 1 || cs < 1) return PTN_ERR_ARG;
  return zqr_keep_impl(static_cast<double2*>(Av), rowoff, m, m, k, cs, static_cast<double2*>(Rv), work,
                       ptn_stream(stream));
}

extern "C" int ptn_zqr_keep_steps(void* Av, const int64_t* rowoff, int64_t m, int64_t k, int64_t cs, void* Rv,
                                  void* work, void* stream) {
  if (!Av || !rowoff || !Rv || !work || m < 1 || k < 1 || cs < 1) return PTN_ERR_ARG;
  if (m > QR_SMALL_M)
    return zqr_keep_impl(static_cast<double2*>(Av), rowoff, m, m, k, cs, static_cast<double2*>(Rv), work,
                         ptn_stream(stream));
  return zqr_keep_small(static_cast<double2*>(Av), rowoff, m, k, cs, static_cast<double2*>(Rv), work,
                        ptn_stream(stream));
}

extern "C" int ptn_zqr_keep_rows(void* Av, const int64_t* rowoff, int64_t m, int64_t m_used, int64_t k, int64_t cs,
                                 void* Rv, void* work, void* stream) {
  if (!Av || !rowoff || !Rv || !work || m < 1 || k < 1 || cs < 1 || m_used < 1 || m_used > m) return PTN_ERR_ARG;
  cudaStream_t s = ptn_stream(stream);
  double2* A = static_cast<double2*>(Av);
  int st = zqr_keep_impl(A, rowoff, m, m_used, k, cs, static_cast<double2*>(Rv), work, s);
  if (st != PTN_OK) return st;
  // Rows m_used.. are zero, so every step j >= m_used of the full factorisation
  // meets a zero column (tau = 0, beta = 0): R keeps zero rows there and Q the
  // unit vector e_j in column j (up to min(m, k)); columns past min(m, k) stay
  // zero (KEEP padding), as the call on m_used rows already left them.
  const int64_t hi = m < k ? m : k;
  if (m_used < hi) {
    PTN_COUNT(1);
    unit_diag_kernel<<<(unsigned)((hi - m_used + QT - 1) / QT), QT, 0, s>>>(A, rowoff, cs, m_used, hi);
  }
  return ptn_launch_status();
}

// Householder QR of the first m rows, with the kernel sequence (and so the
// rounding) of an m_path-row problem.
static int zqr_keep_impl(double2* A, const int64_t* rowoff, int64_t m_path, int64_t m, int64_t k, int64_t cs,
                         double2* R, void* work, cudaStream_t s) {
  if (m_path <= QR_SMALL_M) {
    const int st = zqr_keep_persistent(A, rowoff, m, k, cs, R, work, s);
    if (st != PTN_ERR_UNSUPPORTED) return st;
    return zqr_keep_small(A, rowoff, m, k, cs, R, work, s);
  }
  QRWork q = carve(work, m, k);
  const int64_t p = m < k ? m : k;
  // factorisation
  for (int64_t j = 0; j < p; ++j) {
    const int64_t below = m - (j + 1);
    const int nb_norm = below > 0 ? (int)((below + RB - 1) / RB) : 0;
    if (nb_norm > 0) { PTN_COUNT(1); colnorm_kernel<<<nb_norm, QT, 0, s>>>(A, rowoff, cs, m, j, q.npart); }
    PTN_COUNT(1);
    reflector_kernel<<<1, 32, 0, s>>>(A, rowoff, cs, j, q.npart, nb_norm, q.tau, q.scal);
    const int64_t ncols = k - (j + 1);
    if (ncols > 0) {
      const int nrb = (int)((m - j + RB - 1) / RB);
      dim3 g(nrb, (unsigned)((ncols + CB - 1) / CB));
      PTN_COUNT(1);
      dots_kernel<<<g, QT, 0, s>>>(A, rowoff, cs, m, k, j, j + 1, q.scal, 0, q.dpart);
      PTN_COUNT(1);
      dots_finish_kernel<<<(unsigned)ncols, 32, 0, s>>>(q.dpart, nrb, k, j + 1, q.w);
      PTN_COUNT(1);
      update_kernel<<<g, QT, 0, s>>>(A, rowoff, cs, m, k, j, j + 1, q.tau, q.scal, q.w, 0, 1);
    }
    if (below > 0) { PTN_COUNT(1); store_v_kernel<<<grid1(below), QT, 0, s>>>(A, rowoff, cs, m, j, q.scal); }
  }
  PTN_COUNT(1);
  extract_r_kernel<<<grid1(k * k), QT, 0, s>>>(A, rowoff, cs, k, p, R);
  // Q formation (zung2r): columns p-1 .. 0
  for (int64_t j = p - 1; j >= 0; --j) {
    const int64_t ncols = p - (j + 1);
    if (ncols > 0) {
      const int nrb = (int)((m - j + RB - 1) / RB);
      dim3 g(nrb, (unsigned)((ncols + CB - 1) / CB));
      PTN_COUNT(1);
      dots_kernel<<<g, QT, 0, s>>>(A, rowoff, cs, m, p, j, j + 1, q.scal, 1, q.dpart);
      PTN_COUNT(1);
      dots_finish_kernel<<<(unsigned)ncols, 32, 0, s>>>(q.dpart, nrb, p, j + 1, q.w);
      PTN_COUNT(1);
      update_kernel<<<g, QT, 0, s>>>(A, rowoff, cs, m, p, j, j + 1, q.tau, q.scal, q.w, 1, 0);
    }
    PTN_COUNT(1);
    qcol_kernel<<<grid1(m), QT, 0, s>>>(A, rowoff, cs, m, j, q.tau);
  }
  if (p < k) { PTN_COUNT(1); zero_cols_kernel<<<grid1(m * (k - p)), QT, 0, s>>>(A, rowoff, cs, m, k, p); }
  return ptn_launch_status();
}

// ---- QR with a library-owned scratch area --------------------------------------------
// Some callers cannot allocate device memory at the moment they need a QR: a
// host framework that binds this library through a plain C FFI and owns no
// CUDA allocator, or code that must not allocate while a stream is being
// captured into a graph. ptn_zqr_keep_noalloc runs the same Householder
// kernels as ptn_zqr_keep but takes its scratch from a fixed array compiled
// into the library (every GPU that loads the library keeps these 4 MiB until
// the process exits).
#include <mutex>

#define PTN_QR_STATIC_SCRATCH_BYTES (4ll << 20)
static __device__ __align__(256) unsigned char g_qr_static_scratch[PTN_QR_STATIC_SCRATCH_BYTES];

namespace {
std::mutex g_qr_static_mu;
void* g_qr_static_ptr[256] = {};  // device address of the array, per device ordinal
}  // namespace

extern "C" int64_t ptn_zqr_noalloc_max_bytes(void) { return PTN_QR_STATIC_SCRATCH_BYTES; }

extern "C" int ptn_zqr_keep_noalloc(void* A, const int64_t* rowoff, int64_t m, int64_t k, int64_t colstride,
                                    void* R, void* stream) {
  if (!A || !rowoff || !R || m < 1 || k < 1 || colstride < 1) return PTN_ERR_ARG;
  if (ptn_zqr_work_bytes(m, k) > PTN_QR_STATIC_SCRATCH_BYTES) return PTN_ERR_UNSUPPORTED;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return PTN_ERR_LAUNCH;
  void* work = nullptr;
  {
    std::lock_guard<std::mutex> guard(g_qr_static_mu);
    if (!g_qr_static_ptr[dev]) {
      // Host code cannot pass the array's name to a kernel: it is a host-side
      // stand-in. Resolve its device address once, with this device current.
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_qr_static_scratch) != cudaSuccess || !p) return PTN_ERR_LAUNCH;
      g_qr_static_ptr[dev] = p;
    }
    work = g_qr_static_ptr[dev];
  }
  // Every scratch entry the kernels read is written earlier in the same call
  // (column-norm partials, reflector scalars, dot partials), so nothing needs
  // clearing between calls.
  return ptn_zqr_keep(A, rowoff, m, k, colstride, R, work, stream);
}
