// Singular value decomposition (complex128, FP64) by one-sided Jacobi
// (Hestenes), and a strided permute/conjugate/scale copy.
//
// ptn_zsvd_jacobi factors an m x n matrix (m >= n) as A = U diag(S) V^H with S
// sorted in descending order. One-sided Jacobi orthogonalises the columns of a
// working copy of A by plane rotations applied from the right; V accumulates
// the rotations. A sweep visits every column pair once in the round-robin
// (circle) order: n_even - 1 rounds of n_even / 2 disjoint pairs, one warp per
// pair. Matrices of 8 columns and up to 512 rows run as a ring of CTAs that pass
// columns to their neighbours (zsvd_ring_kernel); fewer columns in one CTA;
// taller ones with rounds separated by a grid-wide barrier. Kernels whose CTAs
// wait on one another are launched cooperatively, so all CTAs are resident. A pair (a, b) is rotated when
// |a^H b| > tol * |a| |b| (tol = 8 sqrt(m) * 2^-53); the
// iteration stops after the first sweep without a rotation. Every barrier wait
// is bounded: on timeout the kernel records PTN_ERR_TIMEOUT in *status and all
// CTAs leave. A sweep limit that is reached records PTN_ERR_NOCONVERGE (the
// outputs are still written).
//
// The reference computes this step with np.linalg.svd (LAPACK gesdd) inside
// tensor_svd / truncated_tensor_svd (util/tensor_splitting.py:122-177, 488-527).
#include <mutex>

#include "ptn_common.cuh"
#include "coop.cuh"

namespace {

constexpr int SVD_WARPS = 4;
constexpr int SVD_THREADS = SVD_WARPS * 32;
constexpr int SVD_MAX_SWEEPS = 56;
constexpr long long SVD_WAIT_CYCLES = 4000000000LL;  // ~2 s at 2 GHz
constexpr int CTRL_WORDS = 64;                       // barrier words + per-sweep rotation counts
constexpr int64_t CTRL_BYTES = 256;

struct SvdArgs {
  const double2* src;
  int64_t rs, cs;
  int64_t m, n;
  double2* Aw;   // m x n column-major working copy
  double2* Vw;   // n x n column-major accumulated rotations
  double* sig;   // n column norms
  unsigned* ctrl;
  double2* U;
  int64_t ldu;
  double* S;
  double2* V;
  int64_t ldv;
  double tol;
  int32_t* status;
};

__device__ __forceinline__ double2 ldcg2(const double2* p) { return __ldcg(p); }
__device__ __forceinline__ void stcg2(double2* p, double2 v) { __stcg(p, v); }

// Grid-wide barrier (coop.cuh); a timeout is also recorded in *status.
__device__ bool grid_barrier(unsigned* ctrl, int32_t* status) {
  const bool ok = ptn_grid_barrier(ctrl, SVD_WAIT_CYCLES);
  if (!ok && threadIdx.x == 0 && *((volatile unsigned*)(ctrl + 2)) != 0u) atomicCAS(status, 0, PTN_ERR_TIMEOUT);
  return ok;
}

// Rotate columns i and j of Aw (and of Vw) so that they become orthogonal.
// Columns whose squared norm is at most `zero2` (numerically zero: norm below
// tol times the largest input column norm) are left alone; their directions
// are rounding noise, and rotating such pairs can cycle without converging.
// Returns true when a rotation was applied.
__device__ bool rotate_pair(const SvdArgs& a, int64_t i, int64_t j, int lane, double zero2) {
  double2* ci = a.Aw + i * a.m;
  double2* cj = a.Aw + j * a.m;
  double al = 0.0, be = 0.0;
  double2 ga = make_double2(0.0, 0.0);
  for (int64_t k = lane; k < a.m; k += 32) {
    const double2 x = ldcg2(ci + k), y = ldcg2(cj + k);
    al += cabs2(x);
    be += cabs2(y);
    ga = cfmac(x, y, ga);  // conj(x) * y
  }
  al = warp_sum(al);
  be = warp_sum(be);
  ga = warp_sum2(ga);
  if (al <= zero2 || be <= zero2) return false;
  const double g = hypot(ga.x, ga.y);
  if (!(g > a.tol * sqrt(al) * sqrt(be))) return false;
  // Real rotation on (a, e^{-i phi} b), e^{i phi} = ga / |ga|, angle from
  // cot(2 theta) = (|b|^2 - |a|^2) / (2 |a^H b|), smaller root for t = tan(theta).
  const double zeta = (be - al) / (2.0 * g);
  double t;
  if (fabs(zeta) > 1e150) {
    t = 0.5 / zeta;
  } else {
    t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
  }
  const double c = 1.0 / sqrt(1.0 + t * t);
  const double s = c * t;
  const double2 e = make_double2(ga.x / g, ga.y / g);
  const double2 s_em = make_double2(s * e.x, -s * e.y);  // s e^{-i phi}
  const double2 s_ep = make_double2(s * e.x, s * e.y);   // s e^{+i phi}
  for (int64_t k = lane; k < a.m; k += 32) {
    const double2 x = ldcg2(ci + k), y = ldcg2(cj + k);
    stcg2(ci + k, csub(cscale(x, c), cmul(s_em, y)));
    stcg2(cj + k, cadd(cmul(s_ep, x), cscale(y, c)));
  }
  double2* vi = a.Vw + i * a.n;
  double2* vj = a.Vw + j * a.n;
  for (int64_t k = lane; k < a.n; k += 32) {
    const double2 x = ldcg2(vi + k), y = ldcg2(vj + k);
    stcg2(vi + k, csub(cscale(x, c), cmul(s_em, y)));
    stcg2(vj + k, cadd(cmul(s_ep, x), cscale(y, c)));
  }
  return true;
}

__global__ void __launch_bounds__(SVD_THREADS) zsvd_jacobi_kernel(SvdArgs a) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = (int64_t)blockIdx.x * SVD_WARPS + (threadIdx.x >> 5);
  const int64_t nw = (int64_t)gridDim.x * SVD_WARPS;
  const int64_t gt = (int64_t)blockIdx.x * SVD_THREADS + threadIdx.x;
  const int64_t nt = (int64_t)gridDim.x * SVD_THREADS;
  const int64_t m = a.m, n = a.n;
  for (int64_t e = gt; e < m * n; e += nt) {
    const int64_t i = e % m, j = e / m;
    stcg2(a.Aw + e, a.src[i * a.rs + j * a.cs]);
  }
  for (int64_t e = gt; e < n * n; e += nt) {
    const int64_t i = e % n, j = e / n;
    stcg2(a.Vw + e, make_double2(i == j ? 1.0 : 0.0, 0.0));
  }
  if (!grid_barrier(a.ctrl, a.status)) return;
  // largest squared column norm (non-negative doubles order like their bit patterns)
  unsigned long long* amax_bits = reinterpret_cast<unsigned long long*>(a.ctrl + 4);
  for (int64_t j = gw; j < n; j += nw) {
    double s2 = 0.0;
    for (int64_t k = lane; k < m; k += 32) s2 += cabs2(ldcg2(a.Aw + j * m + k));
    s2 = warp_sum(s2);
    if (lane == 0) atomicMax(amax_bits, (unsigned long long)__double_as_longlong(s2));
  }
  if (!grid_barrier(a.ctrl, a.status)) return;
  const double amax2 = __longlong_as_double((long long)*((volatile unsigned long long*)amax_bits));
  const double zero2 = a.tol * a.tol * amax2;

  const int64_t np = (n + 1) & ~int64_t(1);
  int sweep = 0;
  bool converged = (n < 2);
  for (; sweep < SVD_MAX_SWEEPS && !converged; ++sweep) {
    for (int64_t r = 0; r + 1 < np; ++r) {
      for (int64_t p = gw; p < np / 2; p += nw) {
        const int64_t x = p, y = np - 1 - p;
        const int64_t i = (x == 0) ? 0 : 1 + (x - 1 + r) % (np - 1);
        const int64_t j = 1 + (y - 1 + r) % (np - 1);
        if (i >= n || j >= n) continue;
        const bool rot = rotate_pair(a, i < j ? i : j, i < j ? j : i, lane, zero2);
        if (rot && lane == 0) atomicAdd(a.ctrl + 8 + (sweep % (CTRL_WORDS - 8)), 1u);
      }
      if (!grid_barrier(a.ctrl, a.status)) return;
    }
    const unsigned cnt = *((volatile unsigned*)(a.ctrl + 8 + (sweep % (CTRL_WORDS - 8))));
    converged = (cnt == 0u);
  }
  if (!converged && blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(a.status, 0, PTN_ERR_NOCONVERGE);

  for (int64_t j = gw; j < n; j += nw) {
    double s2 = 0.0;
    for (int64_t k = lane; k < m; k += 32) s2 += cabs2(ldcg2(a.Aw + j * m + k));
    s2 = warp_sum(s2);
    if (lane == 0) __stcg(a.sig + j, sqrt(s2));
  }
  if (!grid_barrier(a.ctrl, a.status)) return;

  // Sort by rank: position of column j = #{i : sig_i > sig_j or (sig_i == sig_j and i < j)}.
  for (int64_t j = gw; j < n; j += nw) {
    const double sj = __ldcg(a.sig + j);
    int64_t cnt = 0;
    for (int64_t i = lane; i < n; i += 32) {
      const double si = __ldcg(a.sig + i);
      cnt += (si > sj || (si == sj && i < j)) ? 1 : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
    for (int64_t k = lane; k < m; k += 32) a.U[cnt * a.ldu + k] = cscale(ldcg2(a.Aw + j * m + k), inv);
    for (int64_t k = lane; k < n; k += 32) a.V[cnt * a.ldv + k] = ldcg2(a.Vw + j * n + k);
    if (lane == 0) a.S[cnt] = sj;
  }
}

// ---- ring of CTAs: one column pair each ----------------------------------------------------
// The same sweeps, pairs and rotations as above without a grid barrier per
// round. CTA p holds the columns at positions p and np - 1 - p of the circle;
// from one round to the next a column moves one position, so it goes to the
// neighbouring CTA (CTA 0 keeps position 0) and a round only waits for the two
// neighbours. Columns travel through mailboxes in L2 (two per slot, by round
// parity: a CTA sends its round-r columns only after it has the neighbour's of
// round r - 1, which the neighbour sent after reading its mailbox of that
// round). Every 8 bytes of a mailbox carry 4 bytes of the column and the number
// of the round, so the reader polls the data themselves: no fence on either
// side and one L2 round trip less than a separate flag (128 x 128: 7.3 ms with
// flags and fences). Four warps hold the rows of A, four the rows of V; the
// latter take each rotation from shared memory and stay out of the chain of
// dependent rounds.
//
// What bounds it is the FP64 pipe (16 cycles per warp instruction on an SM,
// whatever the active lanes) and the chain poll - dot - rotation - update - send
// of a round. So the four sums of a pair are reduced together (six additions
// instead of twenty), one warp forms the rotation, with two reciprocal square
// roots, while another one decides on it: with d = |b|^2 - |a|^2,
// h = sqrt(d^2 + 4 |a^H b|^2), q = |d| + h,
//   cos = q / sqrt(2 h q),  sin e^{i phi} = sign(d) 2 (a^H b) / sqrt(2 h q),
// the smaller root as above; and the update is 12 FMAs per row, those of V after
// A's columns have been sent. The matrix is scaled by a power of two so that the
// squares stay in range. Measured: 128 x 128 4.2 ms (18.2 ms with the grid barrier
// per round; 5.2 with one warp for the decision and V's FMAs among A's), 256 x 256
// 14.0 (61.0), 384 x 384 38.5 (123; more pairs than SMs).
constexpr int RING_WARPS = 4;                        // per role: rows of A, rows of V
constexpr int RING_ROWS = 32 * RING_WARPS;
constexpr int RING_THREADS = 2 * RING_ROWS;
constexpr int RING_MAX_R = 4;                        // rows per thread: m, n <= 512
constexpr int64_t RING_MIN_N = 8;

struct RingArgs {
  SvdArgs a;
  ulonglong2* box;          // [parity 2][CTA][slot 2][m + n][component 2]
};

// x 2^k for a normal x whose exponent stays in range.
__device__ __forceinline__ double exp_add(double x, int k) {
  return __hiloint2double(__double2hiint(x) + (k << 20), __double2loint(x));
}

// Sum over the warp of four values; every lane of quarter q (8 lanes) gets
// value q.
__device__ __forceinline__ double warp_sum4(double v0, double v1, double v2, double v3, int lane) {
  const bool up = lane & 16;
  const double k0 = up ? v2 : v0, k1 = up ? v3 : v1, s0 = up ? v0 : v2, s1 = up ? v1 : v3;
  const double a = k0 + __shfl_xor_sync(0xffffffffu, s0, 16), b = k1 + __shfl_xor_sync(0xffffffffu, s1, 16);
  const bool odd = lane & 8;
  double r = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
  r += __shfl_xor_sync(0xffffffffu, r, 4);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  return r;
}

// A mailbox entry: a component's low and high words, each in 8 bytes (one
// access of the memory model) with the round's number above it.
__device__ __forceinline__ ulonglong2 ld_mail(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("ld.volatile.global.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_mail1(ulonglong2* p, double v, unsigned long long round) {
  asm volatile("st.volatile.global.v2.u64 [%0], {%1,%2};" ::"l"(p),
               "l"(round | (unsigned)__double2loint(v)), "l"(round | (unsigned)__double2hiint(v))
               : "memory");
}
__device__ __forceinline__ void st_mail(ulonglong2* p, double2 v, unsigned round) {
  st_mail1(p, v.x, (unsigned long long)round << 32);
  st_mail1(p + 1, v.y, (unsigned long long)round << 32);
}
__device__ __forceinline__ double mail_value(ulonglong2 v) { return __hiloint2double((int)v.y, (int)v.x); }

// This thread's rows of two mailboxes once they carry `round`; a bounded wait
// of the warp, false when the kernel must leave.
template <int R>
__device__ __forceinline__ bool ring_read(const ulonglong2* bx, const ulonglong2* by, int tid, int rows, unsigned round,
                                          unsigned* ctrl, int32_t* status, double2* x, double2* y) {
  const volatile unsigned* abort = ctrl + 2;
  const long long t0 = clock64();
  for (unsigned it = 1;; ++it) {
    bool ok = true;
    ulonglong2 v[R][4];
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int t = tid + RING_ROWS * u;
      if (t < rows) {
        v[u][0] = ld_mail(bx + 2 * t);
        v[u][1] = ld_mail(bx + 2 * t + 1);
        v[u][2] = ld_mail(by + 2 * t);
        v[u][3] = ld_mail(by + 2 * t + 1);
      }
    }
#pragma unroll
    for (int u = 0; u < R; ++u) {
      x[u] = y[u] = make_double2(0.0, 0.0);
      if (tid + RING_ROWS * u < rows) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          ok = ok && (unsigned)(v[u][k].x >> 32) == round && (unsigned)(v[u][k].y >> 32) == round;
        x[u] = make_double2(mail_value(v[u][0]), mail_value(v[u][1]));
        y[u] = make_double2(mail_value(v[u][2]), mail_value(v[u][3]));
      }
    }
    if (__all_sync(0xffffffffu, ok)) return true;
    int give_up = 0;
    if ((it & 63u) == 0u && *abort != 0u) give_up = 1;
    if (clock64() - t0 > SVD_WAIT_CYCLES) {
      atomicExch(ctrl + 2, 1u);
      atomicCAS(status, 0, PTN_ERR_TIMEOUT);
      give_up = 1;
    }
    if (__any_sync(0xffffffffu, give_up)) return false;
  }
}

// R: rows per thread (128 R >= m >= n).
template <int R>
__global__ void __launch_bounds__(RING_THREADS) zsvd_ring_kernel(RingArgs g) {
  const SvdArgs& a = g.a;
  const int tid = threadIdx.x & (RING_ROWS - 1), lane = tid & 31, warp = tid >> 5;
  const bool vrole = threadIdx.x >= RING_ROWS;       // rows of V
  const int p = blockIdx.x, P = gridDim.x, m = (int)a.m, n = (int)a.n, np = 2 * P;
  __shared__ double red[2][RING_WARPS][4];
  __shared__ double rot[2][4];                       // cos, Re / Im of sin e^{i phi}, rotated?
  __shared__ int s_fail;
  if (threadIdx.x == 0) s_fail = 0;
  const int64_t len = m + n;
  const int rows = vrole ? n : m, off = vrole ? m : 0;
  auto box = [&](unsigned par, int cta, int slot) {
    return g.box + 2 * (((int64_t)(par & 1u) * 2 * P + 2 * cta + slot) * len + off);
  };
  // where the columns at this CTA's two positions go
  const int to_x = p >= 2 ? p - 1 : 0, slot_x = p == 1 ? 1 : 0;
  const int to_y = p + 1 < P ? p + 1 : p, slot_y = p + 1 < P ? 1 : (P == 1 ? 1 : 0);
  const int cx = p, cy = np - 1 - p;                 // columns at the start of a sweep

  // power of two above the largest component, then the largest column norm
  int* top = reinterpret_cast<int*>(a.ctrl + 3);
  auto src = [&](int c, int r) {
    return (c < n && r < m) ? a.src[r * a.rs + c * a.cs] : make_double2(0.0, 0.0);
  };
  // rounds are numbered from 1: no mailbox carries one yet
  for (unsigned par = 0; par < 2; ++par)
    for (int t = tid; t < rows; t += RING_ROWS)
      for (int k = 0; k < 4; ++k) box(par, p, k & 1)[2 * t + (k >> 1)] = make_ulonglong2(0ull, 0ull);
  if (!vrole) {
    int hi = 0;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const double2 x = src(cx, tid + RING_ROWS * u), y = src(cy, tid + RING_ROWS * u);
      hi = max(hi, max(max(__double2hiint(x.x) & 0x7fffffff, __double2hiint(x.y) & 0x7fffffff),
                       max(__double2hiint(y.x) & 0x7fffffff, __double2hiint(y.y) & 0x7fffffff)));
    }
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0 && hi) atomicMax(top, hi);
  }
  if (!grid_barrier(a.ctrl, a.status)) return;
  const int field = *((volatile int*)top) >> 20;
  const bool scaled = field > 0 && field < 0x7fe;    // 2^(1023 - field) is a normal number
  const double down = scaled ? __hiloint2double((2046 - field) << 20, 0) : 1.0;
  const double upsc = scaled ? __hiloint2double(field << 20, 0) : 1.0;
  unsigned long long* amax_bits = reinterpret_cast<unsigned long long*>(a.ctrl + 4);
  double2 x[R], y[R];
  // |column|^2 of x and y over the A rows: atomically into amax, or to sig
  auto norms = [&](double& sx, double& sy) {
    sx = sy = 0.0;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      sx += cabs2(x[u]);
      sy += cabs2(y[u]);
    }
    const double t = warp_sum4(sx, sy, 0.0, 0.0, lane);
    if (!vrole && (lane & 7) == 0 && lane < 16) red[0][warp][lane >> 3] = t;
    __syncthreads();
    sx = sy = 0.0;
    for (int w = 0; w < RING_WARPS; ++w) {
      sx += red[0][w][0];
      sy += red[0][w][1];
    }
  };
  {
    ulonglong2* bx = box(0, p, 0);
    ulonglong2* by = box(0, p, 1);
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int r = tid + RING_ROWS * u;
      x[u] = vrole ? make_double2(r == cx ? 1.0 : 0.0, 0.0) : cscale(src(cx, r), down);
      y[u] = vrole ? make_double2(r == cy ? 1.0 : 0.0, 0.0) : cscale(src(cy, r), down);
      if (r < rows) {
        st_mail(bx + 2 * r, x[u], 1u);
        st_mail(by + 2 * r, y[u], 1u);
      }
    }
    double sx, sy;
    norms(sx, sy);
    if (threadIdx.x == 0) atomicMax(amax_bits, (unsigned long long)__double_as_longlong(sx > sy ? sx : sy));
  }
  if (!grid_barrier(a.ctrl, a.status)) return;
  const double amax2 = __longlong_as_double((long long)*((volatile unsigned long long*)amax_bits));
  const double tol2 = a.tol * a.tol, zero2 = tol2 * amax2;

  unsigned done = 0;                                 // rounds completed
  bool converged = (n < 2);
  for (int sweep = 0; sweep < SVD_MAX_SWEEPS && !converged; ++sweep) {
    unsigned count = 0;
    for (int r = 0; r + 1 < np; ++r, ++done) {
      const int ci = p == 0 ? 0 : 1 + (p - 1 + r) % (np - 1), cj = 1 + (np - 2 - p + r) % (np - 1);
      const bool swap = ci > cj;                     // the lower column is the rotation's first
      const int q = done & 1;
      // a warp that must leave tells the others at the round's barrier, so all leave
      // there: none is left waiting at a barrier of its own
      const int leave = !ring_read<R>(box(done, p, swap ? 1 : 0), box(done, p, swap ? 0 : 1), tid, rows, done + 1, a.ctrl,
                                      a.status, x, y);
      if (!vrole) {
        double al = 0.0, be = 0.0;
        double2 ga = make_double2(0.0, 0.0);
#pragma unroll
        for (int u = 0; u < R; ++u) {
          al = fma(x[u].x, x[u].x, fma(x[u].y, x[u].y, al));
          be = fma(y[u].x, y[u].x, fma(y[u].y, y[u].y, be));
          ga = cfmac(x[u], y[u], ga);                // conj(x) y
        }
        const double part = warp_sum4(al, be, ga.x, ga.y, lane);
        if ((lane & 7) == 0) red[q][warp][lane >> 3] = part;
        asm volatile("bar.sync 1, %0;" ::"n"(RING_ROWS) : "memory");
        if (warp < 2) {
          double v = red[q][(lane >> 2) & 3][lane & 3];
          v += __shfl_xor_sync(0xffffffffu, v, 4);
          v += __shfl_xor_sync(0xffffffffu, v, 8);
          al = __shfl_sync(0xffffffffu, v, 0);
          be = __shfl_sync(0xffffffffu, v, 1);
          ga.x = __shfl_sync(0xffffffffu, v, 2);
          ga.y = __shfl_sync(0xffffffffu, v, 3);
          const double g2 = fma(ga.x, ga.x, ga.y * ga.y);
          if (warp == 1) {
            const bool turn = al > zero2 && be > zero2 && g2 > tol2 * al * be;
            if (turn) ++count;
            if (lane == 0) rot[q][3] = turn ? 1.0 : 0.0;
          } else {
            // (a pair that is not rotated has no use for these; factors of two on
            // the exponents, where there is a rotation nothing is zero)
            const double d = be - al, xx = fma(d, d, exp_add(g2, 2));
            const double h = xx * rsqrt(xx), qq = fabs(d) + h, rr = rsqrt(exp_add(h, 1) * qq);
            const double f = exp_add(d >= 0.0 ? rr : -rr, 1);
            const double sr = f * ga.x, si = f * ga.y, c = qq * rr;
            if (lane == 0) {
              rot[q][0] = c;
              rot[q][1] = sr;
              rot[q][2] = si;
            }
          }
        }
      }
      if (__syncthreads_or(leave)) return;
      const double c = rot[q][0], sr = rot[q][1], si = rot[q][2];
      const bool turn = rot[q][3] != 0.0;
      ulonglong2* ox = box(done + 1, to_x, slot_x);
      ulonglong2* oy = box(done + 1, to_y, slot_y);
      // V's rows wait until A's are on their way: their FMAs fill the FP64 pipe while
      // the neighbours' columns travel
      if (vrole) asm volatile("bar.sync 2, %0;" ::"n"(RING_THREADS) : "memory");
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int t = tid + RING_ROWS * u;
        if (turn) {
          // x <- c x - s e^{-i phi} y,  y <- s e^{i phi} x + c y
          const double2 s = x[u], w = y[u];
          x[u].x = fma(c, s.x, fma(-sr, w.x, -si * w.y));
          x[u].y = fma(c, s.y, fma(-sr, w.y, si * w.x));
          y[u].x = fma(c, w.x, fma(sr, s.x, -si * s.y));
          y[u].y = fma(c, w.y, fma(sr, s.y, si * s.x));
        }
        if (t < rows) {
          st_mail(ox + 2 * t, swap ? y[u] : x[u], done + 2);
          st_mail(oy + 2 * t, swap ? x[u] : y[u], done + 2);
        }
      }
      if (!vrole) asm volatile("bar.arrive 2, %0;" ::"n"(RING_THREADS) : "memory");
    }
    if (threadIdx.x == 32 && count) atomicAdd(a.ctrl + 8 + (sweep % (CTRL_WORDS - 8)), count);
    if (!grid_barrier(a.ctrl, a.status)) return;
    converged = *((volatile unsigned*)(a.ctrl + 8 + (sweep % (CTRL_WORDS - 8)))) == 0u;
  }
  if (!converged && p == 0 && threadIdx.x == 0) atomicCAS(a.status, 0, PTN_ERR_NOCONVERGE);

  // norms, then every column to its place in descending order (as above)
  {
    if (!ring_read<R>(box(done, p, 0), box(done, p, 1), tid, rows, done + 1, a.ctrl, a.status, x, y)) s_fail = 1;
    __syncthreads();
    if (s_fail) return;
    double sx, sy;
    norms(sx, sy);
    if (threadIdx.x == 0) {
      __stcg(a.sig + cx, sqrt(sx));
      if (cy < n) __stcg(a.sig + cy, sqrt(sy));
    }
  }
  if (!grid_barrier(a.ctrl, a.status)) return;
  for (int e = 0; e < 2; ++e) {
    const int c = e ? cy : cx;
    if (c >= n) continue;
    // compared as bit patterns: the order of non-negative doubles, and a place
    // of its own (first) for a column that is not a number
    const double sj = __ldcg(a.sig + c);
    const long long bj = __double_as_longlong(sj) & 0x7fffffffffffffffll;
    int cnt = 0;
    for (int i = lane; i < n; i += 32) {
      const long long bi = __double_as_longlong(__ldcg(a.sig + i)) & 0x7fffffffffffffffll;
      cnt += (bi > bj || (bi == bj && i < c)) ? 1 : 0;
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
    double2* dst = vrole ? a.V + (int64_t)cnt * a.ldv : a.U + (int64_t)cnt * a.ldu;
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int t = tid + RING_ROWS * u;
      const double2 v = e ? y[u] : x[u];
      if (t < rows) dst[t] = vrole ? v : cscale(v, inv);
    }
    if (threadIdx.x == 0) a.S[cnt] = sj * upsc;
  }
}

// ---- small matrices: one CTA, everything in shared memory --------------------------------
// For n <= SVD_SMALL_N columns whose working copy and rotations fit in shared
// memory (SVD_SMALL_BYTES) and that the ring does not take (n < 8, or more than
// 512 rows) the same sweeps run in one CTA with CTA barriers between rounds (no
// cooperative launch, no global traffic): 86 us for 5 x 3. From 8 columns on one
// SM's FP64 pipe is the bound (8 x 8 296 us, ring 177 us; 32 x 32 5.4 ms, ring 0.90
// ms; 64 x 64 28.4 ms, ring 2.0 ms). Same pair schedule, rotation formula,
// thresholds and ordering as zsvd_jacobi_kernel, one warp per pair (the pairs of
// a round are disjoint, so how they are spread over the warps does not matter),
// so the results are the same bit for bit.
constexpr int64_t SVD_SMALL_N = 64;
constexpr int64_t SVD_SMALL_BYTES = 200 * 1024;
constexpr int SVD_SMALL_THREADS = 1024;

__device__ bool rotate_pair_smem(double2* A, double2* V, int64_t m, int64_t n, int64_t i, int64_t j, double tol,
                                 double zero2, int lane) {
  double2* ci = A + i * m;
  double2* cj = A + j * m;
  double al = 0.0, be = 0.0;
  double2 ga = make_double2(0.0, 0.0);
  for (int64_t k = lane; k < m; k += 32) {
    const double2 x = ci[k], y = cj[k];
    al += cabs2(x);
    be += cabs2(y);
    ga = cfmac(x, y, ga);
  }
  al = warp_sum(al);
  be = warp_sum(be);
  ga = warp_sum2(ga);
  if (al <= zero2 || be <= zero2) return false;
  const double g = hypot(ga.x, ga.y);
  if (!(g > tol * sqrt(al) * sqrt(be))) return false;
  const double zeta = (be - al) / (2.0 * g);
  double t;
  if (fabs(zeta) > 1e150) {
    t = 0.5 / zeta;
  } else {
    t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
  }
  const double c = 1.0 / sqrt(1.0 + t * t);
  const double s = c * t;
  const double2 e = make_double2(ga.x / g, ga.y / g);
  const double2 s_em = make_double2(s * e.x, -s * e.y);
  const double2 s_ep = make_double2(s * e.x, s * e.y);
  for (int64_t k = lane; k < m; k += 32) {
    const double2 x = ci[k], y = cj[k];
    ci[k] = csub(cscale(x, c), cmul(s_em, y));
    cj[k] = cadd(cmul(s_ep, x), cscale(y, c));
  }
  double2* vi = V + i * n;
  double2* vj = V + j * n;
  for (int64_t k = lane; k < n; k += 32) {
    const double2 x = vi[k], y = vj[k];
    vi[k] = csub(cscale(x, c), cmul(s_em, y));
    vj[k] = cadd(cmul(s_ep, x), cscale(y, c));
  }
  return true;
}

__global__ void __launch_bounds__(SVD_SMALL_THREADS) zsvd_jacobi_small_kernel(SvdArgs a) {
  extern __shared__ double2 sm[];
  __shared__ double sig[SVD_SMALL_N];
  __shared__ unsigned rot;
  __shared__ double amax2s;
  const int64_t m = a.m, n = a.n;
  double2* A = sm;
  double2* V = sm + m * n;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  constexpr int NW = SVD_SMALL_THREADS / 32;
  for (int64_t e = threadIdx.x; e < m * n; e += SVD_SMALL_THREADS) {
    const int64_t i = e % m, j = e / m;
    A[e] = a.src[i * a.rs + j * a.cs];
  }
  for (int64_t e = threadIdx.x; e < n * n; e += SVD_SMALL_THREADS) {
    const int64_t i = e % n, j = e / n;
    V[e] = make_double2(i == j ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  for (int64_t j = wp; j < n; j += NW) {
    double s2 = 0.0;
    for (int64_t k = lane; k < m; k += 32) s2 += cabs2(A[j * m + k]);
    s2 = warp_sum(s2);
    if (lane == 0) sig[j] = s2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double mx = 0.0;
    for (int64_t j = 0; j < n; ++j) mx = sig[j] > mx ? sig[j] : mx;
    amax2s = mx;
  }
  __syncthreads();
  const double zero2 = a.tol * a.tol * amax2s;
  const int64_t np = (n + 1) & ~int64_t(1);
  bool converged = (n < 2);
  int sweep = 0;
  for (; sweep < SVD_MAX_SWEEPS && !converged; ++sweep) {
    if (threadIdx.x == 0) rot = 0u;
    __syncthreads();
    for (int64_t r = 0; r + 1 < np; ++r) {
      for (int64_t p = wp; p < np / 2; p += NW) {
        const int64_t x = p, y = np - 1 - p;
        const int64_t i = (x == 0) ? 0 : 1 + (x - 1 + r) % (np - 1);
        const int64_t j = 1 + (y - 1 + r) % (np - 1);
        if (i >= n || j >= n) continue;
        const bool did = rotate_pair_smem(A, V, m, n, i < j ? i : j, i < j ? j : i, a.tol, zero2, lane);
        if (did && lane == 0) atomicAdd(&rot, 1u);
      }
      __syncthreads();
    }
    converged = (rot == 0u);
    __syncthreads();
  }
  if (!converged && threadIdx.x == 0) atomicCAS(a.status, 0, PTN_ERR_NOCONVERGE);
  for (int64_t j = wp; j < n; j += NW) {
    double s2 = 0.0;
    for (int64_t k = lane; k < m; k += 32) s2 += cabs2(A[j * m + k]);
    s2 = warp_sum(s2);
    if (lane == 0) sig[j] = sqrt(s2);
  }
  __syncthreads();
  for (int64_t j = wp; j < n; j += NW) {
    const double sj = sig[j];
    int64_t cnt = 0;
    for (int64_t i = lane; i < n; i += 32) {
      const double si = sig[i];
      cnt += (si > sj || (si == sj && i < j)) ? 1 : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
    for (int64_t k = lane; k < m; k += 32) a.U[cnt * a.ldu + k] = cscale(A[j * m + k], inv);
    for (int64_t k = lane; k < n; k += 32) a.V[cnt * a.ldv + k] = V[j * n + k];
    if (lane == 0) a.S[cnt] = sj;
  }
}

// Co-resident CTAs of a kernel on the current device (kernel: an index into the
// table, one per cooperative kernel).
constexpr int SVD_KERNELS = 1 + RING_MAX_R;
int g_svd_max_blocks[64][SVD_KERNELS] = {};
std::mutex g_svd_mutex;

int svd_max_blocks(int kernel, const void* fn, int threads) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::lock_guard<std::mutex> lock(g_svd_mutex);
  int& cached = g_svd_max_blocks[dev][kernel];
  if (cached == 0) {
    int per_sm = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    cached = per_sm * sms;
  }
  return cached;
}

const void* ring_kernel(int r) {
  switch (r) {
    case 1: return (const void*)zsvd_ring_kernel<1>;
    case 2: return (const void*)zsvd_ring_kernel<2>;
    case 3: return (const void*)zsvd_ring_kernel<3>;
    default: return (const void*)zsvd_ring_kernel<4>;
  }
}

inline int64_t align256(int64_t x) { return (x + 255) & ~int64_t(255); }

// ---- strided permute / conjugate / scale ---------------------------------------
__global__ void zpermute_kernel(ptn_permute_desc d, int64_t total) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t rem = e, so = 0, dof = 0, sidx = 0;
    for (int i = d.n - 1; i >= 0; --i) {
      const int64_t q = rem / d.dim[i];
      const int64_t x = rem - q * d.dim[i];
      rem = q;
      so += x * d.stride_src[i];
      dof += x * d.stride_dst[i];
      if (i == d.scale_mode) sidx = x;
    }
    double2 v = static_cast<const double2*>(d.src)[so];
    if (d.conj) v.y = -v.y;
    if (d.scale) v = cscale(v, d.scale[sidx]);
    static_cast<double2*>(d.dst)[dof] = v;
  }
}

}  // namespace

extern "C" int64_t ptn_zsvd_work_bytes(int64_t m, int64_t n) {
  if (m < 1 || n < 1) return 0;
  // control words, norms, then the working copies of the columns (in the ring
  // two mailboxes each, of twice a column's size)
  const int64_t np = (n + 1) & ~int64_t(1);
  return CTRL_BYTES + align256(8 * n) + align256((n >= RING_MIN_N && m <= RING_MAX_R * RING_ROWS ? 64 : 16) * np * (m + n));
}

extern "C" int ptn_zsvd_jacobi(const ptn_svd_desc* d, void* stream) {
  if (!d || !d->A || !d->U || !d->S || !d->V || !d->work || !d->status) return PTN_ERR_ARG;
  if (d->n < 1 || d->m < d->n || d->ldu < d->m || d->ldv < d->n) return PTN_ERR_ARG;
  SvdArgs a;
  a.src = static_cast<const double2*>(d->A);
  a.rs = d->row_stride;
  a.cs = d->col_stride;
  a.m = d->m;
  a.n = d->n;
  uint8_t* w = static_cast<uint8_t*>(d->work);
  const int64_t np = (d->n + 1) & ~int64_t(1);
  a.ctrl = reinterpret_cast<unsigned*>(w);
  a.sig = reinterpret_cast<double*>(w + CTRL_BYTES);
  double2* cols = reinterpret_cast<double2*>(w + CTRL_BYTES + align256(8 * d->n));
  a.Aw = cols;
  a.Vw = cols + d->m * d->n;
  a.U = static_cast<double2*>(d->U);
  a.ldu = d->ldu;
  a.S = d->S;
  a.V = static_cast<double2*>(d->V);
  a.ldv = d->ldv;
  // sqrt(m) * 2^-53 (LAPACK's zgesvj) sits at the rounding floor of one
  // rotation for small m, and a pair can then cycle without ever passing the
  // test; 8 sqrt(m) * 2^-53 keeps U and V orthonormal to ~1e-14.
  a.tol = 8.0 * sqrt((double)d->m) * 1.1102230246251565e-16;
  a.status = d->status;
  cudaStream_t s = ptn_stream(stream);
  const int r = (int)((d->m + RING_ROWS - 1) / RING_ROWS);
  if (d->n >= RING_MIN_N && r <= RING_MAX_R && np / 2 <= svd_max_blocks(r, ring_kernel(r), RING_THREADS)) {
    if (cudaMemsetAsync(a.ctrl, 0, CTRL_BYTES, s) != cudaSuccess) return PTN_ERR_LAUNCH;
    RingArgs g;
    g.a = a;
    g.box = reinterpret_cast<ulonglong2*>(cols);
    void* args[] = {&g};
    PTN_COUNT(1);
    if (cudaLaunchCooperativeKernel(ring_kernel(r), dim3((unsigned)(np / 2)), dim3(RING_THREADS), args, 0, s) !=
        cudaSuccess) {
      cudaGetLastError();
      return PTN_ERR_LAUNCH;
    }
    return PTN_OK;
  }
  const size_t smem = (size_t)(d->m * d->n + d->n * d->n) * sizeof(double2);
  if (d->n <= SVD_SMALL_N && smem <= (size_t)SVD_SMALL_BYTES) {
    static const cudaError_t attr = cudaFuncSetAttribute(
        zsvd_jacobi_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SVD_SMALL_BYTES);
    if (attr != cudaSuccess) return PTN_ERR_LAUNCH;
    PTN_COUNT(1);
    zsvd_jacobi_small_kernel<<<1, SVD_SMALL_THREADS, smem, s>>>(a);
    return ptn_launch_status();
  }
  const int maxb = svd_max_blocks(0, (const void*)zsvd_jacobi_kernel, SVD_THREADS);
  if (maxb <= 0) return PTN_ERR_LAUNCH;
  if (cudaMemsetAsync(a.ctrl, 0, CTRL_BYTES, s) != cudaSuccess) return PTN_ERR_LAUNCH;
  const int64_t pairs = (((d->n + 1) & ~int64_t(1)) / 2);
  int64_t blocks = (pairs + SVD_WARPS - 1) / SVD_WARPS;
  if (blocks < 1) blocks = 1;
  if (blocks > maxb) blocks = maxb;
  void* args[] = {&a};
  PTN_COUNT(1);
  const cudaError_t e = cudaLaunchCooperativeKernel((const void*)zsvd_jacobi_kernel, dim3((unsigned)blocks),
                                                    dim3(SVD_THREADS), args, 0, s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return PTN_ERR_LAUNCH;
  }
  return PTN_OK;
}

extern "C" int ptn_zpermute(const ptn_permute_desc* d, void* stream) {
  if (!d || !d->src || !d->dst || d->n < 0 || d->n > PTN_MAX_MODES) return PTN_ERR_ARG;
  if (d->scale && (d->scale_mode < 0 || d->scale_mode >= d->n)) return PTN_ERR_ARG;
  int64_t total = 1;
  for (int i = 0; i < d->n; ++i) {
    if (d->dim[i] < 0) return PTN_ERR_ARG;
    total *= d->dim[i];
  }
  if (total == 0) return PTN_OK;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  PTN_COUNT(1);
  zpermute_kernel<<<(unsigned)blocks, 256, 0, ptn_stream(stream)>>>(*d, total);
  return ptn_launch_status();
}
