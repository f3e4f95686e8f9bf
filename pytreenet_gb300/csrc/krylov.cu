// Krylov (Lanczos/Arnoldi) vector kernels in complex128.
//
// The Krylov basis q_0..q_j is stored as rows of one matrix; the Gram-Schmidt
// projections of krylov_exp_action (time_evolution/time_evolution.py:721-821)
// become one multi-dot pass (every vector read once, j+1 sums in registers)
// and one multi-axpy pass. Reductions are deterministic: warp shuffles, then a
// shared-memory tree per CTA, then one CTA summing the per-CTA partials in a
// fixed order, so repeated runs give identical bits.
#include "ptn_common.cuh"

namespace {

constexpr int RT = 256;        // threads per CTA
constexpr int MAXQ = 16;       // vectors per multi-dot launch
constexpr int64_t CHUNK = 1024;   // elements per CTA: enough CTAs to keep HBM busy on 131k-entry vectors

inline int64_t nblocks_for(int64_t n) {
  int64_t b = (n + CHUNK - 1) / CHUNK;
  if (b < 1) b = 1;
  if (b > 1184) b = 1184;  // 8 CTAs per SM on 148+ SMs
  return b;
}

template <int NQ>
__global__ void __launch_bounds__(RT) zdot_partial_kernel(const double2* __restrict__ Q, int64_t ldq,
                                                          int nq, const double2* __restrict__ w,
                                                          int64_t n, double2* __restrict__ partial) {
  double2 acc[NQ];
#pragma unroll
  for (int i = 0; i < NQ; ++i) acc[i] = make_double2(0.0, 0.0);
  for (int64_t x = blockIdx.x * (int64_t)RT + threadIdx.x; x < n; x += (int64_t)gridDim.x * RT) {
    double2 wv = w[x];
#pragma unroll
    for (int i = 0; i < NQ; ++i)
      if (i < nq) acc[i] = cfmac(Q[(int64_t)i * ldq + x], wv, acc[i]);
  }
  __shared__ double2 red[RT / 32][NQ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    if (i >= nq) break;
    double2 v = warp_sum2(acc[i]);
    if (lane == 0) red[warp][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < nq) {
    double2 s = make_double2(0.0, 0.0);
    for (int wi = 0; wi < RT / 32; ++wi) s = cadd(s, red[wi][threadIdx.x]);
    partial[(int64_t)blockIdx.x * MAXQ + threadIdx.x] = s;
  }
}

__global__ void zdot_finish_kernel(const double2* __restrict__ partial, int nb, int nq,
                                   double2* __restrict__ h, int accumulate) {
  // one warp per output, lanes stride over the partials in a fixed order
  const int i = blockIdx.x;
  double2 s = make_double2(0.0, 0.0);
  for (int b = threadIdx.x; b < nb; b += 32) s = cadd(s, partial[(int64_t)b * MAXQ + i]);
  s = warp_sum2(s);
  if (threadIdx.x == 0) h[i] = accumulate ? cadd(h[i], s) : s;
}

__global__ void __launch_bounds__(RT) zaxpy_multi_kernel(const double2* __restrict__ Q, int64_t ldq,
                                                         int nq, const double2* __restrict__ h,
                                                         double2* __restrict__ w, int64_t n) {
  __shared__ double2 hs[64];
  if (threadIdx.x < nq) hs[threadIdx.x] = h[threadIdx.x];
  __syncthreads();
  for (int64_t x = blockIdx.x * (int64_t)RT + threadIdx.x; x < n; x += (int64_t)gridDim.x * RT) {
    double2 v = w[x];
    for (int i = 0; i < nq; ++i) {
      double2 q = Q[(int64_t)i * ldq + x];
      double2 hq = cmul(hs[i], q);
      v = csub(v, hq);
    }
    w[x] = v;
  }
}

__global__ void __launch_bounds__(RT) nrm2_partial_kernel(const double2* __restrict__ w, int64_t n,
                                                          double* __restrict__ partial) {
  double acc = 0.0;
  for (int64_t x = blockIdx.x * (int64_t)RT + threadIdx.x; x < n; x += (int64_t)gridDim.x * RT)
    acc += cabs2(w[x]);
  __shared__ double red[RT / 32];
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < RT / 32; ++i) s += red[i];
    partial[blockIdx.x] = s;
  }
}

__global__ void nrm2_finish_kernel(const double* __restrict__ partial, int nb, double* out) {
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += 32) s += partial[b];
  s = warp_sum(s);
  if (threadIdx.x == 0) out[0] = sqrt(s);
}

__global__ void __launch_bounds__(RT) zscal_inv_kernel(const double2* __restrict__ w,
                                                       const double* __restrict__ scale,
                                                       double2* __restrict__ y, int64_t n) {
  const double inv = 1.0 / scale[0];
  for (int64_t x = blockIdx.x * (int64_t)RT + threadIdx.x; x < n; x += (int64_t)gridDim.x * RT)
    y[x] = cscale(w[x], inv);
}

__global__ void __launch_bounds__(RT) zscal_ratio_kernel(const double2* __restrict__ w,
                                                         const double* __restrict__ num,
                                                         const double* __restrict__ den,
                                                         double2* __restrict__ y, int64_t n) {
  const double f = den[0] > 0.0 ? num[0] / den[0] : 1.0;
  for (int64_t x = blockIdx.x * (int64_t)RT + threadIdx.x; x < n; x += (int64_t)gridDim.x * RT)
    y[x] = cscale(w[x], f);
}

__global__ void __launch_bounds__(RT) zcombine_kernel(const double2* __restrict__ Q, int64_t ldq,
                                                      int nq, const double2* __restrict__ c,
                                                      double2* __restrict__ out, int64_t n) {
  __shared__ double2 cs[64];
  if (threadIdx.x < nq) cs[threadIdx.x] = c[threadIdx.x];
  __syncthreads();
  for (int64_t x = blockIdx.x * (int64_t)RT + threadIdx.x; x < n; x += (int64_t)gridDim.x * RT) {
    double2 v = make_double2(0.0, 0.0);
    for (int i = 0; i < nq; ++i) v = cfma(cs[i], Q[(int64_t)i * ldq + x], v);
    out[x] = v;
  }
}

__global__ void check_finite_kernel(const double* __restrict__ x, int64_t n2, int32_t* flag) {
  for (int64_t i = blockIdx.x * (int64_t)RT + threadIdx.x; i < n2; i += (int64_t)gridDim.x * RT)
    if (!isfinite(x[i])) *flag = 1;
}

}  // namespace

std::atomic<unsigned long long> g_ptn_launches{0};

extern "C" unsigned long long ptn_launch_counter(void) { return g_ptn_launches.load(); }

extern "C" int ptn_stream_synchronize(void* stream) {
  return cudaStreamSynchronize(ptn_stream(stream)) == cudaSuccess ? PTN_OK : PTN_ERR_LAUNCH;
}

// ---- Gram-Schmidt step -------------------------------------------------------------------
// Three passes over w, each ending in a sum over all entries:
//   0: (Q^H w, |w|^2)            -> h[0..nq), norms[0] = |w|
//   1: w -= Q h1, then Q^H w     -> h[nq..2nq)
//   2: w -= Q h2, then |w|^2     -> norms[1] = |w|
// (16 nq + 4) FP64 FMAs per entry, which bound it: GB300 issues 2 per clock and
// SM, a warp instruction holding its scheduler's FP64 unit for 64 cycles whatever
// the active lanes. So the sums over lanes matter as much as those over entries:
// 2 nq values are reduced together, each step halving the values a lane carries
// (16 additions for 8 vectors, where one shuffle tree per value takes 80).
__device__ __forceinline__ double2 axpy_sub(double2 w, double2 h, double2 q) {
  w.x = fma(-h.x, q.x, w.x);
  w.x = fma(h.y, q.y, w.x);
  w.y = fma(-h.x, q.y, w.y);
  w.y = fma(-h.y, q.x, w.y);
  return w;
}

// Sum over the warp of N (a power of two up to 32) values per lane: lane l gets
// the sum of value l / (32 / N).
template <int N>
__device__ __forceinline__ double warp_sums(double (&v)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int cnt = N; cnt > 1; cnt >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < cnt / 2; ++j) {
      const double keep = up ? v[j + cnt / 2] : v[j], send = up ? v[j] : v[j + cnt / 2];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double r = v[0];
#pragma unroll
  for (int k = 16 / N; k > 0; k >>= 1) r += __shfl_xor_sync(0xffffffffu, r, k);
  return r;
}

__host__ __device__ constexpr int pow2_at_least(int n) { return n <= 1 ? 1 : 2 * pow2_at_least((n + 1) / 2); }

// CTA sums of a pass's values (Re, Im of NQ dots, then the squared norm where
// the mode has them) into red[warp][value]; the caller's threads v < count add
// the warps in order.
template <int NQ, int MODE, int WARPS>
__device__ __forceinline__ void cta_sums(const double2 (&acc)[NQ], double nacc, double (*red)[2 * NQ + 1]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (MODE != 2) {
    constexpr int N = pow2_at_least(2 * NQ);
    double v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = i < 2 * NQ ? ((i & 1) ? acc[i / 2].y : acc[i / 2].x) : 0.0;
    const double t = warp_sums(v, lane);
    const int idx = lane / (32 / N);
    if (lane % (32 / N) == 0 && idx < 2 * NQ) red[warp][idx] = t;
  }
  if (MODE != 1) {
    const double t = warp_sum(nacc);
    if (lane == 0) red[warp][2 * NQ] = t;
  }
  __syncthreads();
}

// One entry of a pass.
template <int NQ, int MODE>
__device__ __forceinline__ double2 gs_entry(const double2* __restrict__ Q, int64_t ldq, int64_t x, double2 wv,
                                            const double2 (&hs)[NQ], double2 (&acc)[NQ], double& nacc) {
  double2 q[NQ];
#pragma unroll
  for (int i = 0; i < NQ; ++i) q[i] = Q[(int64_t)i * ldq + x];
  if (MODE != 0) {
#pragma unroll
    for (int i = 0; i < NQ; ++i) wv = axpy_sub(wv, hs[i], q[i]);
  }
  if (MODE != 2) {
#pragma unroll
    for (int i = 0; i < NQ; ++i) acc[i] = cfmac(q[i], wv, acc[i]);
  }
  if (MODE != 1) nacc = fma(wv.x, wv.x, fma(wv.y, wv.y, nacc));
  return wv;
}

// Vectors whose w does not fit in the GPU's shared memory (152 x 12800 entries):
// one launch per pass, at 86 to 93 % of the FP64 pipe (33.5 M entries, 8 vectors:
// 7.6 ms; 10.7 with six-operation updates and a tree per sum). Each CTA writes its sums, and the last CTA
// to finish (atomic ticket, no waiting) adds them up in a fixed tree, so the
// totals are deterministic; it also re-arms the ticket.
template <int NQ, int MODE>
__global__ void __launch_bounds__(RT) gs_pass_kernel(const double2* __restrict__ Q, int64_t ldq,
                                                     double2* __restrict__ w, int64_t n,
                                                     const double2* __restrict__ hin, double* __restrict__ hout,
                                                     double* __restrict__ nout, double* __restrict__ partial,
                                                     unsigned* __restrict__ ticket) {
  constexpr int NV = 2 * NQ + 1, WARPS = RT / 32;
  __shared__ double red[WARPS][NV];
  __shared__ int last;
  double2 hs[NQ], acc[NQ];
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    hs[i] = MODE != 0 ? hin[i] : make_double2(0.0, 0.0);
    acc[i] = make_double2(0.0, 0.0);
  }
  double nacc = 0.0;
  for (int64_t x = blockIdx.x * (int64_t)RT + threadIdx.x; x < n; x += (int64_t)gridDim.x * RT) {
    const double2 wv = gs_entry<NQ, MODE>(Q, ldq, x, w[x], hs, acc, nacc);
    if (MODE != 0) w[x] = wv;
  }
  cta_sums<NQ, MODE, WARPS>(acc, nacc, red);
  // values of this mode: [v0, NV) or [0, v1)
  constexpr int v0 = MODE == 2 ? 2 * NQ : 0, v1 = MODE == 1 ? 2 * NQ : NV;
  const int tv = (int)threadIdx.x;
  if (tv >= v0 && tv < v1) {
    double t = 0.0;
#pragma unroll
    for (int u = 0; u < WARPS; ++u) t += red[u][threadIdx.x];
    __stcg(partial + (int64_t)blockIdx.x * NV + threadIdx.x, t);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  // one warp per value, lanes stride over the CTAs
  for (int v = v0 + (threadIdx.x >> 5); v < v1; v += WARPS) {
    double t = 0.0;
    for (unsigned b = threadIdx.x & 31; b < gridDim.x; b += 32) t += __ldcg(partial + (int64_t)b * NV + v);
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) {
      if (v == 2 * NQ) nout[0] = sqrt(t);
      else hout[v] = t;
    }
  }
  if (threadIdx.x == 0) *ticket = 0u;
}

// Vectors whose w fits the GPU's shared memory: the whole step in one
// cooperative launch. Each CTA keeps its piece of w in shared memory, publishes
// its sums (every 8 bytes carry 4 of the value and a mark, so readers poll the
// data themselves, without fences) and adds those of all CTAs in a fixed tree:
// about 2 us for an exchange, where a kernel boundary with the last CTA adding
// up cost 5 us and more. Per step with 8 vectors: 1024 entries 24 us (88 with one
// launch per pass and the scaling), 4394 27 (89), 131072 58 (120; FP64 bound 28),
// 524288 145 (406; 110). 
constexpr int FT = 256;
constexpr int FUSED_MAX_CTAS = 152;
constexpr int FUSED_MAX_NQ = 16;
constexpr int64_t FUSED_SMEM = 200 * 1024;
constexpr long long GS_WAIT_CYCLES = 4000000000LL;   // ~2 s at 2 GHz

template <int NQ, int MODE>
__device__ __forceinline__ bool gs_exchange(const double2 (&acc)[NQ], double nacc, double (*red)[2 * NQ + 1],
                                            double* tot, ulonglong2* mail) {
  constexpr int NV = 2 * NQ + 1, WARPS = FT / 32;
  constexpr int v0 = MODE == 2 ? 2 * NQ : 0, v1 = MODE == 1 ? 2 * NQ : NV;
  cta_sums<NQ, MODE, WARPS>(acc, nacc, red);
  const int G = gridDim.x;
  const int tv = (int)threadIdx.x;
  double mine = 0.0;
  if (tv >= v0 && tv < v1) {
#pragma unroll
    for (int u = 0; u < WARPS; ++u) mine += red[u][tv];
    if (G == 1) tot[tv] = mine;
  }
  if (G == 1) {
    __syncthreads();
    return true;
  }
  if (tv >= v0 && tv < v1) {
    const unsigned long long mark = 1ull << 32;
    asm volatile("st.volatile.global.v2.u64 [%0], {%1,%2};" ::"l"(mail + (int64_t)tv * G + blockIdx.x),
                 "l"(mark | (unsigned)__double2loint(mine)), "l"(mark | (unsigned)__double2hiint(mine))
                 : "memory");
  }
  // K values per warp at a time, all their loads in flight together
  constexpr int K = NV <= 8 ? 1 : (NV <= 16 ? 2 : 4), J = (FUSED_MAX_CTAS + 31) / 32;
  const int lane = threadIdx.x & 31;
  bool ok = true;
  for (int v = v0 + K * (int)(threadIdx.x >> 5); v < v1; v += K * WARPS) {
    ulonglong2 e[K][J];
    const long long t0 = clock64();
    while (true) {
      bool all = true;
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < J; ++j) {
          const int b = lane + 32 * j;
          e[k][j] = make_ulonglong2(1ull << 32, 1ull << 32);
          if (v + k < v1 && b < G)
            asm volatile("ld.volatile.global.v2.u64 {%0,%1}, [%2];"
                         : "=l"(e[k][j].x), "=l"(e[k][j].y)
                         : "l"(mail + (int64_t)(v + k) * G + b)
                         : "memory");
        }
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll
        for (int j = 0; j < J; ++j) all = all && (e[k][j].x >> 32) == 1ull && (e[k][j].y >> 32) == 1ull;
      if (__all_sync(0xffffffffu, all)) break;
      if (__any_sync(0xffffffffu, clock64() - t0 > GS_WAIT_CYCLES)) {
        ok = false;
        break;
      }
    }
    double s[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      s[k] = 0.0;
#pragma unroll
      for (int j = 0; j < J; ++j)
        if (32 * j < G) s[k] += __hiloint2double((int)(unsigned)e[k][j].y, (int)(unsigned)e[k][j].x);
    }
    const double t = warp_sums(s, lane);
    if (lane % (32 / K) == 0 && v + lane / (32 / K) < v1) tot[v + lane / (32 / K)] = t;
  }
  return __syncthreads_and(ok ? 1 : 0) != 0;
}

template <int NQ>
__global__ void __launch_bounds__(FT) gs_fused_kernel(const double2* __restrict__ Q, int64_t ldq,
                                                      double2* __restrict__ w, int64_t n, int64_t per_cta,
                                                      double* __restrict__ h, double* __restrict__ norms,
                                                      double2* __restrict__ qnext, ulonglong2* __restrict__ mail) {
  extern __shared__ double2 ws[];
  constexpr int NV = 2 * NQ + 1;
  __shared__ double red[FT / 32][NV];
  __shared__ double tot[NV];
  const int64_t x0 = blockIdx.x * per_cta;
  const int len = (int)(n - x0 < per_cta ? n - x0 : per_cta);
  const int64_t slot = (int64_t)NV * gridDim.x;
  // norms[1] only grows, as the bits of a non-negative double: a CTA whose wait runs out
  // leaves a NaN that no other one's result replaces. It starts from zero before this
  // CTA's first sums are out; a CTA that gives up before the last exchange is missed there
  // by all, so only later NaNs have to last.
  unsigned long long* norm_bits = reinterpret_cast<unsigned long long*>(norms + 1);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    atomicExch(norm_bits, 0ull);
    __threadfence();
  }
  double2 hs[NQ], acc[NQ];
  double nacc = 0.0;
  auto clear = [&]() {
#pragma unroll
    for (int i = 0; i < NQ; ++i) acc[i] = make_double2(0.0, 0.0);
    nacc = 0.0;
  };
  auto take = [&]() {
#pragma unroll
    for (int i = 0; i < NQ; ++i) hs[i] = make_double2(tot[2 * i], tot[2 * i + 1]);
  };
  clear();
#pragma unroll
  for (int i = 0; i < NQ; ++i) hs[i] = make_double2(0.0, 0.0);
  for (int e = threadIdx.x; e < len; e += FT) {
    const double2 v = w[x0 + e];
    ws[e] = v;
    gs_entry<NQ, 0>(Q, ldq, x0 + e, v, hs, acc, nacc);
  }
  bool ok = gs_exchange<NQ, 0>(acc, nacc, red, tot, mail);
  if (ok) {
    take();
    if (blockIdx.x == 0 && threadIdx.x < 2 * NQ) h[threadIdx.x] = tot[threadIdx.x];
    if (blockIdx.x == 0 && threadIdx.x == 2 * NQ) norms[0] = sqrt(tot[2 * NQ]);
    clear();
    for (int e = threadIdx.x; e < len; e += FT) ws[e] = gs_entry<NQ, 1>(Q, ldq, x0 + e, ws[e], hs, acc, nacc);
    ok = gs_exchange<NQ, 1>(acc, nacc, red, tot, mail + slot);
  }
  if (ok) {
    take();
    if (blockIdx.x == 0 && threadIdx.x < 2 * NQ) h[2 * NQ + threadIdx.x] = tot[threadIdx.x];
    clear();
    for (int e = threadIdx.x; e < len; e += FT) ws[e] = gs_entry<NQ, 2>(Q, ldq, x0 + e, ws[e], hs, acc, nacc);
    ok = gs_exchange<NQ, 2>(acc, nacc, red, tot, mail + 2 * slot);
  }
  if (!ok) {                                         // the caller sees a norm that is not a number
    if (threadIdx.x == 0) {
      norms[0] = NAN;
      atomicMax(norm_bits, 0x7ff8000000000000ull);
    }
    return;
  }
  const double nrm = sqrt(tot[2 * NQ]), inv = 1.0 / nrm;
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicMax(norm_bits, (unsigned long long)__double_as_longlong(nrm));
  for (int e = threadIdx.x; e < len; e += FT) {
    const double2 v = ws[e];
    w[x0 + e] = v;
    if (qnext) qnext[x0 + e] = cscale(v, inv);
  }
}

// CTAs of the fused step on a device of `sms` SMs: enough entries each that the
// exchange of G partial sums does not outweigh the pass, one to an SM (all of them
// wait on one another, so all have to be resident).
static inline int64_t fused_ctas(int64_t n, int64_t sms) {
  const int64_t g = (n + 127) / 128, most = sms < FUSED_MAX_CTAS ? sms : FUSED_MAX_CTAS;
  return g < most ? g : most;
}

// CTAs of the one-launch Gram-Schmidt step, 0 where w does not fit in their shared memory.
extern "C" int64_t ptn_krylov_fused_ctas(int64_t n, int64_t sms) {
  if (n < 1 || sms < 1) return 0;
  const int64_t g = fused_ctas(n, sms), per = (n + g - 1) / g;
  return per * (int64_t)sizeof(double2) <= FUSED_SMEM ? (n + per - 1) / per : 0;
}

template <int NQ>
static int gs_step_nq(const double2* Q, int64_t ldq, double2* w, int64_t n, double2* h, double2* partial,
                      double* norms, double2* qnext, cudaStream_t s) {
  double* hd = reinterpret_cast<double*>(h);
  static PtnSharedMemory shared_memory;
  const int64_t g = ptn_krylov_fused_ctas(n, ptn_sm_count());
  if (g > 0 && shared_memory((const void*)gs_fused_kernel<NQ>, FUSED_SMEM)) {
    const int64_t most = fused_ctas(n, ptn_sm_count());
    int64_t nn = n, pp = (n + most - 1) / most, ld = ldq;
    ulonglong2* mail = reinterpret_cast<ulonglong2*>(partial);
    if (g == 1) {                                    // nothing to exchange
      PTN_COUNT(1);
      gs_fused_kernel<NQ><<<1, FT, (size_t)pp * sizeof(double2), s>>>(Q, ldq, w, n, pp, hd, norms, qnext, mail);
      return ptn_launch_status();
    }
    if (cudaMemsetAsync(mail, 0, (size_t)(3 * (2 * NQ + 1) * g) * sizeof(ulonglong2), s) != cudaSuccess)
      return PTN_ERR_LAUNCH;
    void* args[] = {&Q, &ld, &w, &nn, &pp, &hd, &norms, &qnext, &mail};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)gs_fused_kernel<NQ>, dim3((unsigned)g), dim3(FT),
                                                      args, (size_t)pp * sizeof(double2), s);
    if (e == cudaSuccess) {
      PTN_COUNT(1);
      return ptn_launch_status();
    }
    cudaGetLastError();
    // fewer SMs to this context than to the device: one launch per pass, below
    if (e != cudaErrorCooperativeLaunchTooLarge) return PTN_ERR_LAUNCH;
  }
  const int nb = (int)nblocks_for(n);
  double* part = reinterpret_cast<double*>(partial);
  unsigned* ticket = reinterpret_cast<unsigned*>(part + (int64_t)nb * (2 * NQ + 1));
  if (cudaMemsetAsync(ticket, 0, sizeof(unsigned), s) != cudaSuccess) return PTN_ERR_LAUNCH;
  PTN_COUNT(3);
  gs_pass_kernel<NQ, 0><<<nb, RT, 0, s>>>(Q, ldq, w, n, nullptr, hd, norms, part, ticket);
  gs_pass_kernel<NQ, 1><<<nb, RT, 0, s>>>(Q, ldq, w, n, h, hd + 2 * NQ, nullptr, part, ticket);
  gs_pass_kernel<NQ, 2><<<nb, RT, 0, s>>>(Q, ldq, w, n, h + NQ, nullptr, norms + 1, part, ticket);
  if (qnext) {
    PTN_COUNT(1);
    zscal_inv_kernel<<<nb, RT, 0, s>>>(w, norms + 1, qnext, n);
  }
  return ptn_launch_status();
}

// The Gram-Schmidt step for nq <= MAXQ (PTN_ERR_UNSUPPORTED otherwise, and the
// caller runs the kernels one by one).
int ptn_gs_step_passes(const void* Q, int64_t ldq, int32_t nq, void* w, int64_t n, void* h, void* partial,
                       double* norms, void* qnext, void* stream) {
  const double2* q = static_cast<const double2*>(Q);
  double2* wv = static_cast<double2*>(w);
  double2* hv = static_cast<double2*>(h);
  double2* pv = static_cast<double2*>(partial);
  double2* qn = static_cast<double2*>(qnext);
  cudaStream_t s = ptn_stream(stream);
  switch (nq) {
#define PTN_GS_CASE(k) \
  case k:              \
    return gs_step_nq<k>(q, ldq, wv, n, hv, pv, norms, qn, s);
    PTN_GS_CASE(1)
    PTN_GS_CASE(2)
    PTN_GS_CASE(3)
    PTN_GS_CASE(4)
    PTN_GS_CASE(5)
    PTN_GS_CASE(6)
    PTN_GS_CASE(7)
    PTN_GS_CASE(8)
    PTN_GS_CASE(9)
    PTN_GS_CASE(10)
    PTN_GS_CASE(11)
    PTN_GS_CASE(12)
    PTN_GS_CASE(13)
    PTN_GS_CASE(14)
    PTN_GS_CASE(15)
    PTN_GS_CASE(16)
#undef PTN_GS_CASE
    default:
      return PTN_ERR_UNSUPPORTED;
  }
}

// per-CTA sums of the kernels above, and the mailboxes of the fused step
extern "C" int64_t ptn_krylov_partials(int64_t n) {
  const int64_t per_pass = nblocks_for(n) * (MAXQ + 1) + 16;
  const int64_t fused = 3 * (2 * FUSED_MAX_NQ + 1) * fused_ctas(n, FUSED_MAX_CTAS);
  return per_pass > fused ? per_pass : fused;
}

extern "C" int ptn_zdot_multi(const void* Q, int64_t ldq, int32_t nq, const void* w, int64_t n,
                              void* h, int32_t accumulate, void* partial, void* stream) {
  if (!Q || !w || !h || !partial || nq < 1 || n < 1 || ldq < n) return PTN_ERR_ARG;
  cudaStream_t s = ptn_stream(stream);
  const int nb = (int)nblocks_for(n);
  for (int i0 = 0; i0 < nq; i0 += MAXQ) {
    int cnt = nq - i0 < MAXQ ? nq - i0 : MAXQ;
    const double2* Qi = static_cast<const double2*>(Q) + (int64_t)i0 * ldq;
    double2* hp = static_cast<double2*>(h) + i0;
    double2* pp = static_cast<double2*>(partial);
    PTN_COUNT(2);
    if (cnt <= 4)
      zdot_partial_kernel<4><<<nb, RT, 0, s>>>(Qi, ldq, cnt, static_cast<const double2*>(w), n, pp);
    else if (cnt <= 8)
      zdot_partial_kernel<8><<<nb, RT, 0, s>>>(Qi, ldq, cnt, static_cast<const double2*>(w), n, pp);
    else
      zdot_partial_kernel<16><<<nb, RT, 0, s>>>(Qi, ldq, cnt, static_cast<const double2*>(w), n, pp);
    zdot_finish_kernel<<<cnt, 32, 0, s>>>(pp, nb, cnt, hp, accumulate);
  }
  return ptn_launch_status();
}

extern "C" int ptn_zaxpy_multi(const void* Q, int64_t ldq, int32_t nq, const void* h, void* w,
                               int64_t n, void* stream) {
  if (!Q || !w || !h || nq < 1 || n < 1 || ldq < n) return PTN_ERR_ARG;
  cudaStream_t s = ptn_stream(stream);
  const int nb = (int)nblocks_for(n);
  for (int i0 = 0; i0 < nq; i0 += 64) {
    int cnt = nq - i0 < 64 ? nq - i0 : 64;
    PTN_COUNT(1);
    zaxpy_multi_kernel<<<nb, RT, 0, s>>>(static_cast<const double2*>(Q) + (int64_t)i0 * ldq, ldq, cnt,
                                         static_cast<const double2*>(h) + i0,
                                         static_cast<double2*>(w), n);
  }
  return ptn_launch_status();
}

extern "C" int ptn_dznrm2(const void* w, int64_t n, void* out_norm, void* partial, void* stream) {
  if (!w || !out_norm || !partial || n < 1) return PTN_ERR_ARG;
  cudaStream_t s = ptn_stream(stream);
  const int nb = (int)nblocks_for(n);
  PTN_COUNT(1);
  nrm2_partial_kernel<<<nb, RT, 0, s>>>(static_cast<const double2*>(w), n, static_cast<double*>(partial));
  PTN_COUNT(1);
  nrm2_finish_kernel<<<1, 32, 0, s>>>(static_cast<const double*>(partial), nb, static_cast<double*>(out_norm));
  return ptn_launch_status();
}

extern "C" int ptn_zscal_inv(const void* w, const double* scale, void* y, int64_t n, void* stream) {
  if (!w || !scale || !y || n < 1) return PTN_ERR_ARG;
  PTN_COUNT(1);
  zscal_inv_kernel<<<(int)nblocks_for(n), RT, 0, ptn_stream(stream)>>>(
      static_cast<const double2*>(w), scale, static_cast<double2*>(y), n);
  return ptn_launch_status();
}

extern "C" int ptn_zscal_ratio(const void* w, const double* num, const double* den, void* y, int64_t n,
                               void* stream) {
  if (!w || !num || !den || !y || n < 1) return PTN_ERR_ARG;
  PTN_COUNT(1);
  zscal_ratio_kernel<<<(int)nblocks_for(n), RT, 0, ptn_stream(stream)>>>(
      static_cast<const double2*>(w), num, den, static_cast<double2*>(y), n);
  return ptn_launch_status();
}

extern "C" int ptn_zcombine(const void* Q, int64_t ldq, int32_t nq, const void* c, void* out,
                            int64_t n, void* stream) {
  if (!Q || !c || !out || nq < 1 || nq > 64 || n < 1 || ldq < n) return PTN_ERR_ARG;
  PTN_COUNT(1);
  zcombine_kernel<<<(int)nblocks_for(n), RT, 0, ptn_stream(stream)>>>(
      static_cast<const double2*>(Q), ldq, nq, static_cast<const double2*>(c),
      static_cast<double2*>(out), n);
  return ptn_launch_status();
}

extern "C" int ptn_check_finite(const void* x, int64_t n, int32_t* flag, void* stream) {
  if (!x || !flag || n < 0) return PTN_ERR_ARG;
  if (n == 0) return PTN_OK;
  PTN_COUNT(1);
  check_finite_kernel<<<(int)nblocks_for(n), RT, 0, ptn_stream(stream)>>>(
      static_cast<const double*>(x), 2 * n, flag);
  return ptn_launch_status();
}
