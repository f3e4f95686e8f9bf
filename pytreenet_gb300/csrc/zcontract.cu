// Strided multi-mode complex128 tensor contraction (FP64 plain path).
//
// C[m, n] = alpha * sum_k opA(A)[m, k] opB(B)[k, n] + beta * C[m, n], where m, n
// and k are each a group of up to PTN_MAX_MODES tensor legs addressed through
// per-operand strides. Legs are never transposed in memory: the environment,
// TTNO and site tensors of a tree node are contracted where they lie.
//
// GB300 FP64 issues about two DFMA per clock per SM, so this kernel is bound by
// the FP64 pipe at modest tile sizes: 64 x 64 complex outputs per CTA, 256
// threads with a 4 x 4 register tile each, K staged through shared memory in
// steps of 8. Tile offsets of the M and N rows are decoded once per CTA; the K
// offsets once per K step.
//
// Outputs of less than 152 tiles run on zcontract_elem_kernel. Skinny outputs of
// more than 4096 entries over a long K (an environment, or the gradient of one, is
// chi x w x chi summed over everything else) would leave most SMs idle with
// one CTA per output tile, so when there are few tiles the K range is split
// over gridDim.y: a first kernel writes beta * C (or zero), and each split
// adds alpha times its partial sums with double-precision atomics. The
// summation order then varies between runs at the level of rounding.
#include <cooperative_groups.h>

#include "ptn_common.cuh"
#include "zmodes.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 8;

__global__ void __launch_bounds__(256) zcontract_kernel(const ContractArgs a) {
  __shared__ double2 As[BK][BM];
  __shared__ double2 Bs[BK][BN];
  __shared__ int64_t offAm[BM], offCm[BM], offBn[BN], offCn[BN];
  __shared__ int64_t offAk[BK], offBk[BK];

  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int64_t tile = blockIdx.x;
  const int64_t tm = tile / a.tiles_n;
  const int64_t tn = tile - tm * a.tiles_n;
  const int64_t m0 = tm * BM, n0 = tn * BN;

  if (tid < BM) {
    int64_t mi = m0 + tid;
    int64_t oa = -1, oc = -1;
    if (mi < a.M) decode(a.m, mi, oa, oc);
    offAm[tid] = oa;
    offCm[tid] = oc;
  } else if (tid < BM + BN) {
    int t = tid - BM;
    int64_t ni = n0 + t;
    int64_t ob = -1, oc = -1;
    if (ni < a.N) decode(a.n, ni, ob, oc);
    offBn[t] = ob;
    offCn[t] = oc;
  }

  double2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_double2(0.0, 0.0);

  const int64_t kbeg = (int64_t)blockIdx.y * a.k_chunk;
  const int64_t kend = (kbeg + a.k_chunk < a.K) ? kbeg + a.k_chunk : a.K;
  for (int64_t k0 = kbeg; k0 < kend; k0 += BK) {
    __syncthreads();
    if (tid < BK) {
      int64_t ki = k0 + tid;
      int64_t oa = -1, ob = -1;
      if (ki < kend) decode(a.k, ki, oa, ob);
      offAk[tid] = oa;
      offBk[tid] = ob;
    }
    __syncthreads();
    // 512 elements of each tile, two per thread.
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      int e = tid + r * 256;
      int kk = e / BM, mm = e - kk * BM;
      double2 v = make_double2(0.0, 0.0);
      if (offAk[kk] >= 0 && offAm[mm] >= 0) {
        v = a.A[offAm[mm] + offAk[kk]];
        if (a.conj_a) v.y = -v.y;
      }
      As[kk][mm] = v;
      int nn = e - kk * BN;
      double2 w = make_double2(0.0, 0.0);
      if (offBk[kk] >= 0 && offBn[nn] >= 0) {
        w = a.B[offBk[kk] + offBn[nn]];
        if (a.conj_b) w.y = -w.y;
      }
      Bs[kk][nn] = w;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      double2 av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = cfma(av[i], bv[j], acc[i][j]);
    }
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int mm = ty + 16 * i;
    if (offCm[mm] < 0) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int nn = tx + 16 * j;
      if (offCn[nn] < 0) continue;
      double2* p = a.C + offCm[mm] + offCn[nn];
      double2 v = cmul(a.alpha, acc[i][j]);
      if (a.split) {
        atomicAdd(&p->x, v.x);
        atomicAdd(&p->y, v.y);
        continue;
      }
      if (!a.beta_zero) v = cfma(a.beta, *p, v);
      *p = v;
    }
  }
}

// Products with fewer output tiles than SMs: the tiled kernel would put a whole
// 64 x 64 tile -- most of it padding when M or N is small -- on each of a few SMs,
// at ~2 FP64 FMAs per clock per SM. Here one thread sums one output over one of S
// interleaved K slices (S = 1, 2, ..., 32) of a CTA, and for long K a cluster of C
// CTAs (up to 8) takes K in equal ranges, so that few outputs still reach the FP64
// units of many SMs; CTAs have four warps, one per scheduler and its FP64 unit.
// The slices are added in order and the CTAs' sums by the first CTA in order,
// through distributed shared memory: the result does not vary between runs. The
// K offsets are decoded once per CTA into shared memory. Measured against one
// thread per output and, for up to 256 outputs, one CTA of 1024 threads: 128 x 64,
// K = 64 16.5 -> 10 us; 64 x 64, K = 128 29 -> 10; 13 x 13, K = 1014 186 -> 12;
// 2 x 2, K = 4096 39 -> 12 (all with ~7 us of host call).
constexpr int ELEM_THREADS = 128;
constexpr int ELEM_MAX_CLUSTER = 8;
constexpr int64_t ELEM_SPLIT_OUT = 4096;   // outputs up to which K ranges go to clusters

template <int S>
__global__ void __launch_bounds__(ELEM_THREADS) zcontract_elem_kernel(const ContractArgs a, const int C) {
  constexpr int OUTS = ELEM_THREADS / S;             // outputs per cluster
  __shared__ int64_t offAk[ELEM_THREADS], offBk[ELEM_THREADS];
  __shared__ double2 part[ELEM_THREADS];
  const int rank = C > 1 ? (int)(blockIdx.x % C) : 0;
  const int slice = threadIdx.x / OUTS;
  const int64_t o = (blockIdx.x / C) * (int64_t)OUTS + (threadIdx.x - slice * OUTS);
  const bool valid = o < a.M * a.N;
  int64_t oa = 0, ocm = 0, ob = 0, ocn = 0;
  if (valid) {
    const int64_t mi = o / a.N, ni = o - mi * a.N;
    decode(a.m, mi, oa, ocm);
    decode(a.n, ni, ob, ocn);
  }
  double2 acc = make_double2(0.0, 0.0);
  const int64_t kbeg = rank * a.k_chunk, kend = kbeg + a.k_chunk < a.K ? kbeg + a.k_chunk : a.K;
  for (int64_t k0 = kbeg; k0 < kend; k0 += ELEM_THREADS) {
    if (k0 != kbeg) __syncthreads();
    {
      const int64_t k = k0 + threadIdx.x;
      int64_t x = 0, y = 0;
      if (k < kend) decode(a.k, k, x, y);
      offAk[threadIdx.x] = x;
      offBk[threadIdx.x] = y;
    }
    __syncthreads();
    const int cnt = (int)(kend - k0 < ELEM_THREADS ? kend - k0 : ELEM_THREADS);
    if (valid) {
      // operand pairs loaded four ahead of their in-order accumulation
      int kk = slice;
      for (; kk + 3 * S < cnt; kk += 4 * S) {
        double2 av[4], bv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          av[u] = a.A[oa + offAk[kk + u * S]];
          bv[u] = a.B[offBk[kk + u * S] + ob];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (a.conj_a) av[u].y = -av[u].y;
          if (a.conj_b) bv[u].y = -bv[u].y;
          acc = cfma(av[u], bv[u], acc);
        }
      }
      for (; kk < cnt; kk += S) {
        double2 av = a.A[oa + offAk[kk]];
        double2 bv = a.B[offBk[kk] + ob];
        if (a.conj_a) av.y = -av.y;
        if (a.conj_b) bv.y = -bv.y;
        acc = cfma(av, bv, acc);
      }
    }
  }
  if (S > 1) {
    part[threadIdx.x] = acc;
    __syncthreads();
    if (slice == 0)
      for (int u = 1; u < S; ++u) acc = cadd(acc, part[threadIdx.x + u * OUTS]);
  }
  if (C > 1) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    if (slice == 0) part[threadIdx.x] = acc;
    cluster.sync();
    if (rank == 0 && slice == 0)
      for (int r = 1; r < C; ++r) acc = cadd(acc, cluster.map_shared_rank(part, r)[threadIdx.x]);
    cluster.sync();                                  // the others' shared memory was being read
    if (rank != 0) return;
  }
  if (valid && slice == 0) {
    double2* p = a.C + ocm + ocn;
    double2 v = cmul(a.alpha, acc);
    if (!a.beta_zero) v = cfma(a.beta, *p, v);
    *p = v;
  }
}

// C <- beta * C (zero when beta == 0) over the M x N output positions.
__global__ void __launch_bounds__(256) zcontract_scale_c(const ContractArgs a) {
  const int64_t total = a.M * a.N;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t mi = i / a.N, ni = i - mi * a.N;
    int64_t oa, ocm, ob, ocn;
    decode(a.m, mi, oa, ocm);
    decode(a.n, ni, ob, ocn);
    double2* p = a.C + ocm + ocn;
    *p = a.beta_zero ? make_double2(0.0, 0.0) : cmul(a.beta, *p);
  }
}

template <int S>
int64_t launch_elem_s(ContractArgs& a, int c, cudaStream_t s) {
  constexpr int64_t outs = ELEM_THREADS / S;
  const int64_t blocks = (a.M * a.N + outs - 1) / outs * c;
  if (blocks > 0x7fffffffLL) return 0;
  a.k_chunk = (a.K + c - 1) / c;
  PTN_COUNT(1);
  if (c == 1) {
    zcontract_elem_kernel<S><<<(unsigned)blocks, ELEM_THREADS, 0, s>>>(a, c);
    return blocks;
  }
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)c;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(ELEM_THREADS);
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, zcontract_elem_kernel<S>, a, c) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return blocks;
}

// The launch of zcontract_elem_kernel. K slices: the count with the least FP64
// time on the fullest SM (CTAs per SM, rounded up, times the k of a slice, plus
// the adding up), at least eight k each; then, for few outputs, a cluster over
// ranges of K. Returns the CTAs launched, 0 when the outputs are too many, -1 on
// an error.
int64_t launch_elem(ContractArgs& a, cudaStream_t s) {
  const int64_t out = a.M * a.N;
  int sl = 1, c = 1;
  int64_t best = INT64_MAX;
  for (int t = 1; t <= 32 && (t == 1 || a.K >= 8 * t); t *= 2) {
    const int64_t blocks = (out * t + ELEM_THREADS - 1) / ELEM_THREADS;
    const int64_t cost = (blocks + 151) / 152 * (4 * ((a.K + t - 1) / t) + 8 + t / 2);
    if (cost < best) {
      best = cost;
      sl = t;
    }
  }
  while (out <= ELEM_SPLIT_OUT && sl == 32 && c < ELEM_MAX_CLUSTER && out * sl * c < 152 * ELEM_THREADS &&
         a.K >= 16 * sl * c)
    c *= 2;
  switch (sl) {
    case 1: return launch_elem_s<1>(a, c, s);
    case 2: return launch_elem_s<2>(a, c, s);
    case 4: return launch_elem_s<4>(a, c, s);
    case 8: return launch_elem_s<8>(a, c, s);
    case 16: return launch_elem_s<16>(a, c, s);
    default: return launch_elem_s<32>(a, c, s);
  }
}

}  // namespace

// Split K when the output tiles cover at most a quarter of the 152 SMs: about
// 304 CTAs in all, each split at least 256 K indices long, chunks a multiple
// of the K step; the chunks cover [0, K) exactly once.
extern "C" int64_t ptn_zcontract_splits(int64_t tiles, int64_t K, int64_t* k_chunk) {
  *k_chunk = K;
  if (tiles > 38 || K < 2048) return 1;
  int64_t want = (304 + tiles - 1) / tiles;
  int64_t most = K / 256;
  int64_t splits = want < most ? want : most;
  if (splits < 2) return 1;
  *k_chunk = ((K + splits - 1) / splits + BK - 1) / BK * BK;
  return (K + *k_chunk - 1) / *k_chunk;
}

extern "C" int ptn_zcontract(const ptn_contract_desc* d, void* stream) {
  if (!d || !d->A || !d->B || !d->C) return PTN_ERR_ARG;
  ContractArgs a;
  if (zcontract_args(*d, a)) return PTN_ERR_ARG;
  const int64_t M = a.M, N = a.N, K = a.K;
  if (M == 0 || N == 0) return PTN_OK;
  cudaStream_t s = ptn_stream(stream);
  int64_t tm = (M + BM - 1) / BM, tn = (N + BN - 1) / BN;
  a.tiles_n = tn;
  int64_t tiles = tm * tn;
  if (tiles > 0x7fffffffLL) return PTN_ERR_UNSUPPORTED;
  int64_t splits = ptn_zcontract_splits(tiles, K, &a.k_chunk);
  a.split = splits > 1;
  if (tiles < 152 && (!a.split || M * N <= ELEM_SPLIT_OUT)) {
    const int64_t blocks = launch_elem(a, s);
    if (blocks != 0) return blocks > 0 ? ptn_launch_status() : PTN_ERR_LAUNCH;
  }
  if (a.split) {
    int64_t total = M * N;
    int64_t blocks = (total + 255) / 256;
    if (blocks > 1024) blocks = 1024;
    PTN_COUNT(1);
    zcontract_scale_c<<<(unsigned)blocks, 256, 0, s>>>(a);
  }
  PTN_COUNT(1);
  zcontract_kernel<<<dim3((unsigned)tiles, (unsigned)splits), 256, 0, s>>>(a);
  return ptn_launch_status();
}
