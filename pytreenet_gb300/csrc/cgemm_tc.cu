// Mixed-precision complex contraction on the 5th-generation tensor cores.
//
// C[m, n] = sum_k A[m, k] * B[n, k] (complex), with A and B split into L BF16
// levels (x = x0 + x1 [+ x2], each bf16, 8 more mantissa bits per level) and
// the products of levels i + j < L accumulated in FP32 in TMEM:
//   L = 2 ("BF16x3"): A0B0 + A0B1 + A1B0, relative error ~2^-16;
//   L = 3 ("BF16x6"): + A0B2 + A1B1 + A2B0, relative error ~2^-24 (FP32 level).
// The complex product is written as one real product with doubled width:
//   [Cr | Ci] = Ar * [Br | Bi] + Ai * [-Bi | Br]
// so each (i, j) term issues two tcgen05.mma (M=128, N=2*NT, K=16; NT = 64 or 128
// complex columns). The
// expanded B keeps the three blocks [-Bi; Br; Bi] of a level adjacent in shared
// memory, so the Ar operand is the window [Br; Bi] and the Ai operand the
// window [-Bi; Br].
//
// Operands (both K-major, K contiguous):
//   A: 2L bf16 planes (Ar_0, Ai_0, Ar_1, Ai_1, ...), each [M][lda]
//   Bx: bf16 [level][block(-Bi, Br, Bi)][N][ldb]
// Tiles are staged by TMA (32-byte swizzle, K=16 per stage, up to 8 stages)
// through an mbarrier ring; two stages make one 32-wide accumulation round;
// one warp issues TMA, one warp issues MMA and owns the TMEM allocation, four or
// eight warps run the epilogue (TMEM -> registers -> global, strided by output mode
// tables so the result lands directly in the layout the next step reads). A CTA
// stays on its SM and goes from tile to tile: while its epilogue writes one tile,
// loads and MMAs of the next run on.
// Every mbarrier wait is bounded; a timeout sets *status and the CTA exits.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <type_traits>

#include "ptn_common.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int MT = 128;         // rows of C per CTA
constexpr int KT = 32;          // K per accumulation round (the unit of the K split)
constexpr int KS = 16;          // K per shared-memory stage (one 32-byte swizzle row, one MMA K)
constexpr int A_PLANE_BYTES = MT * 2 * KS;         // 4 KB
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr int TMEM_COLS = 512;
constexpr int EC = 64;          // complex columns of an epilogue thread's row

// Stages of KS: as many as fit (at most 8). Two stages make one accumulation
// round, so the TMEM partial sums cover 32 K values.
// NT: complex columns of C per CTA (MMA N = 2*NT).
template <int L, int NT>
struct Cfg {
  static constexpr int B_BLOCK = NT * 2 * KS;
  static constexpr int A_STAGE = 2 * L * A_PLANE_BYTES;
  static constexpr int B_STAGE = 3 * L * B_BLOCK;
  static constexpr int STAGE = A_STAGE + B_STAGE;
  static constexpr int STAGES = (SMEM_LIMIT - 4096) / STAGE > 8 ? 8 : (SMEM_LIMIT - 4096) / STAGE;
  static constexpr int SMEM = STAGES * STAGE + 1024;
  static constexpr int EPI_WARPS = 4 * (NT / EC);
  static constexpr int THREADS = 64 + 32 * EPI_WARPS;
  static constexpr int NBUF = TMEM_COLS / (2 * NT);   // TMEM accumulators
};
constexpr long long WAIT_CYCLES = 4000000000LL;    // ~2 s at 2 GHz

struct OutModes {
  int n;
  int64_t dim[PTN_MAX_MODES];
  int64_t stride[PTN_MAX_MODES];
};

struct GemmArgs {
  int64_t M, N, K;
  int out_kind;              // 0: complex128, 1: bf16 planes
  void* C;
  int64_t c_plane;           // plane stride (elements) for out_kind 1
  OutModes mo, no;
  int32_t* status;
  int32_t tiles_m;           // row blocks of C
  int32_t items;             // tiles times K ranges
  int32_t splits;            // K ranges per tile (1: no split)
  int32_t ksplit;            // K tiles (KT) per range
  float2* partial;           // [splits][M][N] FP32 partial sums when splits > 1
  int32_t store;             // how the epilogue writes (StoreKind)
};

// Stores of the epilogue, where a thread holds 64 columns of one row. Single entries
// of BF16 planes whose columns are the contiguous index are 2-byte pieces of 32
// sectors an instruction, 50 us for one 128 x 64 tile; hence
//   ROW8, 4, 2: that many columns of a row together (innermost column mode of stride 1);
//   PAIR4, 2: that many columns of two rows (innermost row mode of stride 1 and even
//         extent, innermost column mode of stride 2: a site's physical leg of
//         dimension 2), neighbour lanes exchange halves;
//   PAIR: one column of two rows (the same row mode, any column modes).
// Every other stride, the plane stride and the base are then multiples of a store
// (store_kind). Complex128 (ROW2) and partial sums (ROW4) go out 32 bytes at a time.
enum StoreKind { ST_ONE = 0, ST_ROW8, ST_ROW4, ST_ROW2, ST_PAIR4, ST_PAIR2, ST_PAIR };

// Split-K: outputs with fewer tiles than this many CTAs get their K range
// split so the launch fills the GPU (one CTA per SM, 152 SMs, two waves);
// each range keeps at least SPLIT_MIN_KT K tiles.
constexpr int64_t SPLIT_TARGET_CTAS = 304;
constexpr int64_t SPLIT_MIN_KT = 4;
// Products with fewer K tiles than this are not split: measured on GB300, the
// partial-sum pass costs more than the parallelism gains below K = 1024
// (512 x 1280 x 256: 70 us split, 47 us not; 256 x 256 x 1280: 54 vs 84 us).
constexpr int64_t SPLIT_MIN_KT_TOTAL = 32;

__device__ __forceinline__ int64_t decode_off(const OutModes& md, int64_t idx) {
  int64_t o = 0;
  for (int d = md.n - 1; d >= 0; --d) {
    int64_t q = idx / md.dim[d];
    o += (idx - q * md.dim[d]) * md.stride[d];
    idx = q;
  }
  return o;
}

// The same for an index and extents below 2^31.
__device__ __forceinline__ int64_t decode_off32(const OutModes& md, uint32_t idx) {
  int64_t o = 0;
  for (int d = md.n - 1; d > 0; --d) {
    const uint32_t dim = (uint32_t)md.dim[d], q = idx / dim;
    o += (int64_t)(idx - q * dim) * md.stride[d];
    idx = q;
  }
  return md.n > 0 ? o + (int64_t)idx * md.stride[0] : 0;   // idx is in range: no division for the first
}

// Work items (K range, tile): CTA b takes b, b + gridDim.x, ... Tiles of a row block of
// C follow one another, so that CTAs which run together share A in L2; the narrow tiles
// that a ragged N leaves come last, where they even out the CTAs' shares.
struct Item {
  int64_t m0, n0;
  int split, k0, stages;         // first stage and stages of KS of the K range
};
template <int NT>
__device__ __forceinline__ Item item_at(const GemmArgs& g, uint32_t w) {
  Item it;
  const uint32_t full = (uint32_t)(g.N / NT), tm_all = (uint32_t)g.tiles_m;
  const uint32_t whole = full * tm_all * (uint32_t)g.splits;
  uint32_t tm;
  if (w < whole) {
    const uint32_t r = w / full;
    it.n0 = (int64_t)(w - r * full) * NT;
    it.split = (int)(r / tm_all);
    tm = r - (uint32_t)it.split * tm_all;
  } else {
    w -= whole;
    it.n0 = (int64_t)full * NT;
    it.split = (int)(w / tm_all);
    tm = w - (uint32_t)it.split * tm_all;
  }
  it.m0 = (int64_t)tm * MT;
  const int all = (int)((g.K + KS - 1) / KS), per = g.ksplit * (KT / KS);
  it.k0 = it.split * per;        // the ranges are whole accumulation rounds (KT)
  it.stages = min(all, it.k0 + per) - it.k0;
  return it;
}

__device__ __forceinline__ void st_global_32(void* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e,
                                             uint32_t f, uint32_t g, uint32_t h) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d), "r"(e),
               "r"(f), "r"(g), "r"(h)
               : "memory");
}

// v = bf16(x); x -= v
__device__ __forceinline__ uint32_t take_bf16(float& x) {
  const __nv_bfloat16 b = __float2bfloat16_rn(x);
  x -= __bfloat162float(b);
  return (uint32_t)__bfloat16_as_ushort(b);
}

__device__ __forceinline__ void put_words(__nv_bfloat16* p, const uint32_t* w, int n) {
  if (n == 4) *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  else if (n == 2) *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
  else *reinterpret_cast<uint32_t*>(p) = w[0];
}

// Eight columns of one plane, x[0..7] (their next BF16 piece), from a lane's row.
// no: the offsets of the eight columns (-1: past the end). Whole warps come here:
// lanes exchange.
template <int KIND>
__device__ __forceinline__ void store_plane8(__nv_bfloat16* __restrict__ C, float* x, const int64_t* no, bool row_ok) {
  constexpr bool ROW = KIND == ST_ROW8 || KIND == ST_ROW4 || KIND == ST_ROW2;
  constexpr bool QUAD = KIND == ST_PAIR4 || KIND == ST_PAIR2;
  uint32_t v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = take_bf16(x[i]);
  const bool odd = threadIdx.x & 1;
  if (KIND == ST_ONE || ((ROW || QUAD) && no[7] < 0)) {      // or the last columns
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (row_ok && no[i] >= 0) C[no[i]] = __ushort_as_bfloat16((unsigned short)v[i]);
  } else if constexpr (ROW) {
    constexpr int V = KIND == ST_ROW8 ? 8 : (KIND == ST_ROW4 ? 4 : 2);
    const uint32_t w[4] = {v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16};
    if (row_ok) {
#pragma unroll
      for (int i = 0; i < 8; i += V) put_words(C + no[i], w + i / 2, V / 2);
    }
  } else if constexpr (QUAD) {
    // of 2 V columns the even lane writes the first V of both rows, the odd one the last
    constexpr int V = KIND == ST_PAIR4 ? 4 : 2;
#pragma unroll
    for (int g = 0; g < 8; g += 2 * V) {
      uint32_t w[V];
#pragma unroll
      for (int i = 0; i < V; i += 2) {
        const uint32_t mine = odd ? (v[g + i] | v[g + i + 1] << 16) : (v[g + V + i] | v[g + V + i + 1] << 16);
        const uint32_t r = __shfl_xor_sync(0xffffffffu, mine, 1);
        w[i] = odd ? ((r & 0xffffu) | v[g + V + i] << 16) : (v[g + i] | r << 16);
        w[i + 1] = odd ? (r >> 16 | v[g + V + i + 1] << 16) : (v[g + i + 1] | (r & 0xffff0000u));
      }
      if (row_ok) put_words(C + (odd ? no[g + V] - 1 : no[g]), w, V);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const uint32_t r = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
      const int64_t n = odd ? no[i + 1] : no[i];
      if (row_ok && n >= 0)
        *reinterpret_cast<uint32_t*>(C + n - (odd ? 1 : 0)) = odd ? (r | v[i + 1] << 16) : (v[i] | r << 16);
    }
  }
}
template <int L, int KIND>
__device__ __forceinline__ void store_planes(__nv_bfloat16* __restrict__ C, int64_t ps, float (&re)[EC],
                                             float (&im)[EC], const int64_t* no, bool row_ok) {
#pragma unroll
  for (int i = 0; i < EC; i += 8) {
    if (no[i] < 0) break;                   // the same in all lanes
#pragma unroll
    for (int lv = 0; lv < L; ++lv) {
      store_plane8<KIND>(C + (2 * lv) * ps, re + i, no + i, row_ok);
      store_plane8<KIND>(C + (2 * lv + 1) * ps, im + i, no + i, row_ok);
    }
  }
}

// What bounds it: the tensor pipe against shared memory. An MMA of N = 128 takes 64
// cycles and reads 8 KB of operands, all that shared memory gives, and the stages
// have to be written too; one of N = 256 reads 12 KB in 128 cycles. And every tile
// pays for its start (barriers, TMEM, tensor maps, first loads) and its output,
// 25 us of a K = 1280 tile's 65 and 13 of a K = 256 tile's 20 when a CTA did one tile
// each. Hence NT = 128 where there are tiles enough (launch_gemm), and persistent
// CTAs: two accumulation rounds of the next tile fit in TMEM while the epilogue
// writes. Measured (BF16x6, tensor-pipe rate counts the six products):
// 655360 x 256 x 1280 8.65 -> 6.86 ms (1190 -> 1500 TFLOP/s), 131072 x 1280 x 256 into
// rows of ten 3.11 -> 1.70, 131072 x 256 x 256 into complex128 0.54 -> 0.34, 40000 x 200
// x 136 into planes by rows 0.51 -> 0.14, 640 x 128 x 640 into pairs 67 -> 47 us.
template <int L, int NT>
__global__ void __launch_bounds__(64 + 128 * (NT / EC), 1)
    cgemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const GemmArgs g) {
  using C_ = Cfg<L, NT>;
  constexpr int STAGES = C_::STAGES;
  constexpr int STAGE_BYTES = C_::STAGE;
  constexpr int A_STAGE_BYTES = C_::A_STAGE;
  constexpr int B_BLOCK_BYTES = C_::B_BLOCK;
  constexpr int NBUF = C_::NBUF;
  constexpr uint32_t ACC_COLS = 2 * NT;          // one accumulator: [Re | Im]
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], tfull_bar[NBUF], tempty_bar[NBUF], drain_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int64_t noff_s[C_::EPI_WARPS][EC];
  __shared__ int s_abort;
  const volatile int32_t* vstatus = g.status;
  if (threadIdx.x == 0) s_abort = *vstatus;
  __syncthreads();
  if (s_abort != 0) return;  // an earlier launch failed: skip the work

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t items = (uint32_t)g.items;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < NBUF; ++b) {
      tc::mbar_init(&tfull_bar[b], 1);
      tc::mbar_init(&tempty_bar[b], C_::EPI_WARPS);   // one arrival per epilogue warp
    }
    tc::mbar_init(&drain_bar, 1);
    tc::fence_mbar_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(&tmem_base, TMEM_COLS);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_base;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      tc::prefetch_tmap(&tmA);
      tc::prefetch_tmap(&tmB);
      uint32_t issued = 0;           // stages loaded so far
      bool aborted = false;
      for (uint32_t w = blockIdx.x; w < items && !aborted; w += gridDim.x) {
        const Item it = item_at<NT>(g, w);
        if (*vstatus != 0) {         // an error elsewhere: the other warps see it in their waits
          aborted = true;
          break;
        }
        for (int kt = 0; kt < it.stages; ++kt) {
          const uint32_t s = issued % STAGES, use = issued / STAGES;
          if (use > 0 && !tc::mbar_wait_abortable(&empty_bar[s], (use - 1) & 1, WAIT_CYCLES, vstatus)) {
            atomicExch(g.status, PTN_ERR_TIMEOUT);
            aborted = true;
            break;
          }
          uint8_t* st = smem + s * STAGE_BYTES;
          tc::mbar_arrive_expect_tx(&full_bar[s], STAGE_BYTES);
          const int kx = (it.k0 + kt) * KS;
          for (int p = 0; p < 2 * L; ++p)
            tc::tma_load_3d(st + p * A_PLANE_BYTES, &tmA, &full_bar[s], kx, (int)it.m0, p);
          for (int b = 0; b < 3 * L; ++b)
            tc::tma_load_3d(st + A_STAGE_BYTES + b * B_BLOCK_BYTES, &tmB, &full_bar[s], kx, (int)it.n0, b);
          ++issued;
        }
      }
      if (aborted) {
        // Drain before the CTA gives up its shared memory: wait (bounded) for
        // the last load issued into each stage. A stage's phase for its last
        // use is the only one still to complete, so a completed one returns
        // at once.
        for (uint32_t s = 0; s < STAGES && s < issued; ++s)
          tc::mbar_wait(&full_bar[s], ((issued - 1 - s) / STAGES) & 1, WAIT_CYCLES);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // Each accumulation round goes into a fresh TMEM buffer (in turn); the
    // epilogue warps add the round's partial sum into FP32 registers. The
    // tensor-core accumulator loses precision in proportion to the number of
    // accumulations it absorbs, so this bounds that loss to one round.
    if (lane == 0) {
      const uint32_t idesc = tc::idesc_bf16(MT, 2 * NT);
      bool aborted = false, any_mma = false;
      uint32_t stage = 0, round = 0;
      for (uint32_t w = blockIdx.x; w < items && !aborted; w += gridDim.x) {
        const int stages = item_at<NT>(g, w).stages;
        for (int kt = 0; kt < stages; ++kt, ++stage) {
          const uint32_t s = stage % STAGES;
          const uint32_t b = round % NBUF, ub = round / NBUF;
          const bool round_start = (kt & 1) == 0;
          if (round_start && ub > 0 &&
              !tc::mbar_wait_abortable(&tempty_bar[b], (ub - 1) & 1, WAIT_CYCLES, vstatus)) {
            atomicExch(g.status, PTN_ERR_TIMEOUT);
            aborted = true;
            break;
          }
          if (!tc::mbar_wait_abortable(&full_bar[s], (stage / STAGES) & 1, WAIT_CYCLES, vstatus)) {
            atomicExch(g.status, PTN_ERR_TIMEOUT);
            aborted = true;
            break;
          }
          any_mma = true;
          tc::fence_after();
          const uint32_t sa = tc::smem_u32(smem + s * STAGE_BYTES);
          const uint32_t sb = sa + A_STAGE_BYTES;
          const uint32_t acc = tmem + b * ACC_COLS;
          bool first = round_start;
          // smallest split products first, the leading (0, 0) product last
#pragma unroll
          for (int lvl = L - 1; lvl >= 0; --lvl) {
#pragma unroll
            for (int i = 0; i <= lvl; ++i) {
              const int j = lvl - i;
              // A planes: 2i = Re level i, 2i+1 = Im level i.
              // B level j at sb + 3j*B_BLOCK: window [Br; Bi] at +1 block, [-Bi; Br] at +0.
              const uint64_t ar = tc::sdesc_sw32(sa + (2 * i) * A_PLANE_BYTES);
              const uint64_t ai = tc::sdesc_sw32(sa + (2 * i + 1) * A_PLANE_BYTES);
              const uint64_t bt = tc::sdesc_sw32(sb + (3 * j + 1) * B_BLOCK_BYTES);
              const uint64_t bb = tc::sdesc_sw32(sb + (3 * j) * B_BLOCK_BYTES);
              tc::mma_bf16(acc, ar, bt, idesc, first ? 0u : 1u);
              tc::mma_bf16(acc, ai, bb, idesc, 1u);
              first = false;
            }
          }
          tc::mma_commit(&empty_bar[s]);
          if (!round_start || kt == stages - 1) {
            tc::mma_commit(&tfull_bar[b]);
            ++round;
          }
        }
      }
      if (aborted && any_mma) {
        // every MMA this thread issued completes before TMEM is freed
        tc::mma_commit(&drain_bar);
        tc::mbar_wait(&drain_bar, 0, WAIT_CYCLES);
      }
    }
  } else {
    // ---------------- epilogue (warps 2 ...) ----------------
    const int q = warp & 3;                 // TMEM lane quarter of this warp
    const int c0 = ((warp - 2) >> 2) * EC;  // its columns
    const int row = q * 32 + lane;
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    uint32_t round = 0;
    bool ok = true;
    for (uint32_t w = blockIdx.x; w < items && ok; w += gridDim.x) {
      const Item it = item_at<NT>(g, w);
      const int nacc = (it.stages + 1) / 2;                // accumulation rounds
      const int64_t m = it.m0 + row, n0 = it.n0 + c0;
      int64_t* noff = noff_s[warp - 2];
      __syncwarp();                         // the tile before has been written
#pragma unroll
      for (int j = lane; j < EC; j += 32) noff[j] = n0 + j < g.N ? decode_off32(g.no, (uint32_t)(n0 + j)) : -1;
      __syncwarp();
      const int64_t moff = m < g.M ? decode_off32(g.mo, (uint32_t)m) : 0;
      float acc_re[EC], acc_im[EC];
#pragma unroll
      for (int i = 0; i < EC; ++i) {
        acc_re[i] = 0.f;
        acc_im[i] = 0.f;
      }
      for (int a = 0; a < nacc; ++a, ++round) {
        const uint32_t b = round % NBUF;
        ok = __all_sync(0xffffffffu,
                        tc::mbar_wait_abortable(&tfull_bar[b], (round / NBUF) & 1, WAIT_CYCLES, vstatus));
        if (!ok) break;
        tc::fence_after();
        const uint32_t tb = tmem + lane_off + b * ACC_COLS + (uint32_t)c0;
        // two loads in flight per wait (re and im of LC columns: 16, or 8 where eight
        // epilogue warps leave 168 registers a thread)
        constexpr int LC = NT > EC ? 8 : 16;
#pragma unroll
        for (int j0 = 0; j0 < EC; j0 += LC) {
          uint32_t vr[LC], vi[LC];
          tc::tmem_ld_nowait<LC>(tb + (uint32_t)j0, vr);
          tc::tmem_ld_nowait<LC>(tb + (uint32_t)(NT + j0), vi);
          tc::tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < LC; ++i) {
            acc_re[j0 + i] += __uint_as_float(vr[i]);
            acc_im[j0 + i] += __uint_as_float(vi[i]);
          }
        }
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&tempty_bar[b]);
      }
      if (!ok) {
        if (lane == 0) atomicExch(g.status, PTN_ERR_TIMEOUT);
        break;
      }
      const bool row_ok = m < g.M;
      if (g.splits > 1) {
        // this K range's FP32 partial sums; splitk_reduce_kernel adds the ranges
        float2* P = g.partial + ((int64_t)it.split * g.M + m) * g.N + n0;
        if (!row_ok) {
        } else if (g.store == ST_ROW4) {
#pragma unroll
          for (int i = 0; i < EC; i += 4)
            if (n0 + i < g.N)
              st_global_32(P + i, __float_as_uint(acc_re[i]), __float_as_uint(acc_im[i]),
                           __float_as_uint(acc_re[i + 1]), __float_as_uint(acc_im[i + 1]),
                           __float_as_uint(acc_re[i + 2]), __float_as_uint(acc_im[i + 2]),
                           __float_as_uint(acc_re[i + 3]), __float_as_uint(acc_im[i + 3]));
        } else {
#pragma unroll
          for (int i = 0; i < EC; ++i)
            if (n0 + i < g.N) P[i] = make_float2(acc_re[i], acc_im[i]);
        }
      } else if (g.out_kind == 0) {
        double2* C = static_cast<double2*>(g.C) + moff;
        if (!row_ok) {
        } else if (g.store == ST_ROW2) {
#pragma unroll
          for (int i = 0; i < EC; i += 2) {
            const int64_t no = noff[i];
            if (i % 8 == 0 && no < 0) break;
            if (no >= 0)
              asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(C + no), "d"((double)acc_re[i]),
                           "d"((double)acc_im[i]), "d"((double)acc_re[i + 1]), "d"((double)acc_im[i + 1])
                           : "memory");
          }
        } else {
#pragma unroll
          for (int i = 0; i < EC; ++i) {
            const int64_t no = noff[i];
            if (i % 8 == 0 && no < 0) break;
            if (no >= 0) C[no] = make_double2((double)acc_re[i], (double)acc_im[i]);
          }
        }
      } else {
        __nv_bfloat16* C = static_cast<__nv_bfloat16*>(g.C) + moff;
        switch (g.store) {
#define PTN_STORE(kind)                                                            \
  case kind:                                                                       \
    store_planes<L, kind>(C, g.c_plane, acc_re, acc_im, noff, row_ok);             \
    break;
          PTN_STORE(ST_ROW8)
          PTN_STORE(ST_ROW4)
          PTN_STORE(ST_ROW2)
          PTN_STORE(ST_PAIR4)
          PTN_STORE(ST_PAIR2)
          PTN_STORE(ST_PAIR)
#undef PTN_STORE
          default:
            store_planes<L, ST_ONE>(C, g.c_plane, acc_re, acc_im, noff, row_ok);
        }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(tmem, TMEM_COLS);
}

// ---- tensor maps ---------------------------------------------------------------------
// cuTensorMapEncodeTiled is fetched through the runtime's driver entry point so
// the library does not link libcuda (it still loads on a machine without a driver).
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  // initialised once, thread-safe (C++11 static initialisation)
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    return nullptr;
  }();
  return fn;
}

int make_map_3d(CUtensorMap* map, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1_bytes,
                uint64_t s2_bytes, uint32_t b0, uint32_t b1) {
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {s1_bytes, s2_bytes};
  cuuint32_t box[3] = {b0, b1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
  if (!enc) return PTN_ERR_LAUNCH;
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims,
                                      strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? PTN_OK : PTN_ERR_ARG;
}

// ---- conversions ---------------------------------------------------------------------
// x ~ out[0] + ... + out[L-1] in BF16 pieces. Only the first remainder needs
// double precision: x - bf16(x) is exact in FP64 (Sterbenz) and is rounded
// once to FP32 (error <= 2^-32 |x|, below the 2^-25 |x| the three pieces
// leave); the later pieces are split in FP32.
__device__ __forceinline__ void split_levels(double x, int L, __nv_bfloat16* out) {
  const __nv_bfloat16 b0 = __double2bfloat16(x);
  out[0] = b0;
  float r = (float)(x - (double)__bfloat162float(b0));
  for (int lv = 1; lv < L; ++lv) {
    const __nv_bfloat16 b = __float2bfloat16_rn(r);
    out[lv] = b;
    r -= __bfloat162float(b);
  }
}
// Values outside [2^-60, 2^120): the pieces may leave FP32's normal range.
template <int L>
__device__ __noinline__ void split_far(double x, uint32_t* out) {
  __nv_bfloat16 b[3];
  split_levels(x, L, b);
#pragma unroll
  for (int lv = 0; lv < L; ++lv) out[lv] = (uint32_t)__bfloat16_as_ushort(b[lv]);
}
// The same pieces with one instruction at FP64 rate, the conversion of the remainder,
// instead of five: a warp instruction of the FP64 pipe takes an SM 16 cycles, and the
// conversion of a 4.2 M entry vector with them 91 us where its traffic takes 17. The
// leading piece is the 53-bit mantissa rounded at its eighth bit in integers; the bits
// below, less one unit if it was rounded up, are the exact remainder.
// flip: 0, or the sign bit to convert -x.
template <int L>
__device__ __forceinline__ void split_bits(double x, uint32_t flip, uint32_t (&out)[L]) {
  const uint32_t h = (uint32_t)__double2hiint(x) ^ flip, lo = (uint32_t)__double2loint(x), ah = h & 0x7fffffffu;
  const int e = (int)(ah >> 20);
  if ((unsigned)(e - 963) >= 180u && (ah | lo) != 0u) {
    split_far<L>(__hiloint2double((int)h, (int)lo), out);
    return;
  }
  const bool zero = (ah | lo) == 0u;
  const uint32_t tail = ah & 0x1fffu;
  const uint32_t up = (tail > 0x1000u || (tail == 0x1000u && (lo != 0u || (ah & 0x2000u)))) ? 1u : 0u;
  // exponent rebased to FP32's, above the seven mantissa bits that are kept
  const uint32_t b0 = zero ? 0u : (ah >> 13) - (896u << 7) + up;
  out[0] = b0 | (h >> 31 << 15);
  const int rh = (int)tail - (int)(up << 13);
  const long long rem = ((long long)rh << 32) | lo;
  // times 2^(e - 1075) with x's sign; an exact zero stays +0
  const float scale = __uint_as_float(((uint32_t)(e - 948) << 23) | (h & 0x80000000u));
  float r = zero || rem == 0 ? 0.f : __ll2float_rn(rem) * scale;
#pragma unroll
  for (int lv = 1; lv < L; ++lv) out[lv] = take_bf16(r);
}

// The pieces of two neighbouring entries, one word per level.
template <int L>
__device__ __forceinline__ void split_pair(double x, double y, uint32_t flip, uint32_t (&w)[L]) {
  uint32_t a[L], b[L];
  split_bits<L>(x, flip, a);
  split_bits<L>(y, flip, b);
#pragma unroll
  for (int lv = 0; lv < L; ++lv) w[lv] = a[lv] | b[lv] << 16;
}

struct ConvArgs {
  const double2* src;
  OutModes rm, km;               // rows and K index of the operand
  int64_t rows, K, ld, plane;
  int conj;
  int words;                     // rows and planes start on 4 bytes
  int64_t kstep;                 // source step from an even K index to the next, 0: look it up
  __nv_bfloat16* dst;
};
// V (2 or 4) entries of row r from K index k into the operand's layout: 2 L planes of A
// (Re_0, Im_0, ...) or, EXPAND, B's blocks [level][-Bi, Br, Bi][row][k]. With V = 2 the
// second may lie past the end, and rows may start on 2 bytes.
template <int L, bool EXPAND, int V>
__device__ __forceinline__ void put_split(const ConvArgs& c, int64_t r, int64_t k, const double2 (&v)[V]) {
  uint32_t re[V / 2][L], im[V / 2][L];
  const uint32_t flip = c.conj ? 0x80000000u : 0u;
#pragma unroll
  for (int i = 0; i < V / 2; ++i) {
    split_pair<L>(v[2 * i].x, v[2 * i + 1].x, 0u, re[i]);
    split_pair<L>(v[2 * i].y, v[2 * i + 1].y, flip, im[i]);
  }
  __nv_bfloat16* p = c.dst + r * c.ld + k;
  const int64_t blk = EXPAND ? c.rows * c.ld : c.plane;
  auto put = [&](int64_t plane, uint32_t a, uint32_t b) {
    __nv_bfloat16* q = p + plane * blk;
    if (V == 4) {
      *reinterpret_cast<uint2*>(q) = make_uint2(a, b);
    } else if (c.words && k + 1 < c.K) {
      *reinterpret_cast<uint32_t*>(q) = a;
    } else {
      q[0] = __ushort_as_bfloat16((unsigned short)a);
      if (k + 1 < c.K) q[1] = __ushort_as_bfloat16((unsigned short)(a >> 16));
    }
  };
#pragma unroll
  for (int lv = 0; lv < L; ++lv) {
    const uint32_t r0 = re[0][lv], r1 = re[V / 2 - 1][lv], i0 = im[0][lv], i1 = im[V / 2 - 1][lv];
    if (EXPAND) {
      put(3 * lv, i0 ^ 0x80008000u, i1 ^ 0x80008000u);
      put(3 * lv + 1, r0, r1);
      put(3 * lv + 2, i0, i1);
    } else {
      put(2 * lv, r0, r1);
      put(2 * lv + 1, i0, i1);
    }
  }
}

// planes[p][m * lda + k] <- split(src[off_m(m) + off_k(k)]); a thread takes two
// neighbouring K indices, or four where rows and K runs allow 8-byte stores. WIDE:
// 64-bit indices.
template <bool WIDE>
__device__ __forceinline__ int64_t mode_off(const OutModes& md, int64_t idx) {
  return WIDE ? decode_off(md, idx) : decode_off32(md, (uint32_t)idx);
}
template <int L, bool EXPAND, bool WIDE, int V>
__global__ void __launch_bounds__(256) convert_kernel(const ConvArgs c) {
  using I = typename std::conditional<WIDE, int64_t, uint32_t>::type;
  const I kp = (I)((c.K + V - 1) / V), total = (I)c.rows * kp;
  for (I e = (I)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (I)gridDim.x * blockDim.x) {
    const I r = e / kp, k = V * (e - r * kp);
    const double2* src = c.src + mode_off<WIDE>(c.rm, r) + mode_off<WIDE>(c.km, k);
    double2 v[V];
    v[0] = src[0];
    if (V == 4 || c.kstep != 0) {
#pragma unroll
      for (int i = 1; i < V; ++i) v[i] = src[i * c.kstep];
    } else {
      v[1] = make_double2(0.0, 0.0);
      if ((int64_t)k + 1 < c.K) v[1] = c.src[mode_off<WIDE>(c.rm, r) + mode_off<WIDE>(c.km, (int64_t)k + 1)];
    }
    put_split<L, EXPAND, V>(c, r, k, v);
  }
}

// The same conversion through a 32 x 64 shared-memory tile, for operands
// whose rows are contiguous in the source while the K index is not (the first
// step of a matvec contracting the parent leg reads x with a stride of the
// whole rest of the tensor): the tile is read with the row index across the
// threads and written with the K index across them, so both sides coalesce.
// Measured, with split_bits: 32768 x 128 (the vector of a 3-leg site at bond 128) 90
// -> 40 us, 131072 x 256 687 -> 232 (940 MB), and along K 584 -> 216.
constexpr int TILE_K = 64;
template <int L, bool EXPAND, bool WIDE>
__global__ void __launch_bounds__(256) convert_tiled_kernel(const ConvArgs c) {
  __shared__ double2 tile[TILE_K][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t tiles_k = (c.K + TILE_K - 1) / TILE_K;
  const int64_t tiles = ((c.rows + 31) / 32) * tiles_k;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int64_t m0 = (t / tiles_k) * 32, k0 = (t - (t / tiles_k) * tiles_k) * TILE_K;
    const bool row = m0 + tx < c.rows;
    const double2* src = c.src + (row ? mode_off<WIDE>(c.rm, m0 + tx) : 0);
#pragma unroll
    for (int q = 0; q < TILE_K / 8; ++q) {
      const int64_t k = k0 + ty + 8 * q;
      tile[ty + 8 * q][tx] = row && k < c.K ? src[mode_off<WIDE>(c.km, k)] : make_double2(0.0, 0.0);
    }
    __syncthreads();
#pragma unroll
    for (int r = ty; r < 32; r += 8) {
      const int64_t m = m0 + r, k = k0 + 2 * tx;
      if (m < c.rows && k < c.K) {
        const double2 v[2] = {tile[2 * tx][r], tile[2 * tx + 1][r]};
        put_split<L, EXPAND, 2>(c, m, k, v);
      }
    }
    __syncthreads();
  }
}

// ---- skinny products on the CUDA cores ----------------------------------------------
// A product with K <= SMALLK_MAX_K (one 32-wide K tile) and N <= SMALLK_MAX_N
// (the contraction with a TTNO tensor over its bond and physical legs, K =
// w d = 10) does too little arithmetic per output for a tensor-core tile
// pipeline: its set-up per CTA dominates (65536 x 10 x 10 measured 60 us).
// Here one thread owns one row: it rebuilds A's row from the BF16 level planes,
// B (same operand layout, staged in shared memory) likewise, accumulates in
// FP32 as the tensor cores do, and writes through the same output modes; the
// cost is the operand traffic.
constexpr int64_t SMALLK_MAX_K = 32;
constexpr int64_t SMALLK_MAX_N = 128;
constexpr int SMALLK_T = 128;

// KK: the K of the instance (EXACT) or an upper bound with K read at run time;
// an exact K leaves no predicated-off steps in the unrolled K loops.
template <int KK, bool EXACT>
__global__ void __launch_bounds__(SMALLK_T)
    cgemm_smallk_kernel(const __nv_bfloat16* __restrict__ A, int64_t lda, int64_t a_plane,
                        const __nv_bfloat16* __restrict__ Bx, int64_t ldb, GemmArgs g, int L) {
  __shared__ float2 sB[SMALLK_MAX_N * KK];
  __shared__ int64_t noff[SMALLK_MAX_N];
  if (*(volatile int32_t*)g.status != 0) return;
  const int N = (int)g.N, K = EXACT ? KK : (int)g.K;
  const int64_t blk = (int64_t)N * ldb;
  for (int e = threadIdx.x; e < N * K; e += SMALLK_T) {
    const int n = e / K, kk = e - n * K;
    float re = 0.f, im = 0.f;
    for (int lv = 0; lv < L; ++lv) {
      re += __bfloat162float(Bx[(3 * lv + 1) * blk + (int64_t)n * ldb + kk]);
      im += __bfloat162float(Bx[(3 * lv + 2) * blk + (int64_t)n * ldb + kk]);
    }
    sB[n * KK + kk] = make_float2(re, im);
  }
  for (int n = threadIdx.x; n < N; n += SMALLK_T) noff[n] = decode_off(g.no, n);
  __syncthreads();
  for (int64_t m = blockIdx.x * (int64_t)SMALLK_T + threadIdx.x; m < g.M; m += (int64_t)gridDim.x * SMALLK_T) {
    float2 a[KK];
#pragma unroll
    for (int kk = 0; kk < KK; ++kk) {
      float re = 0.f, im = 0.f;
      if (EXACT || kk < K) {
        for (int lv = 0; lv < L; ++lv) {
          re += __bfloat162float(A[(2 * lv) * a_plane + m * lda + kk]);
          im += __bfloat162float(A[(2 * lv + 1) * a_plane + m * lda + kk]);
        }
      }
      a[kk] = make_float2(re, im);
    }
    const int64_t moff = decode_off(g.mo, m);
    for (int n = 0; n < N; ++n) {
      float cr = 0.f, ci = 0.f;
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) {
        if (EXACT || kk < K) {
          const float2 b = sB[n * KK + kk];
          cr = fmaf(a[kk].x, b.x, cr);
          cr = fmaf(-a[kk].y, b.y, cr);
          ci = fmaf(a[kk].x, b.y, ci);
          ci = fmaf(a[kk].y, b.x, ci);
        }
      }
      const int64_t o = moff + noff[n];
      if (g.out_kind == 0) {
        static_cast<double2*>(g.C)[o] = make_double2((double)cr, (double)ci);
      } else {
        __nv_bfloat16* C = static_cast<__nv_bfloat16*>(g.C);
        for (int lv = 0; lv < L; ++lv) {
          const __nv_bfloat16 rb = __float2bfloat16_rn(cr);
          const __nv_bfloat16 ib = __float2bfloat16_rn(ci);
          C[(2 * lv) * g.c_plane + o] = rb;
          C[(2 * lv + 1) * g.c_plane + o] = ib;
          cr -= __bfloat162float(rb);
          ci -= __bfloat162float(ib);
        }
      }
    }
  }
}

// d = a b + c in both halves of a register pair.
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  return (unsigned long long)__float_as_uint(y) << 32 | __float_as_uint(x);
}

// The same product for BF16-plane outputs whose rows come in adjacent pairs:
// thread t computes rows 2t and 2t + 1 and stores each plane entry of the pair
// as one 4-byte bf16x2 (the host checks that the innermost row mode has
// output stride 1 and an even extent and that every other stride is even, so
// the pair is adjacent and 4-byte aligned). Half the store instructions, and a
// warp writes 128 contiguous bytes per plane. Same arithmetic per output.
//
// 16777216 x 50 x 10 reads 2 GB and writes 10 GB (1.8 ms at the copy rate) and was bound
// by instruction issue: 2.72 ms. So both rows share an instruction (FP32 pairs), a pair's
// entries of a plane, contiguous where rows are KK apart (DENSE), come in 8-byte
// loads, and both rows of a piece are rounded together: 2.05 ms.
template <int KK, int L, bool DENSE>
__global__ void __launch_bounds__(SMALLK_T)
    cgemm_smallk_pair_kernel(const __nv_bfloat16* __restrict__ A, int64_t lda, int64_t a_plane,
                             const __nv_bfloat16* __restrict__ Bx, int64_t ldb, GemmArgs g) {
  __shared__ ulonglong2 sB[SMALLK_MAX_N * KK];       // (Re, Re), (Im, Im)
  __shared__ int64_t noff[SMALLK_MAX_N];
  if (*(volatile int32_t*)g.status != 0) return;
  const int N = (int)g.N;
  const int64_t blk = (int64_t)N * ldb;
  for (int e = threadIdx.x; e < N * KK; e += SMALLK_T) {
    const int n = e / KK, kk = e - n * KK;
    float re = 0.f, im = 0.f;
    for (int lv = 0; lv < L; ++lv) {
      re += __bfloat162float(Bx[(3 * lv + 1) * blk + (int64_t)n * ldb + kk]);
      im += __bfloat162float(Bx[(3 * lv + 2) * blk + (int64_t)n * ldb + kk]);
    }
    sB[n * KK + kk] = make_ulonglong2(pack2(re, re), pack2(im, im));
  }
  for (int n = threadIdx.x; n < N; n += SMALLK_T) noff[n] = decode_off32(g.no, (uint32_t)n);
  __syncthreads();
  const int64_t pairs = g.M / 2;
  for (int64_t pr = blockIdx.x * (int64_t)SMALLK_T + threadIdx.x; pr < pairs;
       pr += (int64_t)gridDim.x * SMALLK_T) {
    const int64_t m = 2 * pr;
    // row m in the low halves, row m + 1 in the high ones
    unsigned long long ax[KK], ay[KK], nay[KK];
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      float v0[KK], v1[KK];
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) v0[kk] = v1[kk] = 0.f;
#pragma unroll
      for (int lv = 0; lv < L; ++lv) {
        const __nv_bfloat16* p = A + (2 * lv + part) * a_plane + m * lda;
        if (DENSE) {
          uint32_t w[KK];                            // entries 2 i and 2 i + 1 of the 2 KK
#pragma unroll
          for (int i = 0; i < KK / 2; ++i) {
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(p) + i);
            w[2 * i] = u.x;
            w[2 * i + 1] = u.y;
          }
#pragma unroll
          for (int kk = 0; kk < KK; ++kk) {
            const uint32_t x = w[kk / 2], y = w[KK / 2 + kk / 2];
            v0[kk] += __uint_as_float(kk & 1 ? x & 0xffff0000u : x << 16);
            v1[kk] += __uint_as_float(kk & 1 ? y & 0xffff0000u : y << 16);
          }
        } else {
#pragma unroll
          for (int kk = 0; kk < KK; ++kk) {
            v0[kk] += __bfloat162float(p[kk]);
            v1[kk] += __bfloat162float(p[lda + kk]);
          }
        }
      }
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) {
        if (part == 0) {
          ax[kk] = pack2(v0[kk], v1[kk]);
        } else {
          ay[kk] = pack2(v0[kk], v1[kk]);
          nay[kk] = pack2(-v0[kk], -v1[kk]);
        }
      }
    }
    __nv_bfloat16* C = static_cast<__nv_bfloat16*>(g.C) + decode_off32(g.mo, (uint32_t)m);
    for (int n = 0; n < N; ++n) {
      unsigned long long cr = 0ull, ci = 0ull;
#pragma unroll
      for (int kk = 0; kk < KK; ++kk) {
        const ulonglong2 b = sB[n * KK + kk];
        cr = fma2(ax[kk], b.x, cr);
        cr = fma2(nay[kk], b.y, cr);
        ci = fma2(ax[kk], b.y, ci);
        ci = fma2(ay[kk], b.x, ci);
      }
      __nv_bfloat16* p = C + noff[n];
      float c[4] = {__uint_as_float((uint32_t)cr), __uint_as_float((uint32_t)(cr >> 32)),
                    __uint_as_float((uint32_t)ci), __uint_as_float((uint32_t)(ci >> 32))};
#pragma unroll
      for (int lv = 0; lv < L; ++lv)
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          const __nv_bfloat162 v = __floats2bfloat162_rn(c[2 * part], c[2 * part + 1]);
          *reinterpret_cast<__nv_bfloat162*>(p + (2 * lv + part) * g.c_plane) = v;
          if (lv + 1 < L) {
            c[2 * part] -= __low2float(v);
            c[2 * part + 1] -= __high2float(v);
          }
        }
    }
  }
}

// Whether the rows of a BF16-plane output come in adjacent, 4-byte aligned
// pairs (cgemm_smallk_pair_kernel).
static bool smallk_pairs_ok(const GemmArgs& g, int64_t M) {
  if (g.out_kind != 1 || M < 2 || M % 2 || g.mo.n < 1 || (g.c_plane & 1)) return false;
  if (g.mo.stride[g.mo.n - 1] != 1 || g.mo.dim[g.mo.n - 1] % 2) return false;
  for (int i = 0; i + 1 < g.mo.n; ++i)
    if (g.mo.stride[i] & 1) return false;
  for (int i = 0; i < g.no.n; ++i)
    if (g.no.stride[i] & 1) return false;
  return true;
}

// How the tensor-core kernel's epilogue may write this output.
static int store_kind(const GemmArgs& g) {
  const OutModes &m = g.mo, &n = g.no;
  auto all = [](const OutModes& o, int count, int64_t mult) {
    for (int i = 0; i < count; ++i)
      if (o.stride[i] % mult) return false;
    return true;
  };
  const uintptr_t base = reinterpret_cast<uintptr_t>(g.C);
  if (g.splits > 1) return g.N % 4 == 0 && reinterpret_cast<uintptr_t>(g.partial) % 32 == 0 ? ST_ROW4 : ST_ONE;
  if (n.n < 1 || m.n < 1) return ST_ONE;
  const int64_t ns = n.stride[n.n - 1], nd = n.dim[n.n - 1];
  if (g.out_kind == 0)
    return ns == 1 && nd % 2 == 0 && all(n, n.n - 1, 2) && all(m, m.n, 2) && base % 32 == 0 ? ST_ROW2 : ST_ONE;
  // stores of v entries: aligned, and no group of columns goes past a run
  auto fits = [&](int64_t v, int mcount, int64_t cols) {
    return g.c_plane % v == 0 && base % (2 * v) == 0 && all(n, n.n - 1, v) && all(m, mcount, v) &&
           (nd % cols == 0 || n.n == 1);
  };
  if (ns == 1) {
    if (fits(8, m.n, 8)) return ST_ROW8;
    if (fits(4, m.n, 4)) return ST_ROW4;
    if (fits(2, m.n, 2)) return ST_ROW2;
  }
  // rows in runs of 32 and more are written a whole sector at a time as they are
  // (131072 x 1280 x 256: 1.37 ms one by one, 1.59 in pairs)
  if (m.stride[m.n - 1] != 1 || m.dim[m.n - 1] % 2 || m.dim[m.n - 1] >= 32) return ST_ONE;
  if (ns == 2) {
    if (fits(8, m.n - 1, 8)) return ST_PAIR4;
    if (fits(4, m.n - 1, 4)) return ST_PAIR2;
  }
  return g.c_plane % 2 == 0 && base % 4 == 0 && all(m, m.n - 1, 2) && all(n, n.n, 2) ? ST_PAIR : ST_ONE;
}

// Sum of the split-K partial sums (compensated FP32, ranges in order: deterministic),
// written like the GEMM epilogue: complex128 through the output modes, or as
// BF16 level planes.
__global__ void splitk_reduce_kernel(const float2* __restrict__ partial, int splits, int64_t M, int64_t N,
                                     OutModes mo, OutModes no, int out_kind, void* C, int64_t c_plane, int L,
                                     const int32_t* __restrict__ status) {
  if (*status != 0) return;
  const int64_t total = M * N;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = e / N, n = e - (e / N) * N;
    // compensated (Kahan) sums in FP32, ranges in order: the FP32 pipe runs at
    // 64x the FP64 rate on GB300, and the compensation keeps the error at the
    // level of the partials' own rounding
    float sr = 0.f, si = 0.f, cr = 0.f, ci = 0.f;
    for (int s = 0; s < splits; ++s) {
      const float2 p = partial[((int64_t)s * M + m) * N + n];
      const float yr = p.x - cr, yi = p.y - ci;
      const float tr = sr + yr, ti = si + yi;
      cr = (tr - sr) - yr;
      ci = (ti - si) - yi;
      sr = tr;
      si = ti;
    }
    const double re = (double)sr - (double)cr, im = (double)si - (double)ci;
    const int64_t o = decode_off(mo, m) + decode_off(no, n);
    if (out_kind == 0) {
      static_cast<double2*>(C)[o] = make_double2(re, im);
    } else {
      __nv_bfloat16* Cb = static_cast<__nv_bfloat16*>(C);
      __nv_bfloat16 rb[3], ib[3];
      split_levels(re, L, rb);
      split_levels(im, L, ib);
      for (int lv = 0; lv < L; ++lv) {
        Cb[(2 * lv) * c_plane + o] = rb[lv];
        Cb[(2 * lv + 1) * c_plane + o] = ib[lv];
      }
    }
  }
}

// Split of the K range for an M x N x K product: (splits, K tiles per split).
void split_plan(int64_t M, int64_t N, int64_t K, int64_t& splits, int64_t& ksplit) {
  const int64_t tiles = ((M + MT - 1) / MT) * ((N + 63) / 64);
  const int64_t kt_all = (K + KT - 1) / KT;
  splits = 1;
  ksplit = kt_all;
  if (tiles >= SPLIT_TARGET_CTAS / 2 || kt_all < SPLIT_MIN_KT_TOTAL) return;
  int64_t s = (SPLIT_TARGET_CTAS + tiles - 1) / tiles;
  const int64_t smax = kt_all / SPLIT_MIN_KT;
  if (s > smax) s = smax;
  if (s < 2) return;
  ksplit = (kt_all + s - 1) / s;
  splits = (kt_all + ksplit - 1) / ksplit;
  if (splits < 2) {
    splits = 1;
    ksplit = kt_all;
  }
}

// A mode that continues the one before it is part of it.
void add_mode(OutModes& m, int64_t dim, int64_t stride) {
  if (dim == 1) return;
  if (m.n > 0 && m.stride[m.n - 1] == dim * stride) {
    m.dim[m.n - 1] *= dim;
    m.stride[m.n - 1] = stride;
    return;
  }
  m.dim[m.n] = dim;
  m.stride[m.n++] = stride;
}

int fill_out(const ptn_modes& src, OutModes& dst) {
  if (src.n < 0 || src.n > PTN_MAX_MODES) return PTN_ERR_ARG;
  dst.n = 0;
  for (int i = 0; i < src.n; ++i) {
    if (src.dim[i] <= 0) return PTN_ERR_ARG;
    add_mode(dst, src.dim[i], src.stride_c[i]);
  }
  return PTN_OK;
}

int fill_src(const ptn_modes& src, OutModes& dst, int64_t& total) {
  if (src.n < 0 || src.n > PTN_MAX_MODES) return PTN_ERR_ARG;
  dst.n = 0;
  total = 1;
  for (int i = 0; i < src.n; ++i) {
    if (src.dim[i] <= 0) return PTN_ERR_ARG;
    total *= src.dim[i];
    add_mode(dst, src.dim[i], src.stride_a[i]);
  }
  return PTN_OK;
}

unsigned grid_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b < 1) b = 1;
  if (b > 4096) b = 4096;
  return (unsigned)b;
}

}  // namespace

extern "C" int ptn_cgemm_smem_bytes(int32_t levels) {
  return levels == 3 ? max(Cfg<3, 64>::SMEM, Cfg<3, 128>::SMEM) : max(Cfg<2, 64>::SMEM, Cfg<2, 128>::SMEM);
}

extern "C" int64_t ptn_cgemm_partial_bytes(int64_t M, int64_t N, int64_t K) {
  if (M < 1 || N < 1 || K < 1) return 0;
  int64_t splits, ksplit;
  split_plan(M, N, K, splits, ksplit);
  return splits > 1 ? splits * M * N * (int64_t)sizeof(float2) : 0;
}

static int sm_count() {
  static const int n = []() {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      return 0;
    return v;
  }();
  return n;
}

template <int L, int NT>
static int launch_gemm(const ptn_cgemm_desc* d, GemmArgs& g, int64_t tm, cudaStream_t st) {
  // once per process, thread-safe; a failure is returned on every call
  static const cudaError_t attr = cudaFuncSetAttribute(
      cgemm_bf16_kernel<L, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<L, NT>::SMEM);
  const int n_sm = sm_count();
  if (attr != cudaSuccess || n_sm <= 0) return PTN_ERR_LAUNCH;
  CUtensorMap ta, tb;
  if (make_map_3d(&ta, d->A, (uint64_t)d->K, (uint64_t)d->M, 2 * L, (uint64_t)d->lda * 2,
                  (uint64_t)d->a_plane * 2, KS, MT))
    return PTN_ERR_ARG;
  if (make_map_3d(&tb, d->Bx, (uint64_t)d->K, (uint64_t)d->N, 3 * L, (uint64_t)d->ldb * 2,
                  (uint64_t)d->N * (uint64_t)d->ldb * 2, KS, NT))
    return PTN_ERR_ARG;
  const int64_t items = tm * ((d->N + NT - 1) / NT) * g.splits;
  if (items > 0x7fffffffLL - n_sm) return PTN_ERR_UNSUPPORTED;
  g.tiles_m = (int32_t)tm;
  g.items = (int32_t)items;
  PTN_COUNT(1);
  cgemm_bf16_kernel<L, NT><<<(unsigned)(items < n_sm ? items : n_sm), Cfg<L, NT>::THREADS, Cfg<L, NT>::SMEM, st>>>(
      ta, tb, g);
  if (g.splits > 1) {
    PTN_COUNT(1);
    splitk_reduce_kernel<<<grid_for(g.M * g.N), 256, 0, st>>>(g.partial, g.splits, g.M, g.N, g.mo, g.no,
                                                              g.out_kind, g.C, g.c_plane, L, g.status);
  }
  return ptn_launch_status();
}

extern "C" int ptn_cgemm_bf16x3(const ptn_cgemm_desc* d, void* stream) {
  if (!d || !d->A || !d->Bx || !d->C || !d->status) return PTN_ERR_ARG;
  if (d->M < 1 || d->N < 1 || d->K < 1) return PTN_ERR_ARG;
  if (d->levels != 2 && d->levels != 3) return PTN_ERR_ARG;
  // the CUDA-core path (K <= 32, N <= 128) reads A without TMA: any lda >= K
  const bool smallk = d->K <= SMALLK_MAX_K && d->N <= SMALLK_MAX_N;
  if ((!smallk && d->lda % 8) || d->ldb % 8 || d->lda < d->K || d->ldb < d->K) return PTN_ERR_ARG;
  if (d->a_plane % 8 || (reinterpret_cast<uintptr_t>(d->A) & 15) || (reinterpret_cast<uintptr_t>(d->Bx) & 15))
    return PTN_ERR_ARG;
  if (d->M > 0x7fffffffLL || d->N > 0x7fffffffLL) return PTN_ERR_UNSUPPORTED;
  GemmArgs g;
  g.M = d->M;
  g.N = d->N;
  g.K = d->K;
  g.out_kind = d->out_kind;
  g.C = d->C;
  g.c_plane = d->c_plane;
  g.status = d->status;
  if (fill_out(d->m_out, g.mo) || fill_out(d->n_out, g.no)) return PTN_ERR_ARG;
  if (smallk) {
    int64_t blocks = (d->M + SMALLK_T - 1) / SMALLK_T;
    if (blocks > 152 * 16) blocks = 152 * 16;
    PTN_COUNT(1);
    const __nv_bfloat16* A = static_cast<const __nv_bfloat16*>(d->A);
    const __nv_bfloat16* B = static_cast<const __nv_bfloat16*>(d->Bx);
    cudaStream_t st = ptn_stream(stream);
    if (smallk_pairs_ok(g, d->M)) {
      int64_t pb = (d->M / 2 + SMALLK_T - 1) / SMALLK_T;
      if (pb > 152 * 16) pb = 152 * 16;
      // a plane's entries of a pair in 8-byte words
      const bool dense = d->lda == d->K && d->a_plane % 4 == 0;
      switch (d->K) {
#define PTN_SMALLK_PAIR_L(k, l)                                                                            \
  if (dense) cgemm_smallk_pair_kernel<k, l, true><<<(unsigned)pb, SMALLK_T, 0, st>>>(A, d->lda, d->a_plane, \
                                                                                     B, d->ldb, g);         \
  else cgemm_smallk_pair_kernel<k, l, false><<<(unsigned)pb, SMALLK_T, 0, st>>>(A, d->lda, d->a_plane, B,   \
                                                                                d->ldb, g);
#define PTN_SMALLK_PAIR(k)            \
  case k:                             \
    if (d->levels == 3) {             \
      PTN_SMALLK_PAIR_L(k, 3)         \
    } else {                          \
      PTN_SMALLK_PAIR_L(k, 2)         \
    }                                 \
    return ptn_launch_status();
        PTN_SMALLK_PAIR(2)
        PTN_SMALLK_PAIR(4)
        PTN_SMALLK_PAIR(6)
        PTN_SMALLK_PAIR(10)
#undef PTN_SMALLK_PAIR
#undef PTN_SMALLK_PAIR_L
        default:
          break;
      }
    }
    switch (d->K) {
#define PTN_SMALLK_CASE(k)                                                                              \
  case k:                                                                                               \
    cgemm_smallk_kernel<k, true><<<(unsigned)blocks, SMALLK_T, 0, st>>>(A, d->lda, d->a_plane, B, d->ldb, g, \
                                                                        d->levels);                     \
    break;
      PTN_SMALLK_CASE(2)
      PTN_SMALLK_CASE(3)
      PTN_SMALLK_CASE(4)
      PTN_SMALLK_CASE(5)
      PTN_SMALLK_CASE(6)
      PTN_SMALLK_CASE(8)
      PTN_SMALLK_CASE(10)
      PTN_SMALLK_CASE(12)
      PTN_SMALLK_CASE(16)
      PTN_SMALLK_CASE(20)
#undef PTN_SMALLK_CASE
      default:
        cgemm_smallk_kernel<(int)SMALLK_MAX_K, false><<<(unsigned)blocks, SMALLK_T, 0, st>>>(
            A, d->lda, d->a_plane, B, d->ldb, g, d->levels);
    }
    return ptn_launch_status();
  }
  int64_t splits = 1, ksplit = (d->K + KT - 1) / KT;
  if (d->partial) {
    int64_t s_, k_;
    split_plan(d->M, d->N, d->K, s_, k_);
    if (s_ > 1 && s_ * d->M * d->N * (int64_t)sizeof(float2) <= d->partial_bytes &&
        !(reinterpret_cast<uintptr_t>(d->partial) & 7)) {
      splits = s_;
      ksplit = k_;
    }
  }
  g.splits = (int32_t)splits;
  g.ksplit = (int32_t)ksplit;
  g.partial = static_cast<float2*>(d->partial);
  g.store = store_kind(g);
  // 128 columns or 64: the waves of the launch times a tile's cost. A tile of 128
  // columns takes about 1.5 times one of 64: 163840 x 256 x 1280 at 1500 TFLOP/s in wide
  // tiles, 131072 x 64 x 256 at 790 in narrow ones, of whose time a third is the start
  // and the end.
  const int64_t tm = (d->M + MT - 1) / MT;
  const int64_t n_sm = sm_count() > 0 ? sm_count() : 1;
  const int64_t w64 = (tm * ((d->N + 63) / 64) * splits + n_sm - 1) / n_sm;
  const int64_t w128 = (tm * ((d->N + 127) / 128) * splits + n_sm - 1) / n_sm;
  const bool wide = 3 * w128 < 2 * w64;
  cudaStream_t st = ptn_stream(stream);
  if (d->levels == 3) return wide ? launch_gemm<3, 128>(d, g, tm, st) : launch_gemm<3, 64>(d, g, tm, st);
  return wide ? launch_gemm<2, 128>(d, g, tm, st) : launch_gemm<2, 64>(d, g, tm, st);
}

template <int L, bool EXPAND>
static int convert(ConvArgs& c, cudaStream_t st) {
  // 32-bit indices unless they overflow (the grid's stride included)
  const bool wide = c.rows > 0x3fffffffLL || c.K > 0x3fffffffLL || c.rows * ((c.K + 1) / 2) > 0x7fffffffLL;
  const OutModes &rm = c.rm, &km = c.km;
  // innermost (fastest) source strides of the row and K indices
  const int64_t sr = rm.n > 0 ? rm.stride[rm.n - 1] : 0, sk = km.n > 0 ? km.stride[km.n - 1] : 0;
  const int64_t asr = sr < 0 ? -sr : sr, ask = sk < 0 ? -sk : sk;
  PTN_COUNT(1);
  // fewer tiles leave the GPU idle, and so small a source is read from L2 anyway
  // (40 x 40: 14 us tiled, 10 not; 512 x 256: 11 and 16)
  const int64_t tiles = ((c.rows + 31) / 32) * ((c.K + TILE_K - 1) / TILE_K);
  if (c.rows >= 32 && c.K >= 32 && asr <= 2 && ask > 2 && tiles >= 32) {
    const unsigned grid = (unsigned)(tiles < 152 * 16 ? tiles : 152 * 16);
    if (wide) convert_tiled_kernel<L, EXPAND, true><<<grid, 256, 0, st>>>(c);
    else convert_tiled_kernel<L, EXPAND, false><<<grid, 256, 0, st>>>(c);
    return ptn_launch_status();
  }
  // groups of K indices lie in one run of the innermost mode
  const int64_t run = km.n > 0 ? km.dim[km.n - 1] : 1;
  const bool four = run % 4 == 0 && c.ld % 4 == 0 && c.plane % 4 == 0 && reinterpret_cast<uintptr_t>(c.dst) % 8 == 0;
  const unsigned grid = grid_for(c.rows * ((c.K + (four ? 3 : 1)) / (four ? 4 : 2)));
  c.kstep = run % 2 == 0 ? sk : 0;
  if (wide) convert_kernel<L, EXPAND, true, 2><<<grid, 256, 0, st>>>(c);
  else if (four) convert_kernel<L, EXPAND, false, 4><<<grid, 256, 0, st>>>(c);
  else convert_kernel<L, EXPAND, false, 2><<<grid, 256, 0, st>>>(c);
  return ptn_launch_status();
}

static int convert_args(const ptn_convert_desc* d, ConvArgs& c) {
  if (!d || !d->src || !d->dst || (d->levels != 2 && d->levels != 3)) return PTN_ERR_ARG;
  if (fill_src(d->rows, c.rm, c.rows) || fill_src(d->cols, c.km, c.K)) return PTN_ERR_ARG;
  if (d->ld < c.K) return PTN_ERR_ARG;
  c.src = static_cast<const double2*>(d->src);
  c.dst = static_cast<__nv_bfloat16*>(d->dst);
  c.ld = d->ld;
  c.plane = d->plane;
  c.conj = d->conj;
  c.kstep = 0;
  c.words = d->ld % 2 == 0 && d->plane % 2 == 0 && reinterpret_cast<uintptr_t>(d->dst) % 4 == 0;
  return PTN_OK;
}

extern "C" int ptn_to_planes(const ptn_convert_desc* d, void* stream) {
  ConvArgs c;
  const int st = convert_args(d, c);
  if (st != PTN_OK) return st;
  return d->levels == 3 ? convert<3, false>(c, ptn_stream(stream)) : convert<2, false>(c, ptn_stream(stream));
}

extern "C" int ptn_expand_b(const ptn_convert_desc* d, void* stream) {
  ConvArgs c;
  const int st = convert_args(d, c);
  if (st != PTN_OK) return st;
  return d->levels == 3 ? convert<3, true>(c, ptn_stream(stream)) : convert<2, true>(c, ptn_stream(stream));
}
