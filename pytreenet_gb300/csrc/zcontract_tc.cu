// Complex128 contractions on the 5th-generation tensor cores, with every output held
// to its own terms as the FP64 kernels hold it.
//
// GB300 issues about two FP64 FMAs per clock per SM (1.25 TFLOP/s), a 900th of
// its bf16 tensor rate, so a contraction with enough arithmetic is done as
// exact integer products instead (the digit-slicing scheme of Ozaki, Ogita,
// Oishi and Rump, Numer. Algorithms 59, 2012): every row of A and of B is
// scaled by the power of two above its largest entry and rounded to a 63-bit
// fixed-point number, which is written in eight balanced base-256 digits in
// [-128, 128]. A digit is exact in bf16, the product of two is at most 2^14,
// and a K range of 64 adds at most 2^24 of them into one FP32 TMEM
// accumulator, so every tensor-core sum is an exact integer. The products
// d_i(A) d_j(B) of equal i + j share an accumulator (a "group"); groups 0..7
// are kept (36 digit pairs of the 64: group 8 is 2^-64 of the leading one),
// combined in 128-bit integers across the K range and rounded to double once.
//
// What is lost is about 2^-64 sqrt(K) of U, the product of the row's and the
// column's power of two. An FP64 sum loses 2^-53 of S = sum_k |a_mk| |b_kn| and more,
// which is less where an output's own terms are far below U: a row (1, 1e-18) against a
// column (0, 1). So a guard product of the magnitudes (ptn_zguard_kernel) finds S / U
// of every output, and those below 2^-9 are summed in FP64, in the same kernel. With
// seven digits, no headroom was left: one Gaussian entry in five alone in its sum
// (an identity part in the other operand) has S / U below 2^-3; below 2^-9 it is one
// in ten thousand. States whose rows fall off by many powers of two put more outputs
// there (graded by e^-0.3 k on two legs, a third to two thirds of the environment
// products; a Neel state, whose blocks hold rounding noise, a tenth to a half). They are
// taken one by one, by parts or by whole tiles without digits, whichever costs less
// (part_cost, one_cost), and at worst, all outputs in FP64, that takes as long as the
// FP64 kernels (40960 x 64 x 320 6.28 ms, 6.51 there; products of the Neel state 1966080
// x 50 x 50 44 and 47 ms, 5734400 x 15 x 75 65 and 189, 1966080 x 50 x 10 18 and 14).
//
// Before that, index k of both operands is balanced by a power of two (exact, on
// the exponents): the operand with fewer small entries is brought to one size
// along K, so that operands graded along k against each other (a factor and its
// inverse, the channels of a Hamiltonian) lose nothing, and a column with a single
// entry has this entry's size. The sizes of a long operand come from a sample of 64
// rows: a wrong estimate only puts more outputs below the guard's limit.
//
// MMA shape: digit i of A against the digits 0..J of B in one instruction
// stream: B's digits lie one below the other in shared memory ([Br; Bi], 64
// rows each), so the N = 64 (J + 1) columns of the product land in the
// accumulators of groups i..i + J, which are adjacent in TMEM. With 32 complex
// columns per tile eight groups fill TMEM (8 x 64 columns), and A's 4 KB plane
// is read from shared memory 12 times per 36 products instead of 36.
//
// Operands are written by ptn_zdigits_kernel as the images of the
// shared-memory stages (32-byte swizzle applied), so a stage is two contiguous
// bulk copies: no tensor maps, and no host work per call.
//
// Measured (M x N x K; FP64 kernels -> here, all launches): 8192 x 320 x 64
// 1326 -> 90 us, 40960 x 64 x 320 6505 -> 422 us, 262144 x 50 x 10 1873 -> 287
// us, 131072 x 256 x 256 55.8 -> 2.27 ms, 256 x 256 x 2560 2124 -> 134 us, 640 x
// 128 x 128 78 -> 58 us (seven digits without the guard: 78, 358, 218 us, 2.0 ms, 95,
// 46 us). Error against 64-bit mantissas (2-norm, Gaussian operands): 4.6e-17 to 1.6e-16
// for K = 10 to 65536, the FP64 kernels 1.4e-16 to 4.3e-15; largest error of an output
// by its own S, over those and operands of all sizes: 1.2e-16 where digits are kept, the
// FP64 kernels 2.3e-15.
//
// Rows that hold a NaN or an infinity are marked; their outputs are summed in
// FP64 too, so they propagate as in the FP64 kernels. Every wait is bounded; on a
// timeout the CTA's outputs become NaN.
#include <cuda_bf16.h>
#include <limits.h>

#include "ptn_common.cuh"
#include "tc_ptx.cuh"
#include "zmodes.cuh"

namespace {

constexpr int D = 8;                              // digits per operand
constexpr int G = 8;                              // accumulator groups kept
constexpr int TM = 128, TN = 32, KS = 16;         // tile rows, complex columns, K per stage
constexpr int CHUNK_STAGES = 4;                   // 64 K values: 8 pairs x 2 x 64 x 2^14 = 2^24
constexpr int A_STAGE = 2 * D * TM * KS * 2;      // 64 KB: planes Re_0, Im_0, Re_1, ...
constexpr int B_PLANE = TN * KS * 2;              // 1 KB
constexpr int B_STAGE = 4 * D * B_PLANE;          // 32 KB: [Br_j; Bi_j] by digit, then [-Bi_j; Br_j]
constexpr int STAGE = A_STAGE + B_STAGE;
constexpr int STAGES = 2;
constexpr int OUT_BYTES = 16 * 32 * 4 * 16;       // output staging of the epilogue warps
constexpr int SMEM = STAGES * STAGE + OUT_BYTES + 1024;
constexpr int FIRST_EPI = 4, EPI_WARPS = 16;      // warps 0: copies, 1: MMAs, 4..19: epilogue
constexpr int THREADS = 32 * (FIRST_EPI + EPI_WARPS);
constexpr int WC = TN / 4;                        // complex columns of an epilogue warp
constexpr int GROUP_COLS = 2 * TN;                // [Re | Im]
constexpr int GUARD = TM * KS * 2;                // 4 KB: a K step of magnitudes of 128 rows of A or of B
constexpr int GT = TM / TN;                       // column tiles that share a guard tile
constexpr int GUARD_KB = 8, GUARD_STAGES = 3;     // K steps a stage, stages of the guard kernel
constexpr int GUARD_SMEM = GUARD_STAGES * GUARD_KB * 2 * GUARD + 1024;
constexpr int GUARD_THREADS = 32 * 6;
constexpr int SAMPLES = 64;                       // rows of a long operand looked at for the balancing along K
constexpr int LOOK = 256;                         // threads that look at an index, rows up to which all are looked at
constexpr int FAR = 400;                          // rows and columns of larger and smaller exponents stay in FP64
constexpr int EMPTY = -FAR;                       // exponent of a row of zeros
constexpr int SPECIAL = INT_MAX;                  // exponent of a row with a NaN or an infinity
constexpr int NO_ENTRY = INT_MIN;                 // no entry of the row seen that is not zero
// K per split: the conversion's offset table (12 bytes a k) and its row maxima stay
// within the 48 KB of shared memory that a launch gets without asking for more.
constexpr int MAX_SPLIT_STAGES = 248;
static_assert(MAX_SPLIT_STAGES % CHUNK_STAGES == 0 && MAX_SPLIT_STAGES * KS * 12 + 128 * 4 + 64 <= 48 * 1024, "");
constexpr int64_t A_BYTES_MAX = 1ll << 30;        // digits of A held at once; more rows go in turns
// Complex multiply-adds from which scratch is asked for, and from which the digits are
// taken (on 128 x 32 tiles of few CTAs later than on many). In a queue of launches
// 4097 x 47 x 17 (3.3 M) takes 33 us here and on the FP64 kernels, 640 x 32 x 160
// (3.3 M, five tiles) 55 and 31, 2048 x 64 x 32 (4.2 M) 37 and 35, 640 x 128 x 128 (10 M)
// 47 and 76; by itself a call takes 10 us more here, 3 there.
constexpr int64_t PTN_ZTC_MIN_MACS = 3ll << 20;
constexpr int64_t PTN_ZTC_PAYS = 5ll << 20;
constexpr int64_t MIN_OUTPUTS = 256;              // fewer stay with the FP64 kernels
constexpr int64_t WORK_MAX = 8ll << 30;           // workspace a caller is asked for at most
constexpr long long WAIT_CYCLES = 4000000000LL;   // ~2 s at 2 GHz

struct Plan {
  bool swap;                // the roles of A and B exchanged
  int64_t M, N, K;
  int64_t stages;           // ceil(K / 16)
  int64_t tiles_m, tiles_n; // of the whole problem
  int64_t chunk_tiles;      // row tiles per turn
  int64_t splits, split_stages;
  int64_t off_ks, off_ea, off_eb, off_a, off_b, off_ga, off_gb, off_mask, off_cnt, off_sums, off_part, bytes;
};

// What the samples of both operands say of index k.
struct KStat {
  int a, b;                  // exponents of the powers of two above the largest entries (NO_ENTRY: all zero)
  int ca, cb;                // entries within 2^8 of them
};

struct DigitsArgs {
  const double2* src;
  ModeDev rows, ks;          // strides in s0
  int64_t nrows, K;
  int64_t row0;              // first row of this turn
  int64_t tiles;             // row tiles written
  int tile_rows;             // 128 (A) or 32 (B)
  int conj;
  const KStat* ks_stat;      // [K]
  int64_t na, nb, rows_a;    // rows of A and of B looked at for it, rows of A
  int kg;                    // groups of threads along K (power of two)
  int64_t stages, split_stages;
  uint8_t* dst;
  uint8_t* guard;            // magnitudes: [tile / (128 / tile_rows)][stage][128 rows][16]
  int* exps;                 // [splits][tiles * tile_rows]
  int64_t blocks_rows;       // CTAs along the rows
};

struct GemmArgs {
  ContractArgs c;            // m: (A, C) strides, n: (B, C), k: (A, B)
  const uint8_t* a;
  const uint8_t* b;
  const int* ea;
  const int* eb;
  int64_t m0;                // first row of this turn
  int64_t tiles, tiles_m, tiles_n;
  int64_t stages, split_stages;
  int32_t splits;
  double2* partial;          // [splits][rows of this turn][N]
  int64_t rows;
  int32_t* status;
  const uint32_t* mask;      // [tile][128 rows]: bit n set where output n of the tile is summed in FP64
  const int4* count;         // [tile]: their number, in four parts
  int32_t skip_tile;         // above which a tile takes no digits
};

struct GuardArgs {
  const uint8_t* a;
  const uint8_t* b;
  int64_t tiles_m, tiles_n;
  int64_t stages, split_stages;
  int32_t splits;
  float theta;
  uint32_t* mask;            // [tile][128 rows]
  int* count;                // [tile][4]
  float* sums;               // [item][32 columns][128 rows] when K is split, or null
  const int* ea;
  const int* eb;
  int32_t* status;
};

// ---- operands -> digits ----------------------------------------------------------
// Both operands' entries of each index k (one CTA per k): the largest and how many
// come near it; of B, and of A where it has few rows, all of them, of a longer A a
// sample, spread by the golden ratio, so that it meets every index of a tensor leg,
// whatever the dimensions. A thread looks at one row of each where it can: the time is
// the latency of decoding a row's place and of its load (one warp per k, eight loads to
// a lane, took 10 to 20 us; 4 so).
__device__ __forceinline__ int look_at(const DigitsArgs& q, int64_t ok, int64_t n, int64_t s) {
  if (s >= n) return 0;
  int64_t o, unused;
  decode(q.rows, n == q.nrows ? s : (int64_t)__umul64hi((unsigned long long)(s + 1) * 0x9E3779B97F4A7C15ull,
                                                        (unsigned long long)q.nrows), o, unused);
  const double2 v = q.src[ok + o];
  const int f = max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff) >> 20;
  return f == 0x7ff ? 0 : f;                         // zeros, denormals and what is not finite say nothing
}
__global__ void __launch_bounds__(LOOK) ptn_zksample_kernel(const DigitsArgs qa, const DigitsArgs qb,
                                                            KStat* __restrict__ out) {
  __shared__ int top[2], near[2];
  const int tid = threadIdx.x;
  const int64_t k = blockIdx.x;
  if (tid < 2) top[tid] = near[tid] = 0;
  int64_t oa, ob, unused;
  decode(qa.ks, k, oa, unused);
  decode(qb.ks, k, ob, unused);
  // the sample of A on the last threads, which have no row of a short B
  const int fa = look_at(qa, oa, qa.na, LOOK - 1 - tid);      // na <= LOOK
  const int fb = look_at(qb, ob, qa.nb, tid);
  int ta = __reduce_max_sync(0xffffffffu, fa), tb = fb;
  for (int64_t s = tid + LOOK; s < qa.nb; s += LOOK) tb = max(tb, look_at(qb, ob, qa.nb, s));
  tb = __reduce_max_sync(0xffffffffu, tb);
  __syncthreads();
  if ((tid & 31) == 0) {
    if (ta) atomicMax(&top[0], ta);
    if (tb) atomicMax(&top[1], tb);
  }
  __syncthreads();
  ta = top[0];
  tb = top[1];
  const int ca = __reduce_add_sync(0xffffffffu, fa != 0 && fa + 8 >= ta ? 1 : 0);
  int cb = fb != 0 && fb + 8 >= tb ? 1 : 0;
  for (int64_t s = tid + LOOK; s < qa.nb; s += LOOK) {
    const int f = look_at(qb, ob, qa.nb, s);
    cb += f != 0 && f + 8 >= tb ? 1 : 0;
  }
  cb = __reduce_add_sync(0xffffffffu, cb);
  if ((tid & 31) == 0) {
    if (ca) atomicAdd(&near[0], ca);
    if (cb) atomicAdd(&near[1], cb);
  }
  __syncthreads();
  if (tid == 0) out[k] = {ta ? ta - 1022 : NO_ENTRY, tb ? tb - 1022 : NO_ENTRY, near[0], near[1]};
}

// round(|x| 2^(63 - delta')) + 128 (256^0 + ... + 256^6), where the entry lies
// `delta` powers of two below the largest a row may hold: byte b of the result
// less 128 is digit 7 - b, byte 7 is digit 0 (0 to 128). 32-bit integer
// instructions only (about 20).
__device__ __forceinline__ void biased_digits(uint32_t xh, uint32_t xl, int delta, uint32_t& th, uint32_t& tl) {
  const int d1 = min(delta, 32), d2 = min(delta - d1, 32);
  // the mantissa at bit 63 (one bit below the last digit's), shifted down by delta
  uint32_t h = (xh & 0xfffffu) | 0x100000u, l = xl;
  h = __funnelshift_l(l, h, 11);
  l <<= 11;
  l = __funnelshift_rc(l, h, d1);
  h = __funnelshift_rc(h, 0u, d1);
  l = __funnelshift_rc(l, h, d2);
  h = __funnelshift_rc(h, 0u, d2);
  // one down, half units up, and the bias (the sum stays below 2^64)
  const uint32_t bl = 0x80808080u + (l & 1u), bh = 0x00808080u;
  l = __funnelshift_r(l, h, 1);
  h >>= 1;
  asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, %3;" : "+r"(l), "+r"(h) : "r"(bl), "r"(bh));
  tl = l;
  th = h;
}

// Digit d (1..7) of two biased numbers as a bf16 pair. With u the byte, u - 128
// is (128 + u mod 128) - (u >= 128 ? 128 : 256), all four exact in bf16 and
// made of u's bits.
__device__ __forceinline__ uint32_t digit_pair(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl, int d) {
  const int byte = D - 1 - d;                        // 0..6
  // the two bytes to bytes 0 and 2 (bytes 1 and 3 are masked off below)
  const uint32_t x = byte < 4 ? __byte_perm(al, bl, (uint32_t)byte | ((uint32_t)(byte + 4) << 8))
                              : __byte_perm(ah, bh, (uint32_t)(byte - 4) | ((uint32_t)byte << 8));
  const uint32_t p = (x & 0x007f007fu) | 0x43004300u, q = (x & 0x00800080u) ^ 0x43804380u;
  const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&p),
                                   *reinterpret_cast<const __nv_bfloat162*>(&q));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// Digit 0, in [0, 128].
__device__ __forceinline__ uint32_t top_pair(uint32_t ah, uint32_t bh) {
  const float a = __uint_as_float(0x4B000000u | (ah >> 24)) - 8388608.0f;   // 2^23
  const float b = __uint_as_float(0x4B000000u | (bh >> 24)) - 8388608.0f;
  const __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&r);
}

// One CTA: 128 / kg rows x one K split. Thread = (K group, row, half stage of 8
// K values). First the balancing of the split's K indices and the largest exponent
// of each row over the split, then the digits, eight K values (16 bytes per plane)
// at a time, and the guard's magnitudes; consecutive threads write consecutive
// 16-byte pieces of a plane. HBM / L2 bound: 16 bytes read (twice when a thread
// has more than one stage, the second time from L2) and 34 (A) or 66 (B) written
// per entry; the digit arithmetic is 32-bit integer and FP32 only, so that it does
// not wait for the FP64 pipe.
__global__ void __launch_bounds__(256, 3) ptn_zdigits_kernel(const DigitsArgs qa, const DigitsArgs qb,
                                                          const int64_t blocks_a, int32_t* status) {
  extern __shared__ int64_t koff[];                  // source offset of each k, then its exponent
  __shared__ int mx[128], least_a, least_b, thin;
  __shared__ unsigned long long near_a, near_b;
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
  const bool is_a = blockIdx.x < blocks_a;
  const DigitsArgs& q = is_a ? qa : qb;
  const int64_t blk = is_a ? blockIdx.x : blockIdx.x - blocks_a;
  const int64_t split = blk / q.blocks_rows;
  const int rpc = 128 / q.kg;
  const int64_t r_base = (blk - split * q.blocks_rows) * rpc;
  const int64_t st0 = split * q.split_stages;
  const int nst = (int)(min(q.stages, st0 + q.split_stages) - st0);
  const int tid = threadIdx.x;
  int* kx = reinterpret_cast<int*>(koff + q.split_stages * KS);
  for (int e = tid; e < rpc; e += 256) mx[e] = NO_ENTRY;
  if (tid == 0) {
    near_a = near_b = 0ull;
    least_a = least_b = INT_MAX;
    thin = 0;
  }
  __syncthreads();
  // The operand with fewer small entries is brought to one size along K, so that a
  // row of the other one that has a single entry (the identity part of an
  // environment) has this entry's size. A sample of A counts where it is dense at
  // every index: a thin one may have missed the entry that matters. All CTAs of a
  // split come to the same result. An index without entries goes with the smallest.
  {
    unsigned ca = 0, cb = 0;
    int la = INT_MAX, lb = INT_MAX;
    bool few = false;
    for (int e = tid; e < nst * KS; e += 256) {
      const int64_t k = st0 * KS + e;
      if (k >= q.K) break;
      const KStat t = q.ks_stat[k];
      ca += t.ca;
      cb += t.cb;
      if (t.a != NO_ENTRY) la = min(la, t.a);
      if (t.b != NO_ENTRY) lb = min(lb, t.b);
      few |= t.a != NO_ENTRY && 4 * t.ca < q.na;
    }
    if (few && q.na != q.rows_a) thin = 1;
    ca = __reduce_add_sync(0xffffffffu, ca);
    cb = __reduce_add_sync(0xffffffffu, cb);
    la = __reduce_min_sync(0xffffffffu, la);
    lb = __reduce_min_sync(0xffffffffu, lb);
    if ((tid & 31) == 0) {
      atomicAdd(&near_a, (unsigned long long)ca);
      atomicAdd(&near_b, (unsigned long long)cb);
      atomicMin(&least_a, la);
      atomicMin(&least_b, lb);
    }
  }
  __syncthreads();
  const bool by_a = !thin && near_a * (unsigned long long)q.nb >= near_b * (unsigned long long)q.na;
  const int least = by_a ? least_a : least_b;
  for (int e = tid; e < nst * KS; e += 256) {
    const int64_t k = st0 * KS + e;
    int64_t o0 = -1, o1;
    int x = 0;
    if (k < q.K) {
      decode(q.ks, k, o0, o1);
      const KStat t = q.ks_stat[k];
      x = by_a ? t.a : t.b;
      if (x == NO_ENTRY) x = least == INT_MAX ? 0 : least;
      if (by_a == is_a) x = -x;
    }
    koff[e] = o0;
    kx[e] = x;
  }
  const int h = tid & 1, r = (tid >> 1) & (rpc - 1), g = (tid >> 1) / rpc;
  const int64_t lrow = r_base + r;                   // row within this turn
  const int64_t row = q.row0 + lrow;
  const bool valid = row < q.nrows;
  int64_t base = 0, unused;
  if (valid) decode(q.rows, row, base, unused);
  __syncthreads();

  double2 v[8];
  auto load = [&](int st) {
    const int64_t* ko = koff + st * KS + h * 8;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int64_t o = ko[u];
      v[u] = (valid && o >= 0) ? q.src[base + o] : make_double2(0.0, 0.0);
    }
  };
  // |x| 2^kx < 2^E for every entry of the row. Denormals have no digits: a row
  // without larger entries has E below -400 and is summed in FP64, as is one
  // whose denormals meet large entries of B.
  int top = NO_ENTRY;
  for (int st = g; st < nst; st += q.kg) {
    load(st);
    const int* kk = kx + st * KS + h * 8;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int hm = max(__double2hiint(v[u].x) & 0x7fffffff, __double2hiint(v[u].y) & 0x7fffffff);
      const int field = hm >> 20;
      int e = field - 1022 + kk[u];
      if (field == 0) {
        const int any = hm | __double2loint(v[u].x) | __double2loint(v[u].y);
        e = any == 0 ? NO_ENTRY : (kk[u] > 500 ? SPECIAL : e);
      }
      if (field == 0x7ff) e = SPECIAL;
      top = max(top, e);
    }
  }
  if (top != NO_ENTRY) atomicMax(&mx[r], top);
  __syncthreads();
  const int E = mx[r] == NO_ENTRY ? EMPTY : mx[r];
  const int below = E == SPECIAL ? 4096 : E + 1022;  // digits of a special row are not used
  const int gbase = E == SPECIAL ? 77 : E + 896;     // a magnitude's exponent field is field + kx - gbase
  const int64_t padded = q.tiles * q.tile_rows;
  if (lrow >= padded) return;
  if (h == 0 && g == 0) q.exps[split * padded + lrow] = E;
  const int64_t tile = lrow / q.tile_rows;
  const int tr = (int)(lrow - tile * q.tile_rows);
  const int stage_bytes = is_a ? A_STAGE : B_STAGE;
  const int plane = q.tile_rows * KS * 2;
  const int within = tr * 32 + ((h ^ ((tr >> 2) & 1)) << 4);
  const int64_t gtile = is_a ? tile : tile / GT;
  const int gwithin = within + (is_a ? 0 : (int)(tile % GT) * B_PLANE);
  for (int st = g; st < nst; st += q.kg) {
    if (nst > q.kg) load(st);                        // otherwise still in registers
    uint8_t* out = q.dst + (tile * q.stages + st0 + st) * (int64_t)stage_bytes + within;
    const int* kk = kx + st * KS + h * 8;
    // magnitudes max(|Re|, |Im|) 2^(kx - E) for the guard, seven mantissa bits cut off;
    // at least 2^-50 where the entry is not zero, so that no product of two vanishes
    {
      uint32_t w[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int hm = max(__double2hiint(v[u].x) & 0x7fffffff, __double2hiint(v[u].y) & 0x7fffffff);
        const int ex = min((hm >> 20) + kk[u] - gbase, 254);
        const bool small = hm < 0x100000 || ex < 77;
        const bool zero = (hm | __double2loint(v[u].x) | __double2loint(v[u].y)) == 0;
        w[u] = zero ? 0u : (small ? 77u << 7 : (uint32_t)((ex << 7) | ((hm >> 13) & 0x7f)));
      }
      *reinterpret_cast<uint4*>(q.guard + (gtile * q.stages + st0 + st) * (int64_t)GUARD + gwithin) =
          make_uint4(w[0] | w[1] << 16, w[2] | w[3] << 16, w[4] | w[5] << 16, w[6] | w[7] << 16);
    }
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      uint32_t th[8], tl[8], sign[4];
      const uint32_t flip = part && q.conj ? 0x80000000u : 0u;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const double x = part ? v[u].y : v[u].x;
        const uint32_t xh = (uint32_t)__double2hiint(x) ^ flip;
        const int field = (int)(xh >> 20) & 0x7ff;
        // a zero has field 0 and is shifted out (E > -400 wherever digits count)
        const int delta = field == 0 ? 64 : below - field - kk[u];
        biased_digits(xh, (uint32_t)__double2loint(x), delta, th[u], tl[u]);
        if (u & 1) sign[u / 2] |= xh & 0x80000000u;
        else sign[u / 2] = xh >> 31 << 15;
      }
#pragma unroll
      for (int d = 0; d < D; ++d) {
        uint4 w;
        if (d == 0) {
          w.x = top_pair(th[0], th[1]);
          w.y = top_pair(th[2], th[3]);
          w.z = top_pair(th[4], th[5]);
          w.w = top_pair(th[6], th[7]);
        } else {
          w.x = digit_pair(th[0], tl[0], th[1], tl[1], d);
          w.y = digit_pair(th[2], tl[2], th[3], tl[3], d);
          w.z = digit_pair(th[4], tl[4], th[5], tl[5], d);
          w.w = digit_pair(th[6], tl[6], th[7], tl[7], d);
        }
        w.x ^= sign[0];
        w.y ^= sign[1];
        w.z ^= sign[2];
        w.w ^= sign[3];
        *reinterpret_cast<uint4*>(out + (2 * d + part) * plane) = w;
        if (!is_a) {
          // second window: [-Bi_j; Br_j]
          if (part) {
            w.x ^= 0x80008000u;
            w.y ^= 0x80008000u;
            w.z ^= 0x80008000u;
            w.w ^= 0x80008000u;
          }
          *reinterpret_cast<uint4*>(out + (2 * D + 2 * d + (1 - part)) * plane) = w;
        }
      }
    }
  }
}

// ---- products --------------------------------------------------------------------
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   tc::smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(tc::smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld2_nowait(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"(taddr)
               : "memory");
}

// acc + a b in 64 bits: one instruction where a shift and a 64-bit add are four.
__device__ __forceinline__ long long mad_wide(int a, int b, long long acc) {
  long long d;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(acc));
  return d;
}

// (H 2^32 + L) 2^sc for |sc| <= 900 (a result in the normal range), rounded to
// nearest in 32-bit integer arithmetic: a conversion or an addition on the FP64
// pipe costs as much as 64 of these instructions. The magnitude is formed in
// three words, normalised to bit 31 of the upper one, rounded at bit 11 of the
// middle one and packed.
__device__ __forceinline__ double fixed_to_double(long long H, uint32_t L, int sc) {
  const uint32_t sg = (uint32_t)(H >> 63);           // 0 or ~0
  uint32_t w2 = (uint32_t)((unsigned long long)H >> 32) ^ sg, w1 = (uint32_t)H ^ sg, w0 = L ^ sg;
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %2, %2, 0;"
      : "+r"(w0), "+r"(w1), "+r"(w2)
      : "r"(sg & 1u));
  int e = sc + 95 + 1022;                            // biased exponent of the leading bit, less one
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const bool z = w2 == 0u;
    w2 = z ? w1 : w2;
    w1 = z ? w0 : w1;
    w0 = z ? 0u : w0;
    e -= z ? 32 : 0;
  }
  const bool zero = w2 == 0u;
  const int lz = __clz((int)w2) & 31;
  w2 = __funnelshift_l(w1, w2, lz);
  w1 = __funnelshift_l(w0, w1, lz);
  uint32_t carry;                                    // w2 wraps when the mantissa rounds up to 2
  asm("add.cc.u32 %0, %0, 0x400;\n\taddc.cc.u32 %1, %1, 0;\n\taddc.u32 %2, 0, 0;"
      : "+r"(w1), "+r"(w2), "=r"(carry));
  // the mantissa's leading bit adds one to the exponent field
  const uint32_t m1 = ((w2 >> 11) + (carry << 21) + ((uint32_t)(e - lz) << 20)) | (sg & 0x80000000u);
  return __hiloint2double((int)(zero ? 0u : m1), (int)(zero ? 0u : __funnelshift_r(w1, w2, 11)));
}

__device__ __forceinline__ double2 finish(double2 alpha, double2 beta, int beta_zero, double2 v, const double2* p) {
  v = cmul(alpha, v);
  if (!beta_zero) v = cfma(beta, *p, v);
  return v;
}

// The guard of split sums: S of the ranges in units of the largest powers of two of
// the row and the column over all of them. One CTA per tile; a thread has a row and
// four columns.
__global__ void __launch_bounds__(1024) ptn_zguard_split_kernel(const GuardArgs g) {
  __shared__ uint32_t bits[TM];
  __shared__ int total;
  constexpr int CW = TN / 8;
  const int row = threadIdx.x & (TM - 1), c0 = (threadIdx.x / TM) * CW;
  const int64_t tile = blockIdx.x, tm = tile / g.tiles_n, tn = tile - tm * g.tiles_n;
  const int64_t tiles = g.tiles_m * g.tiles_n;
  if (threadIdx.x < TM) bits[threadIdx.x] = 0u;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  const int* ea = g.ea + tm * TM + row;
  const int* eb = g.eb + tn * TN + c0;
  int ra = INT_MIN, rb[CW];
  uint32_t far = 0u;                                 // columns, or all of them, that one range takes to FP64
#pragma unroll
  for (int c = 0; c < CW; ++c) rb[c] = INT_MIN;
  for (int s = 0; s < g.splits; ++s) {
    const int a = ea[s * g.tiles_m * TM];
    if (abs(a) > FAR) far = 0xffffffffu;
    ra = max(ra, a);
#pragma unroll
    for (int c = 0; c < CW; ++c) {
      const int b = eb[s * g.tiles_n * TN + c];
      if (abs(b) > FAR) far |= 1u << c;
      rb[c] = max(rb[c], b);
    }
  }
  float sum[CW];
#pragma unroll
  for (int c = 0; c < CW; ++c) sum[c] = 0.f;
  if (ra <= FAR) {
#pragma unroll 2
    for (int s = 0; s < g.splits; ++s) {
      const int da = ea[s * g.tiles_m * TM] - ra;
#pragma unroll
      for (int c = 0; c < CW; ++c) {
        const float f = g.sums[((s * tiles + tile) * TN + c0 + c) * TM + row];
        const int d = da + (rb[c] > FAR ? 0 : eb[s * g.tiles_n * TN + c] - rb[c]);
        // times 2^d; what underflows stays above zero
        if (f > 0.f) sum[c] += fmaxf(d > -100 ? f * __int_as_float((127 + d) << 23) : 0.f, 7.9e-31f);
      }
    }
  }
  uint32_t m = 0u;
#pragma unroll
  for (int c = 0; c < CW; ++c) m |= (far >> c & 1u) || (sum[c] > 0.f && sum[c] < g.theta) ? 1u << (c0 + c) : 0u;
  if (m) {
    atomicOr(&bits[row], m);
    atomicAdd(&total, __popc(m));
  }
  __syncthreads();
  if (threadIdx.x < TM) g.mask[tile * TM + threadIdx.x] = bits[threadIdx.x];
  if (threadIdx.x < 4) g.count[tile * 4 + threadIdx.x] = threadIdx.x == 0 ? total : 0;
}

__device__ __forceinline__ void plain_store(const GemmArgs& g, int64_t row_in_turn, int64_t n, int64_t om, int64_t on,
                                            int64_t split, double2 v) {
  if (g.splits > 1) {
    g.partial[(split * g.rows + row_in_turn) * g.c.N + n] = v;
  } else {
    double2* p = g.c.C + om + on;
    *p = finish(g.c.alpha, g.c.beta, g.c.beta_zero, v, p);
  }
}
// `count` listed outputs (row * WC + column of the part) of a warp, L lanes to each, which
// share K. (Four k of a lane in flight together: with one after the other, and all lanes
// on one output, K = 320 takes 20 us an output, 3 so.)
template <int L>
__device__ __noinline__ void plain_listed(const GemmArgs& g, uint32_t item, int part, const uint8_t* list, int count) {
  const uint32_t tiles = (uint32_t)g.tiles, s32 = item / tiles, tile = item - s32 * tiles;
  const uint32_t tm = tile / (uint32_t)g.tiles_n, tn = tile - tm * (uint32_t)g.tiles_n;
  const int64_t k0 = s32 * g.split_stages * KS, k1 = min(g.c.K, (s32 + 1) * g.split_stages * KS);
  const int lane = threadIdx.x & 31, sub = lane & (L - 1);
#pragma unroll 1
  for (int t = lane / L; t - lane / L < count; t += 32 / L) {
    const int e = list[min(t, count - 1)];
    const int64_t row_in_turn = (int64_t)tm * TM + (part & 3) * 32 + e / WC;
    const int64_t n = (int64_t)tn * TN + (part >> 2) * WC + e % WC;
    int64_t oa, om, ob, on;
    decode(g.c.m, g.m0 + row_in_turn, oa, om);
    decode(g.c.n, n, ob, on);
    double2 acc = make_double2(0.0, 0.0);
#pragma unroll 1
    for (int64_t kb = k0 + sub; kb - sub < k1; kb += 4 * L) {
      int64_t x[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) decode(g.c.k, min(kb + L * i, k1 - 1), x[i], y[i]);
      double2 av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        av[i] = g.c.A[oa + x[i]];
        bv[i] = g.c.B[ob + y[i]];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (kb - sub + L * i >= k1) break;           // the same in all lanes
        if (g.c.conj_a) av[i].y = -av[i].y;
        if (g.c.conj_b) bv[i].y = -bv[i].y;
        if (kb + L * i < k1) acc = cfma(av[i], bv[i], acc);
      }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
      acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if (sub == 0 && t < count) plain_store(g, row_in_turn, n, om, on, s32, acc);
  }
}
// NaN into part `part` of a tile (an epilogue warp's 32 rows x 8 columns), after a
// timeout. These functions are out of line, and without the digit sums, so that the
// common path keeps its registers.
__device__ __noinline__ void nan_part(const GemmArgs& g, uint32_t item, int part) {
  const uint32_t tiles = (uint32_t)g.tiles, s32 = item / tiles, tile = item - s32 * tiles;
  const uint32_t tm = tile / (uint32_t)g.tiles_n, tn = tile - tm * (uint32_t)g.tiles_n;
  const int64_t row_in_turn = (int64_t)tm * TM + (part & 3) * 32 + (threadIdx.x & 31);
  const int64_t n0 = (int64_t)tn * TN + (part >> 2) * WC;
  if (g.m0 + row_in_turn >= g.c.M) return;
  int64_t oa, om, ob, on;
  decode(g.c.m, g.m0 + row_in_turn, oa, om);
  for (int64_t n = n0; n < n0 + WC && n < g.c.N; ++n) {
    decode(g.c.n, n, ob, on);
    plain_store(g, row_in_turn, n, om, on, s32, make_double2(NAN, NAN));
  }
}

// A part's outputs (those in the lanes' `mm`) in FP64 through a warp's share of the stages' shared memory (they are
// done with): 16 k at a time, loaded with neighbouring lanes on neighbouring k. At the
// FP64 pipe's rate, where a loop over K waits for its operands (every output of 8192 x
// 320 x 64 1.71 ms with that, 1.27 so; of 40960 x 64 x 320 8.36 and 6.28).
constexpr int PK = 16;
static_assert((32 * (PK + 1) + WC * PK) * 16 * EPI_WARPS <= STAGES * STAGE, "");
__device__ __noinline__ void plain_part(const GemmArgs& g, uint32_t item, int part, uint32_t mm, double2* sm) {
  const int lane = threadIdx.x & 31, kk = lane & (PK - 1), hi = lane / PK;
  const uint32_t tiles = (uint32_t)g.tiles, s32 = item / tiles, tile = item - s32 * tiles;
  const uint32_t tm = tile / (uint32_t)g.tiles_n, tn = tile - tm * (uint32_t)g.tiles_n;
  const int64_t row_in_turn = (int64_t)tm * TM + (part & 3) * 32 + lane, m = g.m0 + row_in_turn;
  const int64_t n0 = (int64_t)tn * TN + (part >> 2) * WC;
  const int64_t k0 = s32 * g.split_stages * KS, k1 = min(g.c.K, (s32 + 1) * g.split_stages * KS);
  double2* As = sm;                                  // [32][PK + 1]
  double2* Bs = sm + 32 * (PK + 1);                  // [WC][PK]
  int64_t oa = -1, om = 0, ob = -1, on, x, y;
  if (m < g.c.M) decode(g.c.m, m, oa, om);
  if (lane < WC && n0 + lane < g.c.N) decode(g.c.n, n0 + lane, ob, on);
  double2 acc[WC];
#pragma unroll
  for (int c = 0; c < WC; ++c) acc[c] = make_double2(0.0, 0.0);
  for (int64_t kb = k0; kb < k1; kb += PK) {
    const bool in = kb + kk < k1;
    x = y = 0;
    if (in) decode(g.c.k, kb + kk, x, y);
    __syncwarp();                                    // the block before has been read
#pragma unroll 4
    for (int r = hi; r < 32; r += 32 / PK) {
      const int64_t o = __shfl_sync(0xffffffffu, (long long)oa, r);
      double2 v = make_double2(0.0, 0.0);
      if (in && o >= 0) v = g.c.A[o + x];
      if (g.c.conj_a) v.y = -v.y;
      As[r * (PK + 1) + kk] = v;
    }
#pragma unroll
    for (int c = hi; c < WC; c += 32 / PK) {
      const int64_t o = __shfl_sync(0xffffffffu, (long long)ob, c);
      double2 v = make_double2(0.0, 0.0);
      if (in && o >= 0) v = g.c.B[o + y];
      if (g.c.conj_b) v.y = -v.y;
      Bs[c * PK + kk] = v;
    }
    __syncwarp();
#pragma unroll 1
    for (int k = 0; k < PK; ++k) {
      const double2 a = As[lane * (PK + 1) + k];
#pragma unroll
      for (int c = 0; c < WC; ++c) acc[c] = cfma(a, Bs[c * PK + k], acc[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < WC; ++c)
    if (m < g.c.M && n0 + c < g.c.N && (mm >> c & 1u)) {
      decode(g.c.n, n0 + c, ob, on);
      plain_store(g, row_in_turn, n0 + c, om, on, s32, acc[c]);
    }
}

// What a listed output and all of a part (32 rows x 8 columns) take, in quarters of an
// FP64 instruction of a warp: the measure by which marked outputs are taken one by one, by
// parts, or by whole tiles without digits. A listed output takes three times its
// instructions, it waits for its operands (40960 x 64 x 320 with most of the outputs
// marked 10.3 ms where all that cost less by instructions were listed, 6.3 by parts;
// 998400 x 15 x 75 with two in five marked 32 and 12).
constexpr int64_t LONG_K = 512;                      // eight lanes to an output up to here, 32 above
__host__ __device__ constexpr int64_t one_cost(int64_t K) {
  return 3 * (K > LONG_K ? 4 * ((K + 31) / 32 * 4 + 10) : (K + 7) / 8 * 4 + 6);
}
__host__ __device__ constexpr int64_t part_cost(int64_t K) { return 4 * 4 * WC * K; }

__device__ __forceinline__ int marked_in(const GemmArgs& g, uint32_t tile) {
  const int4 c = g.count[tile];
  return c.x + c.y + c.z + c.w;
}
// Whether all of a tile is summed in FP64: the same for its copies, MMAs and epilogue.
__device__ __forceinline__ bool skips_digits(const GemmArgs& g, uint32_t tile) {
  return marked_in(g, tile) > g.skip_tile;
}

// The guard's outputs, after the digits: the parts of all tiles that have some are dealt
// out to the epilogue warps of all CTAs, one part of a tile to a CTA, so that the FP64
// pipes have equal shares.
__device__ __noinline__ void plain_tiles(const GemmArgs& g, uint8_t* smem, bool failed) {
  const uint32_t tiles = (uint32_t)g.tiles, parts = tiles * (uint32_t)g.splits * EPI_WARPS;   // items fit 27 bits
  const uint32_t stride = gridDim.x * EPI_WARPS, lane = threadIdx.x & 31, ew = (threadIdx.x >> 5) - FIRST_EPI;
  for (uint32_t p0 = ew * gridDim.x + blockIdx.x; p0 < parts; p0 += 32u * stride) {
    const uint32_t mine = p0 + lane * stride;        // a lane looks at one part
    uint32_t todo = __ballot_sync(0xffffffffu, mine < parts && marked_in(g, mine / EPI_WARPS % tiles) > 0);
    for (; todo; todo &= todo - 1u) {
      const uint32_t u = p0 + (uint32_t)(__ffs((int)todo) - 1) * stride, item = u / EPI_WARPS, tile = item % tiles;
      const int part = (int)(u % EPI_WARPS);
      const bool skipped = skips_digits(g, tile);
      const uint32_t row = (uint32_t)(part & 3) * 32u + lane, c0 = (uint32_t)(part >> 2) * WC;
      if (failed) {
        nan_part(g, item, part);
        continue;
      }
      const uint32_t split = item / tiles, tm = tile / (uint32_t)g.tiles_n, tn = tile - tm * (uint32_t)g.tiles_n;
      const int64_t cols = g.c.N - ((int64_t)tn * TN + c0);
      uint32_t mm = cols >= WC ? 0xffu : (cols > 0 ? (1u << (int)cols) - 1u : 0u);
      if (g.m0 + (int64_t)tm * TM + row >= g.c.M) mm = 0u;
      if (!skipped) mm &= g.mask[(int64_t)tile * TM + row] >> c0;
      if (!__any_sync(0xffffffffu, mm != 0u)) continue;
      const int64_t st0 = split * g.split_stages, K = (min(g.stages, st0 + g.split_stages) - st0) * KS;
      if (__reduce_add_sync(0xffffffffu, (unsigned)__popc(mm)) * one_cost(K) > part_cost(K)) {
        plain_part(g, item, part, mm,
                   reinterpret_cast<double2*>(smem) + ew * (STAGES * STAGE / 16 / EPI_WARPS));
        continue;
      }
      const int count = __popc(mm);
      int before = count;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, before, o);
        if ((int)lane >= o) before += t;
      }
      const int total = __shfl_sync(0xffffffffu, before, 31);
      uint8_t* list = smem + ew * (STAGES * STAGE / EPI_WARPS);
      __syncwarp();                                  // the list before has been read
      for (uint8_t* p = list + (before - count); mm; mm &= mm - 1u) *p++ = (uint8_t)(lane * WC + __ffs((int)mm) - 1);
      __syncwarp();
      if (K > LONG_K) plain_listed<32>(g, item, part, list, total);
      else plain_listed<8>(g, item, part, list, total);
    }
  }
}

__device__ __forceinline__ void mma_cols(uint32_t acc, uint32_t sa, uint32_t sb, int col, int ncols, bool overwrite,
                                         int group) {
  // columns [col, col + ncols) of the window at sb into the accumulators from group on
  tc::mma_bf16(acc + (uint32_t)(group * GROUP_COLS + col), tc::sdesc_sw32(sa), tc::sdesc_sw32(sb + (uint32_t)col * 32u),
               tc::idesc_bf16(TM, ncols), overwrite ? 0u : 1u);
}

// Digits of one stage: A digit i against the window of B digits 0..J.
__device__ __forceinline__ void mma_stage(uint32_t acc, uint32_t sa, uint32_t sb, bool first) {
#pragma unroll
  for (int part = 0; part < 2; ++part) {             // Ar with [Br; Bi], Ai with [-Bi; Br]
    const uint32_t b = sb + (uint32_t)part * 2u * D * B_PLANE;
    const bool ow = first && part == 0;
#pragma unroll
    for (int i = 0; i < D; ++i) {
      const uint32_t a = sa + (uint32_t)(2 * i + part) * (TM * KS * 2);
      const int cols = GROUP_COLS * (G - i);         // digit 0 starts all groups
      if (cols > 256) {
        const int half = cols / 2;                   // 256, 224, 192, 160: multiples of 16
        mma_cols(acc, a, b, 0, half, ow && i == 0, i);
        mma_cols(acc, a, b, half, cols - half, ow && i == 0, i);
      } else {
        mma_cols(acc, a, b, 0, cols, false, i);
      }
    }
  }
}

// Which outputs the digits do not hold to FP64: S = sum_k |a_mk| |b_kn| in units of
// the row's and the column's power of two, one BF16 product of the magnitudes (1/36
// of the digits' work, 3 to 15 us). The digits leave an error of about 2^-64 sqrt(K) of those
// units, an FP64 sum one of 2^-53 S or more; where 0 < S < theta the output is summed
// in FP64 (S = 0: all its terms are zero). Tiles of 128 x 128, a bit per output into
// `mask`, by tile of the digit products. Where K is split the units are those of a
// range, whose sum alone may be next to nothing: ptn_zguard_split_kernel adds the
// ranges first.
__global__ void __launch_bounds__(GUARD_THREADS, 1) ptn_zguard_kernel(const GuardArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[GUARD_STAGES], empty_bar[GUARD_STAGES], tfull_bar[2], tempty_bar[2], drain_bar;
  __shared__ uint32_t tmem_base;
  constexpr int SB = GUARD_KB * 2 * GUARD;           // A's K steps, then B's
  const volatile int32_t* vstatus = g.status;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t groups = (uint32_t)((g.tiles_n + GT - 1) / GT), per = (uint32_t)g.tiles_m * groups;
  const uint32_t items = per * (uint32_t)g.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < GUARD_STAGES; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&tfull_bar[b], 1);
      tc::mbar_init(&tempty_bar[b], 4);
    }
    tc::mbar_init(&drain_bar, 1);
    tc::fence_mbar_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(&tmem_base, 2 * TM);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_base;

  if (warp == 0) {
    if (lane == 0) {
      int it = 0;                                    // stages issued so far
      bool go = true;
      for (uint32_t w = blockIdx.x; w < items && go; w += gridDim.x) {
        const uint32_t split = w / per, t = w - split * per, tm = t / groups, gn = t - tm * groups;
        const int64_t st0 = split * g.split_stages;
        const int nst = (int)(min(g.stages, st0 + g.split_stages) - st0);
        const uint8_t* a = g.a + (tm * g.stages + st0) * (int64_t)GUARD;
        const uint8_t* b = g.b + (gn * g.stages + st0) * (int64_t)GUARD;
        for (int st = 0; st < nst; st += GUARD_KB, ++it) {
          const int s = it % GUARD_STAGES, use = it / GUARD_STAGES;
          if (use > 0) go = tc::mbar_wait_abortable(&empty_bar[s], (use - 1) & 1, WAIT_CYCLES, vstatus);
          if (!go) break;
          const uint32_t bytes = (uint32_t)min(GUARD_KB, nst - st) * GUARD;
          uint8_t* dst = smem + s * SB;
          tc::mbar_arrive_expect_tx(&full_bar[s], 2 * bytes);
          bulk_load(dst, a + (int64_t)st * GUARD, bytes, &full_bar[s]);
          bulk_load(dst + GUARD_KB * GUARD, b + (int64_t)st * GUARD, bytes, &full_bar[s]);
        }
      }
      if (!go) {
        atomicExch(g.status, PTN_ERR_TIMEOUT);
        for (int s = 0; s < GUARD_STAGES && s < it; ++s)
          tc::mbar_wait(&full_bar[s], (uint32_t)(((it - 1 - s) / GUARD_STAGES) & 1), WAIT_CYCLES);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int it = 0, acc = 0;
      bool go = true;
      for (uint32_t w = blockIdx.x; w < items && go; w += gridDim.x, ++acc) {
        const int64_t st0 = (w / per) * g.split_stages;
        const int nst = (int)(min(g.stages, st0 + g.split_stages) - st0);
        const uint32_t d = tmem + (uint32_t)((acc & 1) * TM);
        if (acc > 1) go = tc::mbar_wait_abortable(&tempty_bar[acc & 1], ((acc >> 1) - 1) & 1, WAIT_CYCLES, vstatus);
        for (int st = 0; st < nst && go; st += GUARD_KB, ++it) {
          const int s = it % GUARD_STAGES;
          go = tc::mbar_wait_abortable(&full_bar[s], (it / GUARD_STAGES) & 1, WAIT_CYCLES, vstatus);
          if (!go) break;
          tc::fence_after();
          const uint32_t sa = tc::smem_u32(smem + s * SB), sb = sa + GUARD_KB * GUARD;
          const int nk = min(GUARD_KB, nst - st);
          for (int k = 0; k < nk; ++k)
            tc::mma_bf16(d, tc::sdesc_sw32(sa + k * GUARD), tc::sdesc_sw32(sb + k * GUARD), tc::idesc_bf16(TM, TM),
                         st + k > 0 ? 1u : 0u);
          tc::mma_commit(&empty_bar[s]);
        }
        if (!go) break;
        tc::mma_commit(&tfull_bar[acc & 1]);
      }
      if (!go) {
        atomicExch(g.status, PTN_ERR_TIMEOUT);
        tc::mma_commit(&drain_bar);                  // every MMA issued ends before TMEM is freed
        tc::mbar_wait(&drain_bar, 0, WAIT_CYCLES);
      }
    }
  } else {
    const int q = warp & 3, row = q * 32 + lane;
    int acc = 0;
    for (uint32_t w = blockIdx.x; w < items; w += gridDim.x, ++acc) {
      const uint32_t split = w / per, t = w - split * per, tm = t / groups, gn = t - tm * groups;
      const bool ok = __all_sync(0xffffffffu, tc::mbar_wait_abortable(&tfull_bar[acc & 1], (acc >> 1) & 1,
                                                                      WAIT_CYCLES, vstatus));
      if (!ok) {
        if (lane == 0) atomicExch(g.status, PTN_ERR_TIMEOUT);
        break;
      }
      tc::fence_after();
      const uint32_t src = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((acc & 1) * TM);
      uint32_t bits[GT];
      const int64_t item0 = (split * g.tiles_m + tm) * g.tiles_n + (int64_t)gn * GT;
      const bool far_row = abs(g.ea[(split * g.tiles_m + tm) * TM + row]) > FAR;
#pragma unroll
      for (int j = 0; j < GT; ++j) {
        uint32_t v[2][16];
        tc::tmem_ld16_nowait(src + (uint32_t)(j * TN), v[0]);
        tc::tmem_ld16_nowait(src + (uint32_t)(j * TN + 16), v[1]);
        tc::tmem_wait_ld();
        uint32_t m = 0u;
#pragma unroll
        for (int i = 0; i < TN; ++i) {
          const float f = __uint_as_float(v[i / 16][i % 16]);
          m |= f > 0.f && f < g.theta ? 1u << i : 0u;
        }
        if (g.sums && gn * GT + j < (uint32_t)g.tiles_n) {
#pragma unroll
          for (int i = 0; i < TN; ++i) g.sums[((item0 + j) * TN + i) * TM + row] = __uint_as_float(v[i / 16][i % 16]);
        }
        if (!g.sums && gn * GT + j < (uint32_t)g.tiles_n) {
          const bool far_col = abs(g.eb[(int64_t)(gn * GT + j) * TN + lane]) > FAR;
          const uint32_t cols = __ballot_sync(0xffffffffu, far_col);
          m |= far_row ? 0xffffffffu : cols;
        }
        bits[j] = m;
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&tempty_bar[acc & 1]);
#pragma unroll
      for (int j = 0; j < GT; ++j) {
        if (g.sums || gn * GT + j >= (uint32_t)g.tiles_n) break;
        g.mask[(item0 + j) * TM + row] = bits[j];
        const int cnt = __reduce_add_sync(0xffffffffu, __popc(bits[j]));
        if (lane == 0) g.count[(item0 + j) * 4 + q] = cnt;
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(tmem, 2 * TM);
}

// Persistent: a CTA takes the (tile, split) items blockIdx.x, + gridDim.x, ...
// One warp copies stages ahead, one issues MMAs, sixteen drain and write. TMEM
// holds one chunk of 64 K values, so MMAs wait while it is drained into
// registers; the conversion to double and the stores of an item then overlap
// the MMAs of the next. (One item per CTA measured 19 us at K = 16, most of it
// set-up, conversion and stores with the tensor pipe idle.)
// UNIT: alpha = 1, beta = 0 (no FP64 instruction in the common path).
template <bool UNIT>
__global__ void __launch_bounds__(THREADS, 1) ptn_zgemm_digits_kernel(const GemmArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], tfull_bar, tempty_bar, drain_bar;
  __shared__ uint32_t tmem_base;
  const volatile int32_t* vstatus = g.status;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tiles = (uint32_t)g.tiles, tiles_n = (uint32_t)g.tiles_n;     // items fit 31 bits
  const uint32_t items = tiles * (uint32_t)g.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], 1);
    }
    tc::mbar_init(&tfull_bar, 1);
    tc::mbar_init(&tempty_bar, EPI_WARPS);
    tc::mbar_init(&drain_bar, 1);
    tc::fence_mbar_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(&tmem_base, G * GROUP_COLS);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_base;

  if (warp == 0) {
    // ---------------- copies: two contiguous pieces per stage ----------------
    if (lane == 0) {
      int it = 0;                                    // stages issued so far
      bool go = true;
      for (uint32_t w = blockIdx.x; w < items && go; w += gridDim.x) {
        const uint32_t split = w / tiles, tile = w - split * tiles;
        if (skips_digits(g, tile)) continue;
        const uint32_t tm = tile / tiles_n, tn = tile - tm * tiles_n;
        const int64_t st0 = split * g.split_stages;
        const int nst = (int)(min(g.stages, st0 + g.split_stages) - st0);
        const uint8_t* a = g.a + (tm * g.stages + st0) * (int64_t)A_STAGE;
        const uint8_t* b = g.b + (tn * g.stages + st0) * (int64_t)B_STAGE;
        for (int st = 0; st < nst; ++st, ++it) {
          const int s = it % STAGES, use = it / STAGES;
          if (use > 0) go = tc::mbar_wait_abortable(&empty_bar[s], (use - 1) & 1, WAIT_CYCLES, vstatus);
          if (!go) break;
          uint8_t* dst = smem + s * STAGE;
          tc::mbar_arrive_expect_tx(&full_bar[s], STAGE);
          bulk_load(dst, a + (int64_t)st * A_STAGE, A_STAGE, &full_bar[s]);
          bulk_load(dst + A_STAGE, b + (int64_t)st * B_STAGE, B_STAGE, &full_bar[s]);
        }
      }
      if (!go) {
        // the copies in flight land before the CTA gives up its shared memory
        atomicExch(g.status, PTN_ERR_TIMEOUT);
        for (int s = 0; s < STAGES && s < it; ++s) {
          const int last = s + ((it - 1 - s) / STAGES) * STAGES;
          tc::mbar_wait(&full_bar[s], (uint32_t)((last / STAGES) & 1), WAIT_CYCLES);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMAs ----------------
    if (lane == 0) {
      int it = 0, chunk = 0;
      bool go = true;
      for (uint32_t w = blockIdx.x; w < items && go; w += gridDim.x) {
        if (skips_digits(g, w % tiles)) continue;
        const int64_t st0 = (w / tiles) * g.split_stages;
        const int nst = (int)(min(g.stages, st0 + g.split_stages) - st0);
        for (int st = 0; st < nst; ++st, ++it) {
          const int s = it % STAGES;
          const bool first = st % CHUNK_STAGES == 0;
          if (first && chunk > 0) go = tc::mbar_wait_abortable(&tempty_bar, (chunk - 1) & 1, WAIT_CYCLES, vstatus);
          go = go && tc::mbar_wait_abortable(&full_bar[s], (it / STAGES) & 1, WAIT_CYCLES, vstatus);
          if (!go) break;
          tc::fence_after();
          const uint32_t sa = tc::smem_u32(smem + s * STAGE);
          mma_stage(tmem, sa, sa + A_STAGE, first);
          tc::mma_commit(&empty_bar[s]);
          if (st % CHUNK_STAGES == CHUNK_STAGES - 1 || st == nst - 1) {
            tc::mma_commit(&tfull_bar);
            ++chunk;
          }
        }
      }
      if (!go) {
        atomicExch(g.status, PTN_ERR_TIMEOUT);
        tc::mma_commit(&drain_bar);                  // every MMA issued ends before TMEM is freed
        tc::mbar_wait(&drain_bar, 0, WAIT_CYCLES);
      }
    }
  } else if (warp >= FIRST_EPI) {
    // ---------------- epilogue: thread = (row, 8 complex columns) ----------------
    const int q = warp & 3, wc0 = ((warp - FIRST_EPI) >> 2) * WC;
    const int row = q * 32 + lane;
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    double2* out = reinterpret_cast<double2*>(smem + STAGES * STAGE) + (warp - FIRST_EPI) * 32 * 4;
    int chunk = 0;
    bool ok = true;
    for (uint32_t w = blockIdx.x; w < items; w += gridDim.x) {
      const uint32_t split = w / tiles, tile = w - split * tiles;
      if (skips_digits(g, tile)) continue;
      const int64_t tm = tile / tiles_n, tn = tile - (uint32_t)tm * tiles_n;
      const int64_t st0 = split * g.split_stages;
      const int nst = (int)(min(g.stages, st0 + g.split_stages) - st0);
      const int nchunks = (nst + CHUNK_STAGES - 1) / CHUNK_STAGES;
      // offsets and exponents of this thread's row and (lanes 0..7) column
      const int64_t ml = tm * TM + row, n0 = tn * TN + wc0;
      int64_t offm = -1, offn = -1, unused;
      if (g.splits > 1) {
        if (g.m0 + ml < g.c.M) offm = (split * g.rows + ml) * g.c.N;
        if (lane < WC && n0 + lane < g.c.N) offn = n0 + lane;
      } else {
        if (g.m0 + ml < g.c.M) decode(g.c.m, g.m0 + ml, unused, offm);
        if (lane < WC && n0 + lane < g.c.N) decode(g.c.n, n0 + lane, unused, offn);
      }
      const int ea = g.ea[split * g.tiles_m * TM + ml];
      const int eb_l = g.eb[split * g.tiles_n * TN + n0 + (lane & (WC - 1))];
      long long hi[2 * WC];                          // 8 Re, 8 Im: value = hi 2^32 + lo
      uint32_t lo[2 * WC];
#pragma unroll
      for (int i = 0; i < 2 * WC; ++i) {
        hi[i] = 0;
        lo[i] = 0;
      }
      for (int c = 0; c < nchunks && ok; ++c, ++chunk) {
        ok = tc::mbar_wait_abortable(&tfull_bar, chunk & 1, WAIT_CYCLES, vstatus);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc::fence_after();
        // 2 columns of all groups at a time, the next two under way meanwhile
        uint32_t v[2][G][2];
        const uint32_t src = tmem + lane_off + (uint32_t)wc0;
#pragma unroll
        for (int gr = 0; gr < G; ++gr) tmem_ld2_nowait(src + (uint32_t)(gr * GROUP_COLS), v[0][gr]);
#pragma unroll
        for (int b = 0; b < WC; ++b) {
          tc::tmem_wait_ld();
          if (b + 1 < WC) {
            const int col = ((b + 1) / (WC / 2)) * TN + ((b + 1) % (WC / 2)) * 2;
#pragma unroll
            for (int gr = 0; gr < G; ++gr)
              tmem_ld2_nowait(src + (uint32_t)(gr * GROUP_COLS + col), v[(b + 1) & 1][gr]);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            long long h = hi[b * 2 + i], l = (long long)lo[b * 2 + i];
#pragma unroll
            for (int gr = 0; gr < 4; ++gr) {
              h = mad_wide(__float2int_rn(__uint_as_float(v[b & 1][gr][i])), 1 << (8 * (3 - gr)), h);
              l = mad_wide(__float2int_rn(__uint_as_float(v[b & 1][gr + 4][i])), 1 << (8 * (3 - gr)), l);
            }
            hi[b * 2 + i] = h + (l >> 32);
            lo[b * 2 + i] = (uint32_t)l;
          }
        }
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&tempty_bar);
      }
      if (!ok && lane == 0) atomicExch(g.status, PTN_ERR_TIMEOUT);
      // Four columns at a time go through shared memory, so that neighbouring
      // lanes write neighbouring columns (64 contiguous bytes of a row of a
      // chain's intermediate): in turn t a lane stores row 8 t + lane / 4,
      // column lane % 4. (The staging's columns are exchanged by row, so that
      // neither side meets a bank twice.)
      if (ok) {
        const uint32_t mm = (g.mask[(int64_t)tile * TM + row] >> wc0) & 0xffu;
        int64_t om[4];
        uint32_t leave = 0u;                           // the guard's bits of the rows that this lane stores
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          om[t] = __shfl_sync(0xffffffffu, (long long)offm, t * 8 + (lane >> 2));
          leave |= __shfl_sync(0xffffffffu, mm, t * 8 + (lane >> 2)) << (8 * t);
        }
        double2* dst = g.splits > 1 ? g.partial : g.c.C;
#pragma unroll
        for (int b = 0; b < WC / 4; ++b) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int j = b * 4 + i, sc = ea + __shfl_sync(0xffffffffu, eb_l, j) - 70;
            double2 v;
            v.x = fixed_to_double(hi[j], lo[j], sc);
            v.y = fixed_to_double(hi[WC + j], lo[WC + j], sc);
            out[lane * 4 + (i ^ ((lane >> 1) & 3))] = v;
          }
          __syncwarp();
          const int64_t on = __shfl_sync(0xffffffffu, (long long)offn, b * 4 + (lane & 3));
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            if (om[t] >= 0 && on >= 0 && !(leave >> (8 * t + b * 4 + (lane & 3)) & 1u)) {
              double2 v = out[(t * 8 + (lane >> 2)) * 4 + ((lane & 3) ^ ((lane >> 3) & 3))];
              double2* p = dst + om[t] + on;
              if (!UNIT && g.splits == 1) v = finish(g.c.alpha, g.c.beta, g.c.beta_zero, v, p);
              *p = v;
            }
          }
          __syncwarp();
        }
      }
      if (!ok) nan_part(g, w, warp - FIRST_EPI);
    }
    plain_tiles(g, smem, __any_sync(0xffffffffu, *vstatus != 0));
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(tmem, G * GROUP_COLS);
}

// The splits' sums added in order (deterministic), then alpha, beta and the scatter.
__global__ void __launch_bounds__(256) ptn_zgemm_reduce_kernel(const GemmArgs g) {
  const int64_t total = g.rows * g.c.N;
  for (int64_t e = blockIdx.x * 256ll + threadIdx.x; e < total; e += gridDim.x * 256ll) {
    const int64_t r = e / g.c.N, n = e - r * g.c.N;
    double2 v = make_double2(0.0, 0.0);
    for (int s = 0; s < g.splits; ++s) v = cadd(v, g.partial[s * total + e]);
    int64_t x, om, on;
    decode(g.c.m, g.m0 + r, x, om);
    decode(g.c.n, n, x, on);
    double2* p = g.c.C + om + on;
    *p = finish(g.c.alpha, g.c.beta, g.c.beta_zero, v, p);
  }
}

inline int64_t up(int64_t x, int64_t a) { return (x + a - 1) / a * a; }

int64_t count(const ptn_modes& m) {
  if (m.n < 0 || m.n > PTN_MAX_MODES) return -1;
  int64_t t = 1;
  for (int i = 0; i < m.n; ++i) {
    if (m.dim[i] <= 0) return -1;
    t *= m.dim[i];
  }
  return t;
}

// Whether the digit products take an M x N x K contraction, and how.
bool make_plan(int64_t M, int64_t N, int64_t K, Plan& p) {
  if (M < 1 || N < 1 || K < 1 || M > (1ll << 40) / N || K > 0x7fffffffLL) return false;
  const int64_t t0 = up(M, TM) / TM * (up(N, TN) / TN), t1 = up(N, TM) / TM * (up(M, TN) / TN);
  p.swap = t1 < t0 || (t1 == t0 && N > M);
  p.M = p.swap ? N : M;
  p.N = p.swap ? M : N;
  p.K = K;
  if (M * N * K < PTN_ZTC_MIN_MACS) return false;
  p.stages = (K + KS - 1) / KS;
  p.tiles_m = (p.M + TM - 1) / TM;
  p.tiles_n = (p.N + TN - 1) / TN;
  const int64_t tiles = p.tiles_m * p.tiles_n;
  // Both sides are padded to a 128 x 32 tile, and converting those zeros costs like
  // anything else: a few outputs over a long K stay with the FP64 kernels (16 x 16 over
  // 65536 194 us there, 211 here, 8 x 8 over 131072 172 and 351, 2 x 3 over a million 1.3
  // and 2.4 ms; 30 x 30 over 8000 125 us there, 61 here).
  if (M * N <= MIN_OUTPUTS) return false;
  // At least 128 K to a range: the two launches that add ranges up take as long as two
  // chunks of 64 (640 x 32 x 160 55 us in two ranges, 640 x 128 x 128 53, MMAs 16 of them).
  int64_t want = tiles >= 152 ? 1 : 152 / tiles;
  if (want > p.stages / (2 * CHUNK_STAGES)) want = p.stages / (2 * CHUNK_STAGES);
  const int64_t least = (p.stages + MAX_SPLIT_STAGES - 1) / MAX_SPLIT_STAGES;
  if (want < least) want = least;
  if (want < 1) want = 1;
  p.split_stages = (p.stages + want - 1) / want;
  if (want > 1) p.split_stages = up(p.split_stages, CHUNK_STAGES);
  p.splits = (p.stages + p.split_stages - 1) / p.split_stages;
  p.chunk_tiles = A_BYTES_MAX / (p.stages * (A_STAGE + GUARD));
  if (p.chunk_tiles < 1) p.chunk_tiles = 1;
  if (p.chunk_tiles > p.tiles_m) p.chunk_tiles = p.tiles_m;
  if (p.chunk_tiles * p.tiles_n * p.splits > 0x7ffffffLL) return false;
  int64_t o = 256;
  p.off_ks = o;
  o += up((int64_t)sizeof(KStat) * K, 256);
  p.off_ea = o;
  o += up(4 * p.splits * p.chunk_tiles * TM, 256);
  p.off_eb = o;
  o += up(4 * p.splits * p.tiles_n * TN, 256);
  p.off_a = o;
  o += p.chunk_tiles * p.stages * A_STAGE;
  p.off_b = o;
  o += p.tiles_n * p.stages * B_STAGE;
  p.off_ga = o;
  o += p.chunk_tiles * p.stages * GUARD;
  p.off_gb = o;
  o += (p.tiles_n + GT - 1) / GT * p.stages * GUARD;
  const int64_t items = p.chunk_tiles * p.tiles_n * p.splits;
  p.off_mask = o;
  o += 4 * TM * p.chunk_tiles * p.tiles_n;
  p.off_cnt = o;
  o += 16 * p.chunk_tiles * p.tiles_n;
  p.off_sums = up(o, 256);
  if (p.splits > 1) o = p.off_sums + 4 * TM * TN * items;
  p.off_part = up(o, 256);
  p.bytes = p.off_part + (p.splits > 1 ? 16 * p.splits * p.chunk_tiles * TM * p.N : 0);
  return p.bytes <= WORK_MAX;    // (a K of a million and more)
}

// The guard's limit in units of a row's and a column's power of two: where a single
// product of that size is rounded by FP64 (2^-54) as much as by the digits (1.7 2^-64
// with all digits of both in use; sqrt(K) times it where the other terms, though small,
// fill the row and the column).
float guard_theta(int64_t K) { return ldexpf(K > 64 ? sqrtf((float)K / 64.f) : 1.f, -9); }

// Threads along K: one stage per thread when the rows alone fill the GPU (the
// values then stay in registers between the two passes), more when they do not.
int64_t row_blocks(DigitsArgs& q, int64_t padded_rows, int64_t splits) {
  const int64_t st = q.split_stages;
  q.kg = st >= 3 ? 4 : (st == 2 ? 2 : 1);
  while (q.kg < 16 && st >= 2 * q.kg && padded_rows * q.kg / 128 * splits < 304) q.kg *= 2;
  q.blocks_rows = (padded_rows + 128 / q.kg - 1) / (128 / q.kg);
  return q.blocks_rows;
}

}  // namespace

extern "C" int64_t ptn_zcontract_work_bytes(const ptn_contract_desc* d) {
  if (!d) return 0;
  const int64_t M = count(d->m), N = count(d->n), K = count(d->k);
  Plan p;
  if (M < 1 || N < 1 || K < 1 || !make_plan(M, N, K, p)) return 0;
  return p.bytes;
}

extern "C" int ptn_zcontract_ws(const ptn_contract_desc* d, void* work, int64_t work_bytes, void* stream) {
  if (!d || !d->A || !d->B || !d->C) return PTN_ERR_ARG;
  ContractArgs c;
  if (zcontract_args(*d, c)) return PTN_ERR_ARG;
  Plan p;
  if (!work || (reinterpret_cast<uintptr_t>(work) & 255) || !make_plan(c.M, c.N, c.K, p) || work_bytes < p.bytes ||
      c.M * c.N * c.K < PTN_ZTC_PAYS)
    return ptn_zcontract(d, stream);
  static PtnSharedMemory unit_memory, general_memory, guard_memory;
  if (!unit_memory((const void*)ptn_zgemm_digits_kernel<true>, SMEM) ||
      !general_memory((const void*)ptn_zgemm_digits_kernel<false>, SMEM) ||
      !guard_memory((const void*)ptn_zguard_kernel, GUARD_SMEM))
    return PTN_ERR_LAUNCH;
  if (p.swap) {
    const double2* t = c.A;
    c.A = c.B;
    c.B = t;
    const int cj = c.conj_a;
    c.conj_a = c.conj_b;
    c.conj_b = cj;
    const ModeDev md = c.m;
    c.m = c.n;
    c.n = md;
    for (int i = 0; i < c.k.n; ++i) {
      const int64_t s = c.k.s0[i];
      c.k.s0[i] = c.k.s1[i];
      c.k.s1[i] = s;
    }
    c.M = p.M;
    c.N = p.N;
  }
  const bool unit = (c.alpha.x == 1.0 && c.alpha.y == 0.0 && c.beta_zero) || p.splits > 1;
  uint8_t* w = static_cast<uint8_t*>(work);
  cudaStream_t s = ptn_stream(stream);
  DigitsArgs qa = {}, qb = {};
  qa.src = c.A;
  qa.rows = c.m;
  qa.ks = c.k;
  qa.nrows = c.M;
  qa.tile_rows = TM;
  qa.conj = c.conj_a;
  qa.dst = w + p.off_a;
  qa.guard = w + p.off_ga;
  qa.exps = reinterpret_cast<int*>(w + p.off_ea);
  qb.src = c.B;
  qb.rows = c.n;
  qb.ks = c.k;
  for (int i = 0; i < c.k.n; ++i) qb.ks.s0[i] = c.k.s1[i];
  qb.nrows = c.N;
  qb.tile_rows = TN;
  qb.conj = c.conj_b;
  qb.dst = w + p.off_b;
  qb.guard = w + p.off_gb;
  qb.exps = reinterpret_cast<int*>(w + p.off_eb);
  qa.K = qb.K = c.K;
  qa.stages = qb.stages = p.stages;
  qa.split_stages = qb.split_stages = p.split_stages;
  qb.tiles = p.tiles_n;
  const int64_t blocks_b = row_blocks(qb, p.tiles_n * TN, p.splits) * p.splits;
  qa.ks_stat = qb.ks_stat = reinterpret_cast<const KStat*>(w + p.off_ks);
  qa.na = qb.na = c.M <= LOOK ? c.M : SAMPLES;
  qa.nb = qb.nb = c.N;
  qa.rows_a = qb.rows_a = c.M;
  PTN_COUNT(1);
  ptn_zksample_kernel<<<(unsigned)c.K, LOOK, 0, s>>>(qa, qb, reinterpret_cast<KStat*>(w + p.off_ks));
  const size_t koff_bytes = (size_t)(p.split_stages * KS) * (sizeof(int64_t) + sizeof(int));
  GemmArgs g;
  g.c = c;
  g.a = qa.dst;
  g.b = qb.dst;
  g.ea = qa.exps;
  g.eb = qb.exps;
  g.tiles_n = p.tiles_n;
  g.stages = p.stages;
  g.split_stages = p.split_stages;
  g.splits = (int32_t)p.splits;
  g.partial = reinterpret_cast<double2*>(w + p.off_part);
  g.status = reinterpret_cast<int32_t*>(w);
  g.mask = reinterpret_cast<const uint32_t*>(w + p.off_mask);
  g.count = reinterpret_cast<const int4*>(w + p.off_cnt);
  const int64_t k_split = p.split_stages * KS < p.K ? p.split_stages * KS : p.K;
  g.skip_tile = (int32_t)(EPI_WARPS * part_cost(k_split) / one_cost(k_split));
  GuardArgs gd;
  gd.a = qa.guard;
  gd.b = qb.guard;
  gd.tiles_n = p.tiles_n;
  gd.stages = p.stages;
  gd.split_stages = p.split_stages;
  gd.splits = (int32_t)p.splits;
  gd.theta = guard_theta(p.K);
  gd.sums = p.splits > 1 ? reinterpret_cast<float*>(w + p.off_sums) : nullptr;
  gd.ea = qa.exps;
  gd.eb = qb.exps;
  gd.mask = reinterpret_cast<uint32_t*>(w + p.off_mask);
  gd.count = reinterpret_cast<int*>(w + p.off_cnt);
  gd.status = g.status;
  for (int64_t t0 = 0; t0 < p.tiles_m; t0 += p.chunk_tiles) {
    const int64_t tiles = p.tiles_m - t0 < p.chunk_tiles ? p.tiles_m - t0 : p.chunk_tiles;
    qa.row0 = t0 * TM;
    qa.tiles = tiles;
    const int64_t blocks_a = row_blocks(qa, tiles * TM, p.splits) * p.splits;
    const int64_t blocks = blocks_a + (t0 == 0 ? blocks_b : 0);     // B once, with the first rows
    PTN_COUNT(1);
    ptn_zdigits_kernel<<<(unsigned)blocks, 256, koff_bytes, s>>>(qa, qb, blocks_a, g.status);
    g.m0 = t0 * TM;
    g.tiles_m = tiles;
    g.tiles = tiles * p.tiles_n;
    g.rows = c.M - g.m0 < tiles * TM ? c.M - g.m0 : tiles * TM;
    gd.tiles_m = tiles;
    const int64_t guards = tiles * ((p.tiles_n + GT - 1) / GT) * p.splits;
    PTN_COUNT(2);
    ptn_zguard_kernel<<<(unsigned)(guards < 152 ? guards : 152), GUARD_THREADS, GUARD_SMEM, s>>>(gd);
    if (p.splits > 1) {
      PTN_COUNT(1);
      ptn_zguard_split_kernel<<<(unsigned)g.tiles, 1024, 0, s>>>(gd);
    }
    const int64_t items = g.tiles * p.splits;
    const unsigned grid = (unsigned)(items < 152 ? items : 152);
    if (unit) ptn_zgemm_digits_kernel<true><<<grid, THREADS, SMEM, s>>>(g);
    else ptn_zgemm_digits_kernel<false><<<grid, THREADS, SMEM, s>>>(g);
    if (p.splits > 1) {
      const int64_t nb = (g.rows * c.N + 255) / 256;
      PTN_COUNT(1);
      ptn_zgemm_reduce_kernel<<<(unsigned)(nb < 152 * 8 ? nb : 152 * 8), 256, 0, s>>>(g);
    }
  }
  return ptn_launch_status();
}
