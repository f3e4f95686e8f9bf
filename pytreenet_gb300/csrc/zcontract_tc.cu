// Complex128 contractions on the 5th-generation tensor cores, with the
// accuracy of the FP64 kernels.
//
// GB300 issues about two FP64 FMAs per clock per SM (1.25 TFLOP/s), a 900th of
// its bf16 tensor rate, so a contraction with enough arithmetic is done as
// exact integer products instead (the digit-slicing scheme of Ozaki, Ogita,
// Oishi and Rump, Numer. Algorithms 59, 2012): every row of A and of B is
// scaled by the power of two above its largest entry and rounded to a 55-bit
// fixed-point number, which is written in seven balanced base-256 digits in
// [-128, 128]. A digit is exact in bf16, the product of two is at most 2^14,
// and a K range of 64 adds at most 2^24 of them into one FP32 TMEM
// accumulator, so every tensor-core sum is an exact integer. The products
// d_i(A) d_j(B) of equal i + j share an accumulator (a "group"); groups 0..7
// are kept (34 digit pairs of the 49: group 8 is 2^-64 of the leading one),
// combined in 128-bit integers across the K range and rounded to double once.
// What is lost is the rounding of the operands at 2^-56 of the row's power of
// two: for K >= 64 below the rounding of an FP64 dot product, whose K
// additions each lose 2^-53 of the running sum.
//
// Before that, index k of both operands is balanced by a power of two: B's row
// of index k is divided by the power of its largest entry and A's column k
// multiplied by it (exact, on the exponents). A row's scale is then the
// largest |a_mk| max_n |b_kn|, so operands graded along k against each other
// (a factor and its inverse) lose nothing.
//
// MMA shape: digit i of A against the digits 0..J of B in one instruction
// stream: B's digits lie one below the other in shared memory ([Br; Bi], 64
// rows each), so the N = 64 (J + 1) columns of the product land in the
// accumulators of groups i..i + J, which are adjacent in TMEM. With 32 complex
// columns per tile eight groups fill TMEM (8 x 64 columns), and A's 4 KB plane
// is read from shared memory 11 times per 34 products instead of 34.
//
// Operands are written by ptn_zdigits_kernel as the images of the
// shared-memory stages (32-byte swizzle applied), so a stage is two contiguous
// bulk copies: no tensor maps, and no host work per call.
//
// Measured (M x N x K; FP64 kernels -> here, all launches): 8192 x 320 x 64
// 1327 -> 66 us, 40960 x 64 x 320 6510 -> 355 us, 262144 x 50 x 10 1870 -> 219
// us, 131072 x 256 x 256 55.9 -> 2.0 ms, 256 x 256 x 2560 2110 -> 115 us, 640 x
// 128 x 128 87 -> 37 us. Error against 113-bit sums (2-norm, Gaussian operands):
// 5.7e-17 to 2.3e-16 for K = 10 to 5000, the FP64 kernels 1.5e-16 to 1.2e-15.
//
// Rows that hold a NaN or an infinity are marked; their outputs are summed in
// FP64 by the epilogue thread that owns them, so they propagate as in the FP64
// kernels. Every wait is bounded; on a timeout the CTA's outputs become NaN.
#include <cuda_bf16.h>
#include <limits.h>

#include "ptn_common.cuh"
#include "tc_ptx.cuh"
#include "zmodes.cuh"

namespace {

constexpr int D = 7;                              // digits per operand
constexpr int G = 8;                              // accumulator groups kept
constexpr int TM = 128, TN = 32, KS = 16;         // tile rows, complex columns, K per stage
constexpr int CHUNK_STAGES = 4;                   // 64 K values: 7 pairs x 2 x 64 x 2^14 < 2^24
constexpr int A_STAGE = 2 * D * TM * KS * 2;      // 56 KB: planes Re_0, Im_0, Re_1, ...
constexpr int B_PLANE = TN * KS * 2;              // 1 KB
constexpr int B_STAGE = 4 * D * B_PLANE;          // 28 KB: [Br_j; Bi_j] by digit, then [-Bi_j; Br_j]
constexpr int STAGE = A_STAGE + B_STAGE;
constexpr int STAGES = 2;
constexpr int OUT_BYTES = 16 * 32 * 5 * 16;       // output staging of the epilogue warps
constexpr int SMEM = STAGES * STAGE + OUT_BYTES + 1024;
constexpr int FIRST_EPI = 4, EPI_WARPS = 16;      // warps 0: copies, 1: MMAs, 4..19: epilogue
constexpr int THREADS = 32 * (FIRST_EPI + EPI_WARPS);
constexpr int WC = TN / 4;                        // complex columns of an epilogue warp
constexpr int OUT_LD = 5;                         // pitch of an epilogue warp's 32 x 4 output staging
constexpr int GROUP_COLS = 2 * TN;                // [Re | Im]
constexpr int SPECIAL = INT_MAX;                  // exponent of a row with a NaN or an infinity
constexpr int NO_ENTRY = INT_MIN;                 // no entry of the row seen that is not zero
// K per split: the conversion's offset table (12 bytes a k) and its row maxima stay
// within the 48 KB of shared memory that a launch gets without asking for more.
constexpr int MAX_SPLIT_STAGES = 248;
static_assert(MAX_SPLIT_STAGES % CHUNK_STAGES == 0 && MAX_SPLIT_STAGES * KS * 12 + 128 * 4 <= 48 * 1024, "");
constexpr int64_t A_BYTES_MAX = 1ll << 30;        // digits of A held at once; more rows go in turns
// Complex multiply-adds from which this path is taken: its three launches cost
// 25 to 28 us where the FP64 kernels take 16 us (1024 x 32 x 32, 1.0 M), 24 us
// (512 x 64 x 64, 2.1 M), 87 us (640 x 128 x 128, 10 M).
constexpr int64_t PTN_ZTC_MIN_MACS = 3ll << 20;
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
  int64_t off_kx, off_ea, off_eb, off_a, off_b, off_part, bytes;
};

struct DigitsArgs {
  const double2* src;
  ModeDev rows, ks;          // strides in s0
  int64_t nrows, K;
  int64_t row0;              // first row of this turn
  int64_t tiles;             // row tiles written
  int tile_rows;             // 128 (A) or 32 (B)
  int conj;
  int ksign;                 // +1: entries times 2^kx (A), -1: divided (B)
  const int* kx;             // [K]
  int kg;                    // groups of threads along K (power of two)
  int64_t stages, split_stages;
  uint8_t* dst;
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
};

// ---- operands -> digits ----------------------------------------------------------
// kx[k] = exponent of the power of two at or below the largest entry of B's
// row k (0 for a row of zeros or one with a NaN or an infinity). A warp takes
// one k; eight neighbouring k to a CTA.
__global__ void __launch_bounds__(256) ptn_zkmax_kernel(const DigitsArgs q, int* __restrict__ kx) {
  const int lane = threadIdx.x & 31;
  const int64_t k = blockIdx.x * 8ll + (threadIdx.x >> 5);
  if (k >= q.K) return;
  int64_t ok, unused, on;
  decode(q.ks, k, ok, unused);
  int top = 0;
  for (int64_t n = lane; n < q.nrows; n += 32) {
    decode(q.rows, n, on, unused);
    const double2 v = q.src[ok + on];
    top = max(top, max(__double2hiint(v.x) & 0x7fffffff, __double2hiint(v.y) & 0x7fffffff));
  }
  top = __reduce_max_sync(0xffffffffu, top) >> 20;
  if (lane == 0) kx[k] = (top == 0 || top == 0x7ff) ? 0 : top - 1023;
}

// round(x 2^(55 - delta') ) + 128 (256^0 + ... + 256^5), where the entry lies
// `delta` powers of two below the largest a row may hold: byte b of the result
// less 128 is digit 6 - b, the signed rest above bit 48 is digit 0. Half units
// round up. 32-bit integer instructions only (about 20).
__device__ __forceinline__ void biased_digits(uint32_t xh, uint32_t xl, int delta, uint32_t& th, uint32_t& tl) {
  const int d1 = min(delta, 32), d2 = min(delta - d1, 32);
  // the mantissa at bit 55 with one more bit for rounding, shifted down by delta
  uint32_t h = (xh & 0xfffffu) | 0x100000u, l = xl;
  h = __funnelshift_l(l, h, 3);
  l <<= 3;
  l = __funnelshift_rc(l, h, d1);
  h = __funnelshift_rc(h, 0u, d1);
  l = __funnelshift_rc(l, h, d2);
  h = __funnelshift_rc(h, 0u, d2);
  // +-v + (2 bias + 1), then one down
  const uint32_t sg = (uint32_t)((int)xh >> 31);
  l ^= sg;
  h ^= sg;
  const uint32_t bl = 0x01010101u - sg, bh = 0x00010101u;        // the sign's + 1 rides on the constant
  asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, %3;" : "+r"(l), "+r"(h) : "r"(bl), "r"(bh));
  tl = __funnelshift_r(l, h, 1);
  th = (uint32_t)((int)h >> 1);
}

// Digit d (1..6) of two biased numbers as a bf16 pair. With u the byte, u - 128
// is (128 + u mod 128) - (u >= 128 ? 128 : 256), all four exact in bf16 and
// made of u's bits.
__device__ __forceinline__ uint32_t digit_pair(uint32_t ah, uint32_t al, uint32_t bh, uint32_t bl, int d) {
  const int byte = D - 1 - d;                        // 0..5
  // the two bytes to bytes 0 and 2 (bytes 1 and 3 are masked off below)
  const uint32_t x = byte < 4 ? __byte_perm(al, bl, (uint32_t)byte | ((uint32_t)(byte + 4) << 8))
                              : __byte_perm(ah, bh, (uint32_t)(byte - 4) | ((uint32_t)byte << 8));
  const uint32_t p = (x & 0x007f007fu) | 0x43004300u, q = (x & 0x00800080u) ^ 0x43804380u;
  const __nv_bfloat162 r = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&p),
                                   *reinterpret_cast<const __nv_bfloat162*>(&q));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// Digit 0, in [-128, 128].
__device__ __forceinline__ uint32_t top_pair(uint32_t ah, uint32_t bh) {
  const float a = __uint_as_float(0x4B400000u + (uint32_t)((int)ah >> 16)) - 12582912.0f;   // 1.5 2^23
  const float b = __uint_as_float(0x4B400000u + (uint32_t)((int)bh >> 16)) - 12582912.0f;
  const __nv_bfloat162 r = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&r);
}

// One CTA: 128 / kg rows x one K split. Thread = (K group, row, half stage of 8
// K values). First the largest exponent of each row over the split, then the
// digits, eight K values (16 bytes per plane) at a time; consecutive threads
// write consecutive 16-byte pieces of a plane. HBM / L2 bound: 16 bytes read
// (twice when a thread has more than one stage, the second time from L2) and 28
// (A) or 56 (B) written per entry; the digit arithmetic is 32-bit integer and
// FP32 only, so that it does not wait for the FP64 pipe.
__global__ void __launch_bounds__(256, 3) ptn_zdigits_kernel(const DigitsArgs qa, const DigitsArgs qb,
                                                          const int64_t blocks_a, int32_t* status) {
  extern __shared__ int64_t koff[];                  // source offset of each k, then its exponent
  __shared__ int mx[128];
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
  for (int e = tid; e < nst * KS; e += 256) {
    const int64_t k = st0 * KS + e;
    int64_t o0 = -1, o1;
    int x = 0;
    if (k < q.K) {
      decode(q.ks, k, o0, o1);
      x = q.ksign * q.kx[k];
    }
    koff[e] = o0;
    kx[e] = x;
  }
  for (int e = tid; e < rpc; e += 256) mx[e] = NO_ENTRY;
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
  const int E = mx[r] == NO_ENTRY ? 0 : mx[r];
  const int below = E == SPECIAL ? 4096 : E + 1022;  // digits of a special row are not used
  const int64_t padded = q.tiles * q.tile_rows;
  if (lrow >= padded) return;
  if (h == 0 && g == 0) q.exps[split * padded + lrow] = E;
  const int64_t tile = lrow / q.tile_rows;
  const int tr = (int)(lrow - tile * q.tile_rows);
  const int stage_bytes = is_a ? A_STAGE : B_STAGE;
  const int plane = q.tile_rows * KS * 2;
  const int within = tr * 32 + ((h ^ ((tr >> 2) & 1)) << 4);
  for (int st = g; st < nst; st += q.kg) {
    if (nst > q.kg) load(st);                        // otherwise still in registers
    uint8_t* out = q.dst + (tile * q.stages + st0 + st) * (int64_t)stage_bytes + within;
    const int* kk = kx + st * KS + h * 8;
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      uint32_t th[8], tl[8];
      const uint32_t flip = part && q.conj ? 0x80000000u : 0u;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const double x = part ? v[u].y : v[u].x;
        const uint32_t xh = (uint32_t)__double2hiint(x) ^ flip;
        const int field = (int)(xh >> 20) & 0x7ff;
        // a zero has field 0 and is shifted out (E > -400 wherever digits count)
        const int delta = field == 0 ? 64 : below - field - kk[u];
        biased_digits(xh, (uint32_t)__double2loint(x), delta, th[u], tl[u]);
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

// The outputs of one epilogue warp (32 rows x 8 columns) whose rows hold a NaN,
// an infinity or magnitudes near the ends of the double range, summed as the
// FP64 kernels do; NaN after a timeout. Out of line, and without the digit
// sums, so that the common path keeps its registers.
__device__ __noinline__ void plain_outputs(const GemmArgs& g, int64_t row_in_turn, int64_t n0, int64_t split,
                                           int64_t k0, int64_t k1, bool failed) {
  const int64_t m = g.m0 + row_in_turn;
  if (m >= g.c.M) return;
  int64_t oa, om, x, y;
  decode(g.c.m, m, oa, om);
  for (int64_t n = n0; n < n0 + TN / 4 && n < g.c.N; ++n) {
    int64_t ob, on;
    decode(g.c.n, n, ob, on);
    double2 acc = make_double2(0.0, 0.0);
    for (int64_t k = k0; k < k1; ++k) {
      decode(g.c.k, k, x, y);
      double2 av = g.c.A[oa + x], bv = g.c.B[ob + y];
      if (g.c.conj_a) av.y = -av.y;
      if (g.c.conj_b) bv.y = -bv.y;
      acc = cfma(av, bv, acc);
    }
    if (failed) acc = make_double2(NAN, NAN);
    if (g.splits > 1) {
      g.partial[(split * g.rows + row_in_turn) * g.c.N + n] = acc;
    } else {
      double2* p = g.c.C + om + on;
      *p = finish(g.c.alpha, g.c.beta, g.c.beta_zero, acc, p);
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
      const int cols = GROUP_COLS * (i == 0 ? D : G - i);
      if (i == 1 && ow) {
        // groups 1..6 were started by digit 0, group 7 starts here
        mma_cols(acc, a, b, 0, 256, false, i);
        mma_cols(acc, a, b, 256, 128, false, i);
        mma_cols(acc, a, b, 384, 64, true, i);
      } else if (cols > 256) {
        const int half = cols / 2;                   // 224, 192, 160: multiples of 16
        mma_cols(acc, a, b, 0, half, ow && i == 0, i);
        mma_cols(acc, a, b, half, cols - half, ow && i == 0, i);
      } else {
        mma_cols(acc, a, b, 0, cols, false, i);
      }
    }
  }
}

// Persistent: a CTA takes the (tile, split) items blockIdx.x, + gridDim.x, ...
// One warp copies stages ahead, one issues MMAs, eight drain and write. TMEM
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
    double2* out = reinterpret_cast<double2*>(smem + STAGES * STAGE) + (warp - FIRST_EPI) * 32 * OUT_LD;
    int chunk = 0;
    bool ok = true;
    for (uint32_t w = blockIdx.x; w < items; w += gridDim.x) {
      const uint32_t split = w / tiles, tile = w - split * tiles;
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
      // column lane % 4.
      if (!ok || !__all_sync(0xffffffffu, abs(ea) <= 400 && abs(eb_l) <= 400)) {
        plain_outputs(g, ml, n0, split, st0 * KS, min(g.c.K, (st0 + nst) * KS), !ok);
        continue;
      }
      int64_t om[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) om[t] = __shfl_sync(0xffffffffu, (long long)offm, t * 8 + (lane >> 2));
      double2* dst = g.splits > 1 ? g.partial : g.c.C;
#pragma unroll
      for (int b = 0; b < WC / 4; ++b) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int j = b * 4 + i, sc = ea + __shfl_sync(0xffffffffu, eb_l, j) - 70;
          double2 v;
          v.x = fixed_to_double(hi[j], lo[j], sc);
          v.y = fixed_to_double(hi[WC + j], lo[WC + j], sc);
          out[lane * OUT_LD + i] = v;
        }
        __syncwarp();
        const int64_t on = __shfl_sync(0xffffffffu, (long long)offn, b * 4 + (lane & 3));
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (om[t] >= 0 && on >= 0) {
            double2 v = out[(t * 8 + (lane >> 2)) * OUT_LD + (lane & 3)];
            double2* p = dst + om[t] + on;
            if (!UNIT && g.splits == 1) v = finish(g.c.alpha, g.c.beta, g.c.beta_zero, v, p);
            *p = v;
          }
        }
        __syncwarp();
      }
    }
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
  if (M < 1 || N < 1 || K < 1 || M > (1ll << 40) / N) return false;
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
  int64_t want = tiles >= 152 ? 1 : 152 / tiles;
  if (want > p.stages / CHUNK_STAGES) want = p.stages / CHUNK_STAGES;
  const int64_t least = (p.stages + MAX_SPLIT_STAGES - 1) / MAX_SPLIT_STAGES;
  if (want < least) want = least;
  if (want < 1) want = 1;
  p.split_stages = (p.stages + want - 1) / want;
  if (want > 1) p.split_stages = up(p.split_stages, CHUNK_STAGES);
  p.splits = (p.stages + p.split_stages - 1) / p.split_stages;
  p.chunk_tiles = A_BYTES_MAX / (p.stages * A_STAGE);
  if (p.chunk_tiles < 1) p.chunk_tiles = 1;
  if (p.chunk_tiles > p.tiles_m) p.chunk_tiles = p.tiles_m;
  if (p.chunk_tiles * p.tiles_n * p.splits > 0x7fffffffLL) return false;
  int64_t o = 256;
  p.off_kx = o;
  o += up(4 * K, 256);
  p.off_ea = o;
  o += up(4 * p.splits * p.chunk_tiles * TM, 256);
  p.off_eb = o;
  o += up(4 * p.splits * p.tiles_n * TN, 256);
  p.off_a = o;
  o += p.chunk_tiles * p.stages * A_STAGE;
  p.off_b = o;
  o += p.tiles_n * p.stages * B_STAGE;
  p.off_part = up(o, 256);
  p.bytes = p.off_part + (p.splits > 1 ? 16 * p.splits * p.chunk_tiles * TM * p.N : 0);
  return p.bytes <= WORK_MAX;    // (a K of a million and more)
}

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
  if (!work || (reinterpret_cast<uintptr_t>(work) & 255) || !make_plan(c.M, c.N, c.K, p) || work_bytes < p.bytes)
    return ptn_zcontract(d, stream);
  // once per process, thread-safe; a failure is returned on every call
  static const bool attr = cudaFuncSetAttribute(ptn_zgemm_digits_kernel<true>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess &&
                           cudaFuncSetAttribute(ptn_zgemm_digits_kernel<false>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess;
  if (!attr) return PTN_ERR_LAUNCH;
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
  qa.exps = reinterpret_cast<int*>(w + p.off_ea);
  qb.src = c.B;
  qb.rows = c.n;
  qb.ks = c.k;
  for (int i = 0; i < c.k.n; ++i) qb.ks.s0[i] = c.k.s1[i];
  qb.nrows = c.N;
  qb.tile_rows = TN;
  qb.conj = c.conj_b;
  qb.dst = w + p.off_b;
  qb.exps = reinterpret_cast<int*>(w + p.off_eb);
  qa.K = qb.K = c.K;
  qa.stages = qb.stages = p.stages;
  qa.split_stages = qb.split_stages = p.split_stages;
  qb.tiles = p.tiles_n;
  const int64_t blocks_b = row_blocks(qb, p.tiles_n * TN, p.splits) * p.splits;
  qa.kx = qb.kx = reinterpret_cast<const int*>(w + p.off_kx);
  qa.ksign = 1;
  qb.ksign = -1;
  PTN_COUNT(1);
  ptn_zkmax_kernel<<<(unsigned)((c.K + 7) / 8), 256, 0, s>>>(qb, reinterpret_cast<int*>(w + p.off_kx));
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
    PTN_COUNT(1);
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
