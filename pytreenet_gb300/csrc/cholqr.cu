// Device-side pieces of CholeskyQR2 for the mixed-precision QR split, and the
// row scan that lets a Householder QR skip exactly-zero trailing rows.
//
// The QR split of a site tensor (tensor_qr_decomposition, util/tensor_splitting.py:60-107)
// is, for a tall matrix A (m x k) of full numerical rank, done as CholeskyQR2:
//   G1 = A^H A,   G1 = R1^H R1,   Q1 = A R1^{-1},
//   G2 = Q1^H Q1, G2 = R2^H R2,   Q  = Q1 R2^{-1},   R = R2 R1.
// The Gram matrices and the products with R^{-1} run on the tensor cores
// (BF16 splits, FP32 accumulation); this file holds the k x k factorisations
// (Cholesky, triangular inverse), done in FP32 on one cluster of CTAs so that no
// host round trip sits between the Gram matrix and its use, and the product R2 R1.
// Q differs from the Householder Q by a diagonal phase only, which one-site
// TDVP absorbs as a gauge change on the bond.
//
// A matrix that is not of full numerical rank (a pivot below ratio * the
// largest, or not positive) is reported through *status; the caller then
// takes the Householder path, whose orthonormal complement the reference's
// results depend on.
#include <cooperative_groups.h>
#include <math.h>

#include "ptn_common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int CH_B = 32;       // block size
constexpr int CH_MAXK = 256;   // largest k
constexpr int CH_UT = 256;     // threads of the block products (8 warps, 2 x 2 outputs a thread)
constexpr int CH_GT = 128;     // threads of one elimination: four warps, one per scheduler
constexpr int CH_T = CH_UT + CH_GT;   // four warps are there for the diagonal blocks
constexpr int CH_C = 8;        // CTAs of the cluster
constexpr int CH_NB = CH_MAXK / CH_B;
constexpr int CH_SLOTS = (CH_NB * (CH_NB + 1) / 2 + CH_C - 1) / CH_C;   // blocks a CTA owns
constexpr int WLD = CH_B + 1;  // padded row of a work block
constexpr int BLK = CH_B * CH_B;

// acc += a * conj(b)
__device__ __forceinline__ void fma_cb(float2& acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, acc.x);
  acc.x = fmaf(a.y, b.y, acc.x);
  acc.y = fmaf(a.y, b.x, acc.y);
  acc.y = fmaf(-a.x, b.y, acc.y);
}
// acc += a * b
__device__ __forceinline__ void fma_c(float2& acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, acc.x);
  acc.x = fmaf(-a.y, b.y, acc.x);
  acc.y = fmaf(a.x, b.y, acc.y);
  acc.y = fmaf(a.y, b.x, acc.y);
}

// (bi, bj), bj <= bi, from the row-wise index of a lower-triangular block list.
__device__ __forceinline__ void tri_decode(int idx, int& bi, int& bj) {
  int r = (int)((sqrtf(8.0f * idx + 1.0f) - 1.0f) * 0.5f);
  while ((r + 1) * (r + 2) / 2 <= idx) ++r;
  while (r * (r + 1) / 2 > idx) --r;
  bi = r;
  bj = idx - r * (r + 1) / 2;
}

// acc[2][2] += sum_c P[c][r] op(Q)[..][s] for rows r = ty, ty + 16 and columns
// s = tx, tx + 16 of a block: P is kept transposed, and so is Q when its conjugate
// transpose is meant (CB), so every read is contiguous over threads.
template <bool CB>
__device__ __forceinline__ void block_mul(const float2* __restrict__ P, const float2* __restrict__ Q, int ty, int tx,
                                          float2 (&acc)[2][2]) {
#pragma unroll 8
  for (int c = 0; c < CH_B; ++c) {
    const float2 a0 = P[c * CH_B + ty], a1 = P[c * CH_B + ty + 16];
    const float2 b0 = Q[c * CH_B + tx], b1 = Q[c * CH_B + tx + 16];
    if (CB) {
      fma_cb(acc[0][0], a0, b0);
      fma_cb(acc[0][1], a0, b1);
      fma_cb(acc[1][0], a1, b0);
      fma_cb(acc[1][1], a1, b1);
    } else {
      fma_c(acc[0][0], a0, b0);
      fma_c(acc[0][1], a0, b1);
      fma_c(acc[1][0], a1, b0);
      fma_c(acc[1][1], a1, b1);
    }
  }
}

struct CholShared {
  float2 work[CH_SLOTS][CH_B * WLD];   // own blocks: A_ij until panel j, then W_ij, T_ij
  float2 diag[BLK];                    // L_pp D_p, transposed: columns before their scaling
  float2 lpp[BLK];                     // L_pp, transposed (in its owner only)
  float2 panel[CH_NB][BLK];            // L_ip, transposed, for i > p; T_pj, row-major, for j <= p
  float2 fin[CH_SLOTS][BLK];           // own L_ij, transposed
  float ip[CH_B], d[CH_B];             // 1 / pivot and its root, the diagonal of L_pp
  float acc[CH_C];
  float mn[CH_NB], mx[CH_NB];
  int bad;
};
static_assert(sizeof(float2) * (CH_NB + CH_SLOTS) * BLK >= sizeof(double2) * CH_SLOTS * CH_B * WLD,
              "the staged blocks of G fit over panel and fin");

// q - a conj(b) ip, the elimination step of all columns: the division by the pivot
// comes after the product.
__device__ __forceinline__ float2 elim(float2 q, float2 a, float2 b, float ip) {
  float2 t = make_float2(0.f, 0.f);
  fma_cb(t, a, b);
  return make_float2(fmaf(-t.x, ip, q.x), fmaf(-t.y, ip, q.y));
}
__device__ __forceinline__ void group_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(CH_GT) : "memory");
}

// 32 dependent steps on a 32 x 32 block by a group of four warps. Lane = row (a column
// for the inverse), warp w holds entries w, w + 4, ... of it: v[u] is entry w + 4 (u0 + u)
// in steps 4 u0 .. 4 u0 + 3. The owner of entry c publishes it, everyone updates the
// rest; entries that are done are updated too, to no effect. A loop, not unrolled
// code: the 3000 instructions that 32 unrolled steps take run once and cost
// 20 us to fetch.
template <int U, class Pub, class Upd>
__device__ __forceinline__ void steps32(float2 (&v)[8], int bar, int first, int last, Pub pub, Upd upd) {
  const int w = (threadIdx.x >> 5) & 3;
#pragma unroll 1
  for (int c0 = first; c0 < last; c0 += 4) {
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      if (w == o) pub(c0 + o, v[0]);
      group_sync(bar);
      upd(c0 + o, [&](auto f) {
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = f(v[u], c0 + 4 * u + w);
      });
    }
#pragma unroll
    for (int u = 0; u + 1 < U; ++u) v[u] = v[u + 1];
  }
}
template <class Pub, class Upd>
__device__ __forceinline__ void steps32_all(float2 (&v)[8], int bar, Pub pub, Upd upd) {
  steps32<8>(v, bar, 0, 16, pub, upd);
  steps32<4>(v, bar, 16, 32, pub, upd);
}

// Elimination of the diagonal block of panel p. diag, the pivots' reciprocals and
// roots and the range of the roots go to every CTA.
__device__ __noinline__ void chol_diag(const float2* __restrict__ W, int real_cols, CholShared* sh, int p, int C) {
  cg::cluster_group cluster = cg::this_cluster();
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 3, gt = threadIdx.x % CH_GT;
  float2 v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = W[lane * WLD + w + 4 * u];
  steps32_all(
      v, 1, [&](int c, float2 x) { sh->diag[c * CH_B + lane] = x; },
      [&](int c, auto each) {
        const float2* col = &sh->diag[c * CH_B];
        const float2 a = col[lane];
        const float ip = 1.0f / col[c].x;
        each([&](float2 q, int t) { return elim(q, a, col[t], ip); });
      });
  const float pv = sh->diag[lane * CH_B + lane].x;
  const unsigned bad = __ballot_sync(0xffffffffu, !(pv > 0.f) || !isfinite(pv));
  const float d = sqrtf(pv), ip = 1.0f / pv;
  float mn = lane < real_cols ? d : INFINITY, mx = lane < real_cols ? d : 0.f;   // without the identity padding
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  const float4* from = reinterpret_cast<const float4*>(sh->diag);
  for (int r = 0; r < C; ++r) {
    CholShared* to = cluster.map_shared_rank(sh, r);
    if (r != (int)cluster.block_rank()) {
      float4* dst = reinterpret_cast<float4*>(to->diag);
#pragma unroll
      for (int e = 0; e < BLK / 2 / CH_GT; ++e) dst[e * CH_GT + gt] = from[e * CH_GT + gt];
    }
    if (w == 0) {
      to->ip[lane] = ip;
      to->d[lane] = d;
      if (lane == 0) {
        to->mn[p] = mn;
        to->mx[p] = mx;
        if (bad) to->bad = 1;
      }
    }
  }
}

// X L_pp^H = A_ip by the same elimination; L_ip (transposed) to every CTA and to fin.
__device__ __noinline__ void chol_solve(const float2* __restrict__ W, CholShared* sh, int i, float2* fin, int bar) {
  cg::cluster_group cluster = cg::this_cluster();
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 3, gt = threadIdx.x % CH_GT;
  float2 v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = W[lane * WLD + w + 4 * u];
  steps32_all(
      v, bar, [&](int c, float2 x) { fin[c * CH_B + lane] = x; },
      [&](int c, auto each) {
        const float2* col = &sh->diag[c * CH_B];
        const float2 a = fin[c * CH_B + lane];
        const float ip = sh->ip[c];
        each([&](float2 q, int t) { return elim(q, a, col[t], ip); });
      });
  float4 l[BLK / 2 / CH_GT];
#pragma unroll
  for (int e = 0; e < BLK / 2 / CH_GT; ++e) {
    float4* f = reinterpret_cast<float4*>(fin) + e * CH_GT + gt;
    const float d = sh->d[(e * CH_GT + gt) / (CH_B / 2)];
    const float4 x = *f;
    l[e] = make_float4(x.x / d, x.y / d, x.z / d, x.w / d);
    *f = l[e];
  }
#pragma unroll
  for (int r = 0; r < CH_C; ++r) {
    float4* dst = reinterpret_cast<float4*>(cluster.map_shared_rank(sh, r)->panel[i]);
#pragma unroll
    for (int e = 0; e < BLK / 2 / CH_GT; ++e) dst[e * CH_GT + gt] = l[e];
  }
}

// T_pp = L_pp^{-1} by substitution, lane = column; to every CTA and to the work block.
__device__ __noinline__ void chol_inv_diag(float2* W, CholShared* sh, int p, int C) {
  cg::cluster_group cluster = cg::this_cluster();
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 3, gt = threadIdx.x % CH_GT;
  float2 v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = make_float2(w + 4 * u == lane ? 1.f : 0.f, 0.f);
  float2* T = sh->panel[p];
  steps32_all(
      v, 1,
      [&](int l, float2 x) {
        // column l is (1, 0) still and those above it 0: a zero numerator would send
        // the division to its slow path (22 thousand cycles for the block, not 15)
        const float d = sh->d[l];
        if (lane < l) x = make_float2(x.x / d, x.y / d);
        else if (lane == l) x.x = 1.0f / d;
        T[l * CH_B + lane] = x;
        W[l * WLD + lane] = x;
      },
      [&](int l, auto each) {
        const float2* col = &sh->lpp[l * CH_B];
        const float2 t = T[l * CH_B + lane];
        each([&](float2 o, int r) {
          const float2 q = col[r];
          o.x = fmaf(-q.x, t.x, o.x);
          o.x = fmaf(q.y, t.y, o.x);
          o.y = fmaf(-q.x, t.y, o.y);
          o.y = fmaf(-q.y, t.x, o.y);
          return o;
        });
      });
  const float4* from = reinterpret_cast<const float4*>(T);
  for (int r = 0; r < C; ++r) {
    if (r == (int)cluster.block_rank()) continue;
    float4* dst = reinterpret_cast<float4*>(cluster.map_shared_rank(sh, r)->panel[p]);
#pragma unroll
    for (int e = 0; e < BLK / 2 / CH_GT; ++e) dst[e * CH_GT + gt] = from[e * CH_GT + gt];
  }
}

// G (k x k, row-major with leading dimension ldg, Hermitian up to rounding)
// = R^H R with R upper triangular. Writes R and R^{-1} (k x k row-major,
// zero below the diagonal). series != 0 allows the first-order form for a Gram
// matrix close to the identity: with E = G - I and ||E||_F <= series_tol,
// R = I + U, R^{-1} = I - U where U is E's strict upper part plus half its
// diagonal (the neglected terms are O(||E||^2)).
//
// With L = R^H and T = L^{-1}, panel p of 32 columns of the blocked elimination of
// [G | I] is
//   L_pp, T_pp = L_pp^{-1}, L_ip = A_ip L_pp^{-H}, T_pj = T_pp W_pj,
//   A_ij -= L_ip L_jp^H (i >= j > p),  W_ij -= L_ip T_pj (i > p >= j).
// It is a chain of small dependent steps, so the time is latency: one CTA of 1024
// threads with G, L and T in L2 took 640 us at k = 256, of which the block products
// 500 (two shared-memory loads per four FMAs, one block at a time) and the 256
// elimination steps, each behind a barrier of the whole CTA, 100. Here a cluster of
// eight CTAs keeps all blocks in shared memory. The lower blocks are dealt out in
// row order, which leaves each CTA the same number of active ones in every panel;
// the panel's L_ip and T_pj are written to every CTA as they are formed. Diagonal
// blocks and substitutions are left to groups of four warps; the W products wait
// for the next diagonal block's elimination, which they overlap. Nothing goes to
// memory before the end: a cluster barrier waits for the stores before it.
// k = 256: full form 640 -> 179 us, first-order form 230 -> 33 us; k = 64:
// 62 -> 41 (a launch of some 8 us included).
__global__ void __launch_bounds__(CH_T, 1)
    chol_inv_kernel(const double2* __restrict__ G, int64_t ldg, int k, int nb, double2* __restrict__ R,
                    double2* __restrict__ Rinv, float ratio, int series, float series_tol,
                    int32_t* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char chol_sm[];
  CholShared* sh = reinterpret_cast<CholShared*>(chol_sm);
  __shared__ float red_s[CH_T / 32];
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = nb * (nb + 1) / 2;
  double2* stage = reinterpret_cast<double2*>(&sh->panel[0][0]);   // [CH_SLOTS][32][WLD], until the panels

  // ---- own blocks of the Hermitian part of G, identity padding
  for (int idx = rank, sl = 0; idx < nblk; idx += C, ++sl) {
    int bi, bj;
    tri_decode(idx, bi, bj);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int e = tid + q * CH_T;
      const int r = e / CH_B, c = e % CH_B, gi = bj * CH_B + r, gj = bi * CH_B + c;
      if (e < BLK)
        stage[(sl * CH_B + r) * WLD + c] = gi < k && gj < k ? G[gi * ldg + gj] : make_double2(0.0, 0.0);
    }
  }
  __syncthreads();
  float nrm = 0.f;
  for (int idx = rank, sl = 0; idx < nblk; idx += C, ++sl) {
    int bi, bj;
    tri_decode(idx, bi, bj);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int e = tid + q * CH_T;
      const int r = e / CH_B, c = e % CH_B, gi = bi * CH_B + r, gj = bj * CH_B + c;
      float2 v = make_float2(gi == gj ? 1.f : 0.f, 0.f);
      if (e < BLK) {
        if (gi < k && gj < k) {
          const double2 a = G[gi * ldg + gj], b = stage[(sl * CH_B + c) * WLD + r];
          v = make_float2(0.5f * (float)(a.x + b.x), 0.5f * (float)(a.y - b.y));
          const float ex = v.x - (gi == gj ? 1.f : 0.f);
          nrm = fmaf(bi == bj ? 1.f : 2.f, fmaf(ex, ex, v.y * v.y), nrm);
        }
        sh->work[sl][r * WLD + c] = v;
      }
    }
  }
  if (tid == 0) sh->bad = 0;
  if (series) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    if (lane == 0) red_s[warp] = nrm;
    __syncthreads();
    cluster.sync();                    // every CTA runs
    if (tid < C) {
      float t = 0.f;
      for (int w = 0; w < CH_T / 32; ++w) t += red_s[w];
      cluster.map_shared_rank(sh, tid)->acc[rank] = t;
    }
    cluster.sync();
    float t = 0.f;
    for (int r = 0; r < C; ++r) t += sh->acc[r];
    if (sqrtf(t) <= series_tol) {      // the same sum in every CTA
      for (int idx = rank, sl = 0; idx < nblk; idx += C, ++sl) {
        int bj, bi;                    // upper block (bi, bj): what is staged; the lower one is read again
        tri_decode(idx, bj, bi);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int e = tid + q * CH_T;
          const int r = e / CH_B, c = e % CH_B, gi = bj * CH_B + r, gj = bi * CH_B + c;
          if (e < BLK && gi < k && gj < k) {
            // E's entry (gj, gi) above the diagonal into the stage
            const double2 b = G[gi * ldg + gj];
            double2* a = &stage[(sl * CH_B + c) * WLD + r];
            *a = gi == gj ? make_double2(0.5 * (b.x - 1.0), 0.0)
                          : (gi > gj ? make_double2(0.5 * (a->x + b.x), 0.5 * (a->y - b.y)) : *a);
            if (bi != bj) {
              R[(int64_t)gi * k + gj] = make_double2(0.0, 0.0);
              Rinv[(int64_t)gi * k + gj] = make_double2(0.0, 0.0);
            }
          }
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int e = tid + q * CH_T;
          const int r = e / CH_B, c = e % CH_B, i = bi * CH_B + r, j = bj * CH_B + c;
          if (e >= BLK || i >= k || j >= k) continue;
          const double2 u = j >= i ? stage[(sl * CH_B + r) * WLD + c] : make_double2(0.0, 0.0);
          const double one = (i == j) ? 1.0 : 0.0;
          R[(int64_t)i * k + j] = make_double2(one + u.x, u.y);
          Rinv[(int64_t)i * k + j] = make_double2(one - u.x, -u.y);
        }
      }
      return;
    }
  }
  cluster.sync();

  const int tx = tid & 15, ty = (tid >> 4) & 15;
  for (int p = 0; p < nb; ++p) {
    const int pd = p * (p + 1) / 2 + p;                  // index of block (p, p)
    // ---- L_pp; elsewhere W_ij -= L_i,p-1 T_p-1,j
    if (tid >= CH_UT) {
      if (pd % C == rank) chol_diag(sh->work[pd / C], k - p * CH_B, sh, p, C);
    } else if (p > 0) {
      for (int idx = rank, sl = 0; idx < nblk; idx += C, ++sl) {
        int bi, bj;
        tri_decode(idx, bi, bj);
        if (bi < p || bj >= p) continue;
        float2 acc[2][2] = {};
        block_mul<false>(sh->panel[bi], sh->panel[bj], ty, tx, acc);
        float2* W = sh->work[sl];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            float2* w = &W[(ty + 16 * u) * WLD + tx + 16 * v];
            const float2 o = bj == p - 1 ? make_float2(0.f, 0.f) : *w;   // W starts at zero
            *w = make_float2(o.x - acc[u][v].x, o.y - acc[u][v].y);
          }
      }
    }
    if (pd % C == rank) {
      __syncthreads();
      for (int e = tid; e < BLK; e += CH_T) {
        const int c = e / CH_B, r = e % CH_B;
        const float2 a = sh->diag[e];
        const float d = sh->d[c];
        const float2 l = r < c ? make_float2(0.f, 0.f) : (r == c ? make_float2(d, 0.f) : make_float2(a.x / d, a.y / d));
        sh->lpp[e] = l;
        sh->fin[pd / C][e] = l;
      }
    }
    cluster.sync();
    if (sh->bad) {                                       // the same in every CTA
      if (rank == 0 && tid == 0) atomicExch(status, PTN_ERR_NOCONVERGE);
      return;
    }
    // ---- L_ip; T_pp
    if (tid >= CH_UT) {
      if (pd % C == rank) chol_inv_diag(sh->work[pd / C], sh, p, C);
    } else {
      int job = 0;
      for (int idx = rank, sl = 0; idx < nblk; idx += C, ++sl) {
        int bi, bj;
        tri_decode(idx, bi, bj);
        if (bj != p || bi == p) continue;
        if ((job++ & 1) == tid / CH_GT) chol_solve(sh->work[sl], sh, bi, sh->fin[sl], 2 + tid / CH_GT);
      }
    }
    cluster.sync();
    // ---- A_ij -= L_ip L_jp^H; T_pj = T_pp W_pj
    if (tid < CH_UT) {
      for (int idx = rank, sl = 0; idx < nblk; idx += C, ++sl) {
        int bi, bj;
        tri_decode(idx, bi, bj);
        float2* W = sh->work[sl];
        float2 acc[2][2] = {};
        if (bj > p) {
          block_mul<true>(sh->panel[bi], sh->panel[bj], ty, tx, acc);
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
              float2* w = &W[(ty + 16 * u) * WLD + tx + 16 * v];
              *w = make_float2(w->x - acc[u][v].x, w->y - acc[u][v].y);
            }
        } else if (bi == p && bj < p) {
          const float2* T = sh->panel[p];
#pragma unroll 8
          for (int c = 0; c < CH_B; ++c) {               // T_pp is zero above its diagonal
            const float2 a0 = T[ty * CH_B + c], a1 = T[(ty + 16) * CH_B + c];
            const float2 b0 = W[c * WLD + tx], b1 = W[c * WLD + tx + 16];
            fma_c(acc[0][0], a0, b0);
            fma_c(acc[0][1], a0, b1);
            fma_c(acc[1][0], a1, b0);
            fma_c(acc[1][1], a1, b1);
          }
          asm volatile("bar.sync 4, %0;" ::"n"(CH_UT) : "memory");   // W has been read
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) W[(ty + 16 * u) * WLD + tx + 16 * v] = acc[u][v];
          if (p + 1 < nb)
            for (int r = 0; r < C; ++r) {
              float2* dst = cluster.map_shared_rank(sh, r)->panel[bj];
#pragma unroll
              for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int v = 0; v < 2; ++v) dst[(ty + 16 * u) * CH_B + tx + 16 * v] = acc[u][v];
            }
        }
      }
    }
    cluster.sync();
  }
  float mn = INFINITY, mx = 0.f;
  for (int p = 0; p < nb; ++p) {
    mn = fminf(mn, sh->mn[p]);
    mx = fmaxf(mx, sh->mx[p]);
  }
  if (!(mn > ratio * mx)) {                              // the same in every CTA
    if (rank == 0 && tid == 0) atomicExch(status, PTN_ERR_NOCONVERGE);
    return;
  }
  // ---- R = L^H, R^{-1} = T^H: block (bj, bi) from L_ij and T_ij, zeros below the diagonal
  for (int idx = rank, sl = 0; idx < nblk; idx += C, ++sl) {
    int bi, bj;
    tri_decode(idx, bi, bj);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int e = tid + q * CH_T;
      const int c = e / CH_B, r = e % CH_B, row = bj * CH_B + c, col = bi * CH_B + r;
      if (e >= BLK || row >= k || col >= k) continue;
      const float2 l = sh->fin[sl][c * CH_B + r], t = sh->work[sl][r * WLD + c];
      R[(int64_t)row * k + col] = make_double2((double)l.x, -(double)l.y);
      Rinv[(int64_t)row * k + col] = make_double2((double)t.x, -(double)t.y);
    }
    if (bi == bj) continue;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int e = tid + q * CH_T;
      const int r = e / CH_B, c = e % CH_B, row = bi * CH_B + r, col = bj * CH_B + c;
      if (e >= BLK || row >= k || col >= k) continue;
      R[(int64_t)row * k + col] = make_double2(0.0, 0.0);
      Rinv[(int64_t)row * k + col] = make_double2(0.0, 0.0);
    }
  }
}

// C[i][j] = sum_{l=i..j} A[i][l] B[l][j] for upper-triangular A, B (k x k row-major),
// or with NEWTON 2 A[i][j] - that sum: the Newton step R = R0 (2I - W) with A = R0 and
// W = X R0.
//
// The FP64 pipe bounds it: k^3 / 6 products of four instructions, each of which
// holds one of an SM's four schedulers for 64 cycles whatever its active lanes; 19 us
// at k = 256 when all 608 of them share the work. A warp that sums a row of
// 256 by itself takes 35 us, so a CTA is one row and 32 columns, and its four
// warps (one per scheduler) take every fourth l. The longest sums come first.
// k = 256: 69 -> 34 us (a launch of some 8 us included).
constexpr int TRI_W = 4;
template <bool NEWTON>
__global__ void __launch_bounds__(32 * TRI_W) tri_mul_kernel(const double2* __restrict__ A,
                                                             const double2* __restrict__ B,
                                                             double2* __restrict__ C, int64_t k, int64_t ncb) {
  __shared__ double2 part[TRI_W][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t jb = ncb - 1 - blockIdx.x / k, i = blockIdx.x % k, j = jb * 32 + lane;
  const int64_t last = min(jb * 32 + 31, k - 1);
  if (i > last) {
    if (warp == 0 && j < k) C[i * k + j] = make_double2(0.0, 0.0);
    return;
  }
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int64_t l = i + warp; l <= last; l += TRI_W)
    if (l <= j && j < k) acc = cfma(A[i * k + l], B[l * k + j], acc);
  part[warp][lane] = acc;
  __syncthreads();
  if (warp != 0 || j >= k) return;
#pragma unroll
  for (int w = 1; w < TRI_W; ++w) acc = cadd(acc, part[w][lane]);
  if (NEWTON) {
    const double2 r0 = j >= i ? A[i * k + j] : make_double2(0.0, 0.0);
    acc = j >= i ? make_double2(2.0 * r0.x - acc.x, 2.0 * r0.y - acc.y) : make_double2(0.0, 0.0);
  }
  C[i * k + j] = acc;
}

template <bool NEWTON>
int launch_tri(const void* A, const void* B, void* C, int64_t k, cudaStream_t s) {
  const int64_t ncb = (k + 31) / 32;
  if (k * ncb > 0x7fffffffLL) return PTN_ERR_UNSUPPORTED;
  PTN_COUNT(1);
  tri_mul_kernel<NEWTON><<<(unsigned)(k * ncb), 32 * TRI_W, 0, s>>>(
      static_cast<const double2*>(A), static_cast<const double2*>(B), static_cast<double2*>(C), k, ncb);
  return ptn_launch_status();
}

// out[0] = 1 + the largest row index i with a nonzero entry (0 when A is zero);
// out must start at 0.
__global__ void nonzero_rows_kernel(const double2* __restrict__ A, const int64_t* __restrict__ rowoff, int64_t m,
                                        int64_t k, int64_t cs, unsigned long long* __restrict__ out) {
  const int64_t total = m * k;
  int64_t best = -1;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / k, c = e - (e / k) * k;
    const double2 v = A[rowoff[i] + c * cs];
    if ((v.x != 0.0 || v.y != 0.0) && i > best) best = i;
  }
  unsigned long long b = (unsigned long long)(best + 1);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long x = __shfl_xor_sync(0xffffffffu, b, o);
    b = x > b ? x : b;
  }
  if ((threadIdx.x & 31) == 0 && b > 0) atomicMax(out, b);
}

__global__ void init_u64_kernel(unsigned long long* p) { *p = 0ull; }

inline int64_t kpad(int64_t k) { return (k + CH_B - 1) / CH_B * CH_B; }

}  // namespace

extern "C" int64_t ptn_zchol_work_bytes(int64_t k) {
  if (k < 1) return 0;
  const int64_t kp = kpad(k);
  return 2 * kp * kp * (int64_t)sizeof(float2) + 256;
}

extern "C" int64_t ptn_zchol_max_k(void) { return CH_MAXK; }

extern "C" int ptn_zchol_upper(const void* G, int64_t ldg, int64_t k, void* R, void* Rinv, double pivot_ratio,
                               int32_t series, double series_tol, int32_t* status, void* work, void* stream) {
  if (!G || !R || !Rinv || !status || !work || k < 1 || ldg < k) return PTN_ERR_ARG;
  if (k > CH_MAXK) return PTN_ERR_UNSUPPORTED;
  if (reinterpret_cast<uintptr_t>(work) & 15) return PTN_ERR_ARG;
  static const cudaError_t attr = cudaFuncSetAttribute(
      chol_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CholShared));
  if (attr != cudaSuccess) return PTN_ERR_LAUNCH;
  const int nb = (int)(kpad(k) / CH_B);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = nb > 1 ? CH_C : 1;               // one block: nothing to share
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.gridDim = dim3(at.val.clusterDim.x);
  cfg.blockDim = dim3(CH_T);
  cfg.dynamicSmemBytes = sizeof(CholShared);
  cfg.stream = ptn_stream(stream);
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  PTN_COUNT(1);
  if (cudaLaunchKernelEx(&cfg, chol_inv_kernel, static_cast<const double2*>(G), ldg, (int)k, nb,
                         static_cast<double2*>(R), static_cast<double2*>(Rinv), (float)pivot_ratio,
                         series ? 1 : 0, (float)series_tol, status) != cudaSuccess)
    return PTN_ERR_LAUNCH;
  return ptn_launch_status();
}

extern "C" int ptn_ztri_mul_upper(const void* A, const void* B, void* C, int64_t k, void* stream) {
  if (!A || !B || !C || k < 1) return PTN_ERR_ARG;
  if (C == A || C == B) return PTN_ERR_ARG;
  return launch_tri<false>(A, B, C, k, ptn_stream(stream));
}

extern "C" int ptn_ztri_inv_newton(const void* X, const void* R0, void* R, void* work, int64_t k, void* stream) {
  if (!X || !R0 || !R || !work || k < 1) return PTN_ERR_ARG;
  if (R == X || R == R0 || work == X || work == R0 || work == R) return PTN_ERR_ARG;
  const int st = launch_tri<false>(X, R0, work, k, ptn_stream(stream));
  return st == PTN_OK ? launch_tri<true>(R0, work, R, k, ptn_stream(stream)) : st;
}

extern "C" int ptn_znonzero_rows(const void* A, const int64_t* rowoff, int64_t m, int64_t k, int64_t colstride,
                                     int64_t* out, void* stream) {
  if (!A || !rowoff || !out || m < 1 || k < 1 || colstride < 1) return PTN_ERR_ARG;
  cudaStream_t s = ptn_stream(stream);
  unsigned long long* o = reinterpret_cast<unsigned long long*>(out);
  PTN_COUNT(2);
  init_u64_kernel<<<1, 1, 0, s>>>(o);
  int64_t blocks = (m * k + 255) / 256;
  if (blocks > 1216) blocks = 1216;   // 8 CTAs per SM on 152 SMs
  nonzero_rows_kernel<<<(unsigned)blocks, 256, 0, s>>>(static_cast<const double2*>(A), rowoff, m, k, colstride,
                                                           o);
  return ptn_launch_status();
}
