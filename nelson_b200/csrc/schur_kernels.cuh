// schur_kernels.cuh -- reduced camera system S = U - W V^-1 W' and back-substitution.
//
// The algebra of SolverCholeskySchur::computeIncrement
// (nelson/SolverCholeskySchur.hpp:91-157), laid out the way
// SolverDiagonalBlocksInverseWWtMultSchur runs it
// (nelson/SolverDiagonalBlocksInverseWWtMultSchur.hpp:99-140):
//   vinv_kernel      MatrixDiagInv::compute (nelson/MatrixDiagInv.hpp:32-43):
//                    Vinv_p = inv(sym_upper(V_p) (1 + rel) + abs), register-resident
//                    3x3 LDL'.
//   wvinv_bs_kernel  MatrixWVinvMultiplier::multiply (MatrixWVinvMultiplier.hpp:33-35)
//                    Y = W Vinv per W block, and bS = -bU + Y bV per camera
//                    (= -bU - W xV0 of SolverCholeskySchur.hpp:114).
//   schur_kernel     MatrixWWtMultiplier::multiply (MatrixWWtMultiplier.hpp:139-152):
//                    S_ij = U_ij - sum_pairs Y_a W_b', the block's pair list in
//                    one or more warps (no float atomics), plus the diagonal damping of
//                    SolverCholeskySchur.hpp:121-124, written to dense lower storage.
//   backsub_kernel   MatrixWtXMultiplier::rightMultVectorSub + MatrixDiagInv::rightMultVector
//                    (MatrixWtXMultiplier.hpp:58-62, MatrixDiagInv.hpp:153-156):
//                    xV_p = Vinv_p (-bV_p - sum W' xU).
#pragma once

#include <type_traits>

#include "nl_common.cuh"

namespace nl {

struct SchurDev {
  int bc, nci, np, nU, nW, nS;
  int n, ld;                   // S size and leading dimension (n padded)
  const int* v_uid;            // point -> V uid (-1: none)
  const int* w_row_ptr;        // nci + 1 (CSR over internal cameras)
  const int* w_col;            // W uid -> point
  const int* w_row;            // W uid -> internal camera
  const int* w_col_ptr;        // np + 1 (CSC over points)
  const int* w_col_uid;        // W uids of a point, rows ascending
  const int* u_diag_uid;       // internal camera -> U uid of its diagonal block (-1: none)
  const int* s_i;              // output block -> block row i (i <= j)
  const int* s_j;              // output block -> block column j
  const int* s_uuid;           // output block -> U uid (-1: none)
  const long long* s_pair_ptr; // nS + 1
  const int* pair_a;           // W uid of (i, p)
  const int* pair_b;           // W uid of (j, p)
};

// ---------------------------------------------------------------------------
template <typename T, int BC>
static __global__ void vinv_kernel(SchurDev d, const T* __restrict__ V, T* __restrict__ Vinv, const double* __restrict__ lam,
                            int* __restrict__ status, int* __restrict__ counter, int* __restrict__ tickets, int ntickets,
                            unsigned long long* __restrict__ call, const int* __restrict__ active) {
  constexpr int LV = Layout<T, BC>::V;
  chain_start(V, lam, active);
  if (active && !*active) return;
  // first kernel of a call: also clears the Schur work counter and the solves'
  // tickets, and numbers the call
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) {
      *counter = 0;
      (*call)++;
    }
    for (int i = threadIdx.x; i < ntickets; i += blockDim.x) tickets[i] = 0;
  }
  const double rel = lam[0], abs = lam[1];
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= d.np) return;
  const int q = d.v_uid[p];
  double a00 = 0, a01 = 0, a02 = 0, a11 = 0, a12 = 0, a22 = 0;
  if (q >= 0) {
    const T* v = V + (size_t)q * LV;
    a00 = v[0]; a01 = v[1]; a02 = v[2];
    a11 = v[4]; a12 = v[5]; a22 = v[8];
  }
  if (rel != 0.0 || abs != 0.0) {
    a00 = a00 * (1.0 + rel) + abs;
    a11 = a11 * (1.0 + rel) + abs;
    a22 = a22 * (1.0 + rel) + abs;
  }
  // LDL' of the symmetric 3x3 block (from its upper triangle)
  const double d0 = a00;
  const double l10 = a01 / d0, l20 = a02 / d0;
  const double d1 = a11 - l10 * a01;
  const double l21 = (a12 - l20 * a01) / d1;
  const double d2 = a22 - l20 * a02 - l21 * l21 * d1;
  const bool ok = d0 > 0.0 && d1 > 0.0 && d2 > 0.0 && isfinite(d0 + d1 + d2);
  if (!ok) atomicOr(status, ST_VINV_FAIL);
  // inv(L') D^-1 inv(L):  inv(L) = [[1,0,0],[-l10,1,0],[l10 l21 - l20, -l21, 1]]
  const double m10 = -l10, m21 = -l21, m20 = l10 * l21 - l20;
  const double i0 = 1.0 / d0, i1 = 1.0 / d1, i2 = 1.0 / d2;
  const double b00 = i0 + m10 * m10 * i1 + m20 * m20 * i2;
  const double b01 = m10 * i1 + m20 * m21 * i2;
  const double b02 = m20 * i2;
  const double b11 = i1 + m21 * m21 * i2;
  const double b12 = m21 * i2;
  const double b22 = i2;
  T* o = Vinv + (size_t)p * LV;
  o[0] = (T)b00; o[1] = (T)b01; o[2] = (T)b02;
  o[3] = (T)b01; o[4] = (T)b11; o[5] = (T)b12;
  o[6] = (T)b02; o[7] = (T)b12; o[8] = (T)b22;
}

// ---------------------------------------------------------------------------
// One CTA per camera, one W block per lane.  The 32 blocks of a warp are
// consecutive: they pass through shared memory so that every access to W and Y is
// to whole lines (a lane reading its own 112 bytes takes 32 lines per access).
// Bound by the L1 lines of the Vinv / bV gather.  375k blocks of 9x3 FP32 33 -> 24
// us, FP64 67 -> 55 us, 1,500 cameras 338 -> 184 us; several CTAs per camera were
// slower (28 us: the sums wait for the stores).
template <typename T, int BC, int NT>
constexpr size_t wvinv_smem() {
  return sizeof(T) * NT * Layout<T, BC>::W;
}
template <typename T, int BC, int NT>
static __global__ void __launch_bounds__(NT) wvinv_bs_kernel(SchurDev d, const T* __restrict__ W,
                                                      const T* __restrict__ Vinv, T* __restrict__ Y,
                                                      const T* __restrict__ bU, const T* __restrict__ bV,
                                                      double* __restrict__ bS, const int* __restrict__ active) {
  constexpr int LW = Layout<T, BC>::W;
  constexpr int LV = Layout<T, BC>::V;
  using V16 = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  constexpr int EPV = 16 / (int)sizeof(T), PW = LW / EPV;  // elements per piece, pieces per block
  extern __shared__ float4 w_stage[];
  __shared__ double red[NT / 32][BC];
  chain_start(W, Vinv, bU, bV, active);
  if (active && !*active) return;
  const int c = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  V16* st = reinterpret_cast<V16*>(w_stage) + warp * 32 * PW;
  double acc[BC];
#pragma unroll
  for (int i = 0; i < BC; i++) acc[i] = 0.0;
  const int end = d.w_row_ptr[c + 1];
  for (int q0 = d.w_row_ptr[c] + warp * 32; q0 < end; q0 += NT) {
    const int m = min(32, end - q0);
    const V16* src = reinterpret_cast<const V16*>(W + (size_t)q0 * LW);
    V16 in[PW];
#pragma unroll
    for (int i = 0; i < PW; i++)
      if (lane + 32 * i < m * PW) in[i] = src[lane + 32 * i];
#pragma unroll
    for (int i = 0; i < PW; i++)
      if (lane + 32 * i < m * PW) st[lane + 32 * i] = in[i];
    __align__(16) T v[LV];
    T bv0 = 0, bv1 = 0, bv2 = 0;
    if (lane < m) {
      const int p = d.w_col[q0 + lane];
#pragma unroll
      for (int i = 0; i < LV / EPV; i++)
        reinterpret_cast<V16*>(v)[i] = reinterpret_cast<const V16*>(Vinv + (size_t)p * LV)[i];
      bv0 = bV[3 * (size_t)p];
      bv1 = bV[3 * (size_t)p + 1];
      bv2 = bV[3 * (size_t)p + 2];
    }
    __syncwarp();
    if (lane < m) {
      __align__(16) T w[LW];
#pragma unroll
      for (int i = 0; i < PW; i++) reinterpret_cast<V16*>(w)[i] = st[lane * PW + i];
#pragma unroll
      for (int i = 0; i < BC; i++) {
        const T w0 = w[i * 3], w1 = w[i * 3 + 1], w2 = w[i * 3 + 2];
        const T y0 = w0 * v[0] + w1 * v[3] + w2 * v[6];
        const T y1 = w0 * v[1] + w1 * v[4] + w2 * v[7];
        const T y2 = w0 * v[2] + w1 * v[5] + w2 * v[8];
        w[i * 3] = y0;
        w[i * 3 + 1] = y1;
        w[i * 3 + 2] = y2;
        acc[i] += (double)y0 * (double)bv0 + (double)y1 * (double)bv1 + (double)y2 * (double)bv2;
      }
#pragma unroll
      for (int i = BC * 3; i < LW; i++) w[i] = (T)0;
#pragma unroll
      for (int i = 0; i < PW; i++) st[lane * PW + i] = reinterpret_cast<const V16*>(w)[i];
    }
    __syncwarp();
    V16* dst = reinterpret_cast<V16*>(Y + (size_t)q0 * LW);
#pragma unroll
    for (int i = 0; i < PW; i++)
      if (lane + 32 * i < m * PW) dst[lane + 32 * i] = st[lane + 32 * i];
    __syncwarp();
  }
#pragma unroll
  for (int i = 0; i < BC; i++) {
    const double v = warp_sum(acc[i]);
    if (lane == 0) red[warp][i] = v;
  }
  __syncthreads();
  if (threadIdx.x < BC) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < NT / 32; w++) s += red[w][threadIdx.x];
    bS[(size_t)c * BC + threadIdx.x] = -(double)bU[(size_t)c * BC + threadIdx.x] + s;
  }
}

// ---------------------------------------------------------------------------
// S_ij = U_ij - sum_pairs Y_a W_b'.  A work item is one warp's share of an
// output block: `chunk` pairs of its list at most, so that the long lists (the
// diagonal blocks: every observation of a camera) are spread over many warps.
// Items are taken from a work counter, longest first.  The partial sums of a
// block of several items are added by whichever of its warps finishes last, in
// item order, so S does not depend on the schedule and no warp waits.
//
// Inside an item the pairs' blocks are copied to shared memory as they are
// (16-byte asynchronous copies, kStages batches in flight per warp), and a lane
// owns a TR x TR tile of the result (TR = 3, or 2 for BC = 2) of one pair in
// flight: (BC / TR)^2 lanes a pair, G pairs side by side, so a lane reads 6 TR
// values for 3 TR^2 FMAs.  A batch's products are summed before they join the
// running sum (blocked summation: a diagonal block sums thousands of pairs in
// the working precision).
//
// One warp per block was bound by the longest list on small scenes and by the
// re-laying of the operands in padded rows (a register round trip and scalar
// stores) on large ones.  200 cameras, 1.6 M pairs: 100 us against 413 us in
// FP32, 177 against 578 us in FP64; 1,500 cameras, 16.5 M pairs (3.7 GB of
// gathered blocks): 0.87 ms against 1.71.  Two stages of 12 pairs (9 x 9 blocks)
// measured 100 / 871 us; three stages 122 / 936, two of 15 pairs 105 / 883,
// three of 6 pairs 113 / 910.
template <typename T, int BC>
struct SchurCfg {
  static constexpr int LW = Layout<T, BC>::W;
  static constexpr int TR = BC % 3 == 0 ? 3 : 2;
  static constexpr int TD = BC / TR;                // tiles along a block row
  static constexpr int LP = TD * TD;                // lanes per pair
  static constexpr int G = 32 / LP;                 // pairs side by side
  static constexpr int ROUNDS = G >= 32 ? 1 : G >= 8 ? 2 : 4;
  static constexpr int PB = G * ROUNDS;             // pairs per batch (<= 32)
  static constexpr int kStages = 2;
  static constexpr int kWarps = 8;
  static constexpr int VB = LW * (int)sizeof(T) / 16;  // 16-byte vectors per block
  static constexpr size_t kSmem = (size_t)kWarps * kStages * 2 * PB * LW * sizeof(T);
};

// one work item: pairs [first, first + chunk) of a block's list
struct SchurItem {
  int block, part;
};

template <typename T, int BC>
static __global__ void __launch_bounds__(SchurCfg<T, BC>::kWarps * 32)
    schur_kernel(SchurDev d, const T* __restrict__ U, const T* __restrict__ Y, const T* __restrict__ W,
                 const double* __restrict__ lam, T* __restrict__ S, T* __restrict__ S0,
                 const SchurItem* __restrict__ items, int nitems, int chunk, const int* __restrict__ slot,
                 T* __restrict__ partial, int* __restrict__ arrived, int* __restrict__ counter,
                 const int* __restrict__ active) {
  using Cfg = SchurCfg<T, BC>;
  constexpr int LW = Cfg::LW, LU = Layout<T, BC>::U, TR = Cfg::TR, TD = Cfg::TD, LP = Cfg::LP, G = Cfg::G,
                ROUNDS = Cfg::ROUNDS, PB = Cfg::PB, kStages = Cfg::kStages, VB = Cfg::VB;
  extern __shared__ float4 schur_smem[];
  chain_start(U, Y, W, lam, active);
  if (active && !*active) return;
  const double rel = lam[0], abs = lam[1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T* const sh = reinterpret_cast<T*>(schur_smem) + (size_t)warp * kStages * 2 * PB * LW;
  const uint32_t sh_a = (uint32_t)__cvta_generic_to_shared(sh);
  const int q = lane / LP, tile = lane % LP;  // pair slot, tile of the block
  const int r0 = TR * (tile / TD), c0 = TR * (tile % TD);
  const bool on = q < G;
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = atomicAdd(counter, 1);
    idx = __shfl_sync(0xffffffffu, idx, 0);
    if (idx >= nitems) break;
    const SchurItem item = items[idx];
    const int b = item.block;
    const long long pb = d.s_pair_ptr[b], pe = d.s_pair_ptr[b + 1];
    const long long p0 = pb + (long long)item.part * chunk;
    const int cnt = (int)min((long long)chunk, pe - p0), nbatch = (cnt + PB - 1) / PB;
    // UIDs of a batch's blocks: lane l holds pair l's
    int ua = 0, ub = 0;
    auto load_uids = [&](int t) {
      if (lane < PB && t * PB + lane < cnt) {
        ua = __ldg(d.pair_a + p0 + t * PB + lane);
        ub = __ldg(d.pair_b + p0 + t * PB + lane);
      }
    };
    // the 2 n blocks of batch t, Y blocks first, into its stage
    auto copy_batch = [&](int t) {
      const int n = min(PB, cnt - t * PB);
      const uint32_t dst = sh_a + (uint32_t)((t % kStages) * 2 * PB * LW * (int)sizeof(T));
#pragma unroll
      for (int v0 = 0; v0 < 2 * PB * VB; v0 += 32) {
        const int v = v0 + lane, blk = v / VB, part = v - blk * VB;
        const int pair = blk < PB ? blk : blk - PB;
        const int y = __shfl_sync(0xffffffffu, ua, pair & 31), w = __shfl_sync(0xffffffffu, ub, pair & 31);
        if (blk < 2 * PB && pair < n) {
          const T* src = (blk < PB ? Y + (size_t)y * LW : W + (size_t)w * LW) + part * (16 / (int)sizeof(T));
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16u * (uint32_t)v), "l"(src) : "memory");
        }
      }
    };
    T acc[TR][TR];
#pragma unroll
    for (int i = 0; i < TR; i++)
#pragma unroll
      for (int j = 0; j < TR; j++) acc[i][j] = (T)0;
    load_uids(0);
#pragma unroll
    for (int t = 0; t < kStages - 1; t++) {
      if (t < nbatch) {
        copy_batch(t);
        load_uids(t + 1);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int t = 0; t < nbatch; t++) {
      if (t + kStages - 1 < nbatch) {
        copy_batch(t + kStages - 1);
        load_uids(t + kStages);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      asm volatile("cp.async.wait_group %0;\n" ::"n"(kStages - 1) : "memory");
      __syncwarp();
      const T* st = sh + (t % kStages) * 2 * PB * LW;
      T part[TR][TR];
#pragma unroll
      for (int i = 0; i < TR; i++)
#pragma unroll
        for (int j = 0; j < TR; j++) part[i][j] = (T)0;
#pragma unroll
      for (int r = 0; r < ROUNDS; r++) {
        const int pair = r * G + q;
        if (on && t * PB + pair < cnt) {
          const T* y = st + pair * LW + 3 * r0;
          const T* w = st + (PB + pair) * LW + 3 * c0;
          T yv[TR][3], wv[TR][3];
#pragma unroll
          for (int i = 0; i < TR; i++)
#pragma unroll
            for (int m = 0; m < 3; m++) {
              yv[i][m] = y[3 * i + m];
              wv[i][m] = w[3 * i + m];
            }
#pragma unroll
          for (int i = 0; i < TR; i++)
#pragma unroll
            for (int j = 0; j < TR; j++)
#pragma unroll
              for (int m = 0; m < 3; m++) part[i][j] += yv[i][m] * wv[j][m];
        }
      }
#pragma unroll
      for (int i = 0; i < TR; i++)
#pragma unroll
        for (int j = 0; j < TR; j++) acc[i][j] += part[i][j];
      __syncwarp();  // the stage is free for the copy of the next iteration
    }
    // the pair slots' sums, onto slot 0 in a fixed order
    if (G == 3) {
#pragma unroll
      for (int i = 0; i < TR; i++)
#pragma unroll
        for (int j = 0; j < TR; j++) {
          const T x = __shfl_down_sync(0xffffffffu, acc[i][j], LP), z = __shfl_down_sync(0xffffffffu, acc[i][j], 2 * LP);
          acc[i][j] += x + z;
        }
    } else {
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < TR; i++)
#pragma unroll
          for (int j = 0; j < TR; j++) acc[i][j] += __shfl_down_sync(0xffffffffu, acc[i][j], o * LP);
    }
    const int sl = slot[b];  // first partial of a block of several items, -1 otherwise
    if (sl >= 0) {
      const int nparts = (int)((pe - pb + chunk - 1) / chunk);
      T* mine = partial + (size_t)(sl + item.part) * LU;
      if (lane < LP) {
#pragma unroll
        for (int i = 0; i < TR; i++)
#pragma unroll
          for (int j = 0; j < TR; j++) mine[(r0 + i) * BC + c0 + j] = acc[i][j];
      }
      __threadfence();
      __syncwarp();
      int last = 0;
      if (lane == 0) {
        last = atomicAdd(arrived + b, 1) == nparts - 1;
        if (last) arrived[b] = 0;  // for the next call
      }
      if (!__shfl_sync(0xffffffffu, last, 0)) continue;
      __threadfence();
      if (lane < LP) {
#pragma unroll
        for (int i = 0; i < TR; i++)
#pragma unroll
          for (int j = 0; j < TR; j++) acc[i][j] = (T)0;
        for (int k = 0; k < nparts; k++) {
          const T* p = partial + (size_t)(sl + k) * LU;
#pragma unroll
          for (int i = 0; i < TR; i++)
#pragma unroll
            for (int j = 0; j < TR; j++) acc[i][j] += __ldcg(p + (r0 + i) * BC + c0 + j);
        }
      }
    }
    // damping on the diagonal of diagonal blocks, then the store (lower storage:
    // S_lower[j*BC + c][i*BC + r] = S_ij[r][c])
    if (lane < LP) {
      const int bi = d.s_i[b], bj = d.s_j[b], uu = d.s_uuid[b];
#pragma unroll
      for (int i = 0; i < TR; i++)
#pragma unroll
        for (int j = 0; j < TR; j++) {
          const int r = r0 + i, cc = c0 + j;
          const T u = uu >= 0 ? U[(size_t)uu * LU + r * BC + cc] : (T)0;
          T val = u - acc[i][j];
          if (bi == bj && r == cc && (rel != 0.0 || abs != 0.0)) {
            const int ud = d.u_diag_uid[bi];
            const double udg = ud >= 0 ? (double)U[(size_t)ud * LU + r * BC + r] : 0.0;
            val = (T)((double)val + rel * udg + abs);
          }
          const size_t o = (size_t)(bj * BC + cc) * d.ld + (size_t)(bi * BC + r);
          if (bi != bj || cc >= r) {
            S[o] = val;
            if (S0) S0[o] = val;
          }
        }
    }
  }
}

// Zero S (and S0), with the identity on the padded rows n .. ld - 1.  With
// env_first and *dirty zero only the tiles that can hold nonzeros: row r of tile
// row I over columns [env_first[I] NB, (I + 1) NB), the Cholesky envelope.  The
// other tiles are zero after a full clear and stay exactly zero: the Schur blocks
// lie inside the envelope, and the factorisation writes only zeros there (TRSM
// and trailing updates of zero tiles) as long as it does not fail.  *dirty says on the
// device whether that holds (set from the start and by a failed call, cleared by
// any other, in backsub_kernel), so that it is right for launches that are captured,
// replayed or skipped by `active` as well.  One CTA per row.
template <typename T>
static __global__ void clear_kernel(T* __restrict__ S, T* __restrict__ S0, int n, int ld, int nb,
                                    const int* __restrict__ env_first, const int* __restrict__ dirty,
                                    const int* __restrict__ active) {
  chain_start(dirty, active);
  const int r = blockIdx.x, I = r / nb;
  // the three loads together, not one after another (64 cameras 2.1 -> 1.9 us)
  const int first = env_first ? env_first[I] : 0, all = env_first ? *dirty : 1, on = active ? *active : 1;
  if (!on) return;
  const size_t c0 = all ? 0 : (size_t)first * nb, c1 = all ? (size_t)ld : (size_t)(I + 1) * nb;
  constexpr int EPV = 16 / (int)sizeof(T);  // elements per 16-byte store
  using V16 = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  for (size_t c = c0 + (size_t)threadIdx.x * EPV; c < c1; c += (size_t)blockDim.x * EPV) {
    __align__(16) T z[EPV];
#pragma unroll
    for (int i = 0; i < EPV; i++) z[i] = r >= n && c + i == (size_t)r ? (T)1 : (T)0;
    *reinterpret_cast<V16*>(S + (size_t)r * ld + c) = *reinterpret_cast<const V16*>(z);
    if (S0) *reinterpret_cast<V16*>(S0 + (size_t)r * ld + c) = *reinterpret_cast<const V16*>(z);
  }
}

// ---------------------------------------------------------------------------
// Lanes == kBackLanes: eight lanes per point, lane l holds the 16-byte piece l of each
// of the point's W blocks, so a block is read as one run; FP64 sixteen lanes.  Bound
// by the latency of the index chain (point -> W block -> camera).
// Lanes == 1: a thread per point, its block in registers.  The lanes of a point repeat
// its index chain and add up at the end; where the points alone fill the chip and
// W is not far larger than L2, a thread each is the faster one (backsub_lanes).
// us, thread / lanes (9x3 blocks, W in MB): FP32 30k points, 23 MB 21 / 15; 50k, 42 MB
// 30 / 22; 100k, 34 MB 17 / 22; 150k, 59 MB 27 / 38; 150k, 117 MB 50 / 62; 270k, 212 MB
// 89 / 99; 500k, 392 MB 311 / 177.  FP64 50k, 84 MB 47 / 35; 75k, 117 MB 54 / 47; 100k,
// 67 MB 26 / 35; 150k, 117 MB 40 / 53; 150k, 235 MB 76 / 84; 270k, 424 MB 293 / 137.
template <typename T>
constexpr int kBackLanes = sizeof(T) == 4 ? 8 : 16;
// Lanes for np points and w_bytes of W.  FP32 is even at 75,000 points of 7 observations
// (34 / 33 us) and sooner with fewer, FP64 at about 100,000; between 235 and 392 MB of W
// the lanes begin to win.
template <typename T>
inline int backsub_lanes(int np, size_t w_bytes) {
  return np >= (sizeof(T) == 4 ? 1 << 16 : 3 << 15) && w_bytes <= ((size_t)256 << 20) ? 1 : kBackLanes<T>;
}
// Sixteen lanes keep to 32 registers, every warp of an SM resident: 200 cameras FP64 35 us
// against 41 with 36 registers.
template <typename T, int BC, int LANES>
static __global__ void __launch_bounds__(128, LANES == 16 ? 16 : 0)
    backsub_kernel(SchurDev d, const T* __restrict__ W, const T* __restrict__ Vinv, const T* __restrict__ bV,
                   double* xU, int nxu, double* __restrict__ xV, const int* __restrict__ ok_flag,
                   int* __restrict__ dirty, const int* __restrict__ active) {
  constexpr int LW = Layout<T, BC>::W;
  constexpr int LV = Layout<T, BC>::V;
  using V16 = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  constexpr int EPV = 16 / (int)sizeof(T), PW = LW / EPV, LP = LANES, NP = (PW + LP - 1) / LP;
  chain_start(W, Vinv, bV, ok_flag, active);
  if (active && !*active) return;
  const int l = threadIdx.x & (LP - 1);
  const bool failed = ok_flag && *ok_flag != 0;  // zero increment
  // last kernel of a call that formed S (dirty given): its clear has run; a failed
  // factorisation overflows, and 0 * inf is not zero outside the envelope (clear_kernel)
  if (dirty && blockIdx.x == 0 && threadIdx.x == 0) *dirty = failed ? 1 : 0;
  if (failed) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
    for (long long i = t; i < nxu; i += nt) xU[i] = 0.0;
    for (long long i = t; i < 3LL * d.np; i += nt) xV[i] = 0.0;
    return;
  }
  const int p = group_item(blockIdx.x, 128, threadIdx.x, LP);
  if constexpr (LANES == 1) {
    if (p >= d.np) return;
    double t[3];
#pragma unroll
    for (int k = 0; k < 3; k++) t[k] = -(double)bV[3 * (size_t)p + k];
    const int s1 = d.w_col_ptr[p + 1];
    for (int s = d.w_col_ptr[p]; s < s1; s++) {
      const int q = d.w_col_uid[s];
      const double* x = xU + (size_t)d.w_row[q] * BC;
      __align__(16) T w[LW];
#pragma unroll
      for (int i = 0; i < PW; i++)
        reinterpret_cast<V16*>(w)[i] = reinterpret_cast<const V16*>(W + (size_t)q * LW)[i];
#pragma unroll
      for (int i = 0; i < BC; i++)
#pragma unroll
        for (int k = 0; k < 3; k++) t[k] -= (double)w[3 * i + k] * x[i];
    }
    const T* v = Vinv + (size_t)p * LV;
#pragma unroll
    for (int k = 0; k < 3; k++)
      xV[3 * (size_t)p + k] = (double)v[3 * k] * t[0] + (double)v[3 * k + 1] * t[1] + (double)v[3 * k + 2] * t[2];
    return;
  }
  if (group_item(blockIdx.x, 128, threadIdx.x & ~31, LP) >= d.np) return;  // whole warps leave
  const bool valid = p < d.np;
  const int s0 = valid ? d.w_col_ptr[p] : 0, s1 = valid ? d.w_col_ptr[p + 1] : 0;
  // piece i of this lane: elements m0 = (l + LP i) EPV .., rows from m0 / 3 on; sum[i][r]
  // collects W' x at component (m0 + r) % 3
  double sum[NP][3] = {};
  int most = s1 - s0;  // of the warp's points
#pragma unroll
  for (int o = LP; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
  for (int base = 0; base < most; base += LP) {
    const int s = s0 + base + l;
    const int ql = s < s1 ? d.w_col_uid[s] : -1;
    const int cl = ql >= 0 ? d.w_row[ql] : 0;
    const int cnt = min(LP, most - base);
#pragma unroll 4
    for (int e = 0; e < cnt; e++) {
      const int q = __shfl_sync(0xffffffffu, ql, e, LP), c = __shfl_sync(0xffffffffu, cl, e, LP);
      if (q < 0) continue;
      const double* x = xU + (size_t)c * BC;
#pragma unroll
      for (int i = 0; i < NP; i++) {
        const int pc = l + LP * i;
        if (pc < PW) {
          __align__(16) T w[EPV];
          *reinterpret_cast<V16*>(w) = reinterpret_cast<const V16*>(W + (size_t)q * LW)[pc];
          const int m0 = pc * EPV, i0 = m0 / 3, k0 = m0 - 3 * i0;
          const double xa = i0 < BC ? x[i0] : 0.0, xb = i0 + 1 < BC ? x[i0 + 1] : 0.0;
#pragma unroll
          for (int j = 0; j < EPV; j++)
            if (m0 + j < 3 * BC) sum[i][j % 3] += (double)w[j] * (k0 + j < 3 ? xa : xb);
        }
      }
    }
  }
  double a[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 0; i < NP; i++) {
    const int k0 = (l + LP * i) * EPV % 3;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const int r = k >= k0 ? k - k0 : k - k0 + 3;
      a[k] += r == 0 ? sum[i][0] : r == 1 ? sum[i][1] : sum[i][2];
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
#pragma unroll
    for (int o = 1; o < LP; o <<= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
  }
  if (valid && l < 3) {
    const double t0 = -(double)bV[3 * (size_t)p] - a[0], t1 = -(double)bV[3 * (size_t)p + 1] - a[1],
                 t2 = -(double)bV[3 * (size_t)p + 2] - a[2];
    const T* v = Vinv + (size_t)p * LV + 3 * l;
    xV[3 * (size_t)p + l] = (double)v[0] * t0 + (double)v[1] * t1 + (double)v[2] * t2;
  }
}

}  // namespace nl
