// batch_lm.cu -- many independent small BA problems in one persistent launch.
//
// LevenbergMarquardt<SolverCholeskySchur>::solve
// (nelson/LevenbergMarquardt.hpp:36-146, nelson/SolverCholeskySchur.hpp:91-157)
// for n problems of uneven sizes at once: one kernel launch whose CTAs take
// problems from a device work queue (an atomic counter over the problems in
// descending order of estimated work) and run each problem's whole LM solve,
// sub-iteration by sub-iteration, with the CTA's threads:
//   update(true)     cost, then U / bU / W per camera (one warp per camera, its
//                    edges over the lanes, butterfly reduction) and V / bV per
//                    variable point (one thread per point over its edges);
//   computeIncrement damped V^-1 and xV0 = -V^-1 bV per point, Y = W V^-1 per
//                    edge row; bS = -bU - W xV0 per camera; S = U - sum Y W'
//                    block by block over (Y, W) edge pairs of a common point
//                    (one warp per block, points ascending, operands staged in
//                    shared memory), damping on the diagonal; Cholesky of S in
//                    32-column panels held in shared memory, with bS as one
//                    more row (which the factorisation turns into the forward
//                    solve's result); backward solve by 32-row blocks; back-
//                    substitution per edge, then per point;
//   the LM decisions (gain ratio, accept / reject, damping, termination) on
//                    one thread, exactly as the reference orders them.
// Everything is FP64.  No CTA ever waits for another, so nothing can hang;
// every loop is bounded by the problem sizes and the LM iteration limits.
// Edge blocks are read and written through shared memory by coalesced 16-byte
// copies: a lane per 144-byte block costs the L1 a line per lane and
// instruction, which bound every phase that touches W and Y.  128 problems of 8
// .. 64 cameras (200 .. 4,000 points), 6 iterations, as long as the largest one:
// 11.2 ms against 23.2 ms for 512 threads (27.5 ms for 256), of which per
// increment S 0.65 ms (0.80 before), Y, bS and V^-1 0.14 (0.73), Cholesky 0.28
// (0.86), solves 0.06 (0.15), back-substitution 0.11 (0.14) and the Jacobian pass
// 0.22 (0.42).  Another draw of 128 problems, 6 and 9 parameters: 24.9 -> 10.4 and
// 52.5 -> 20.1 ms (the 9-parameter kernel spills 1,756 bytes at its 128 registers).
// What bounds it now is the L1 again: the pairs' blocks are 2.3 KB
// of gathered lines per 8 pairs.
// Every sum has a fixed order that does not depend on the CTA size or on which
// CTA takes the problem (per-thread loops, warp butterflies, 32-element chunk
// sums added in order), so a problem's result does not depend on the launch
// shape or on the other problems of the batch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <numeric>
#include <vector>

#include "ba_kernels.cuh"
#include "problem_view.h"
#include "schur_core.cuh"

namespace nl {
namespace {

constexpr int kPW = 32;         // Cholesky / solve panel width
constexpr int kPLd = kPW + 4;   // shared panel row stride (doubles): conflict-free MMA operands
constexpr int kMaxN = 768;      // largest reduced camera system of the persistent path

// The CTA's dynamic shared memory (declared here, not passed: a pointer through
// a call that is not inlined would be read by generic loads): the Cholesky
// panel, or the warps' work areas.
extern __shared__ __align__(16) double smem[];

struct BProb {
  int ncv, nc_all, npv, np_all, ne, n, nS, pad;
  double f, cx, cy;
  const int* e_cam;     // E-order edges: camera slot (variable: user index; fixed: ncv + index)
  const int* e_pt;      // point slot (variable: index; fixed: npv + index)
  const double* e_obs;  // 2 per edge
  const double* e_w;
  const int* cam_ptr;   // ncv + 1: E-order edges of internal camera c
  const int* cam_slot;  // internal camera -> slot
  const int* slot2int;  // camera slot -> internal camera, -1 for a fixed camera
  const int* pt_ptr;    // npv + 1: P-order edges of point p
  const int* p2e;       // P-order -> E-order
  const int* s_i;       // S blocks (i <= j, internal cameras)
  const int* s_j;
  const int* s_ptr;     // nS + 1: pairs of block b
  const int* pa;        // pair: E-order edge of camera i
  const int* pb;        // pair: E-order edge of camera j, same point
  double* cam;          // nc_all x 16 camera state
  double* pt;           // np_all x 3
  double* cam_bck;
  double* pt_bck;
  double* W;            // ne x Layout::W (edges with a variable camera and a variable point)
  double* Y;            // same; after S is formed, W' xU per edge (4 doubles each)
  double* U;            // ncv x BC*BC (internal order)
  double* bU;           // ncv x BC
  double* V;            // npv x 9
  double* Vinv;         // npv x 10: upper triangle of (V + mu)^-1 (6), xV0 (3), pad
  double* bV;           // npv x 3
  double* S;            // (n + 1) x n: lower triangle, then bS as row n
  double* inc;          // n + 3 npv: internal camera order, then points
  double* part;         // chunk partials
};

struct BSettings {
  int maxNumIt, maxNumSubIt, minNumIt, pad;
  double epsBVector, epsIncSquare, epsChi2, tau, penaltyV, initV, maxScale, minScale;
};

struct BReport {
  int reason, iterations, subiterations, pad;
  double chi2, mu;
  unsigned long long t_start, t_end;  // %globaltimer (ns)
};

// One problem's camera states and points, in its handle and in the arena.
struct ParamCopy {
  double *h_cam, *h_pt, *a_cam, *a_pt;
  int nc, np;  // doubles
};

struct LmS {
  double mu, curV, oldChi2, chi2, chi2_new, rho, incSq, den, maxAbsB;
  int iter, subiter, nsub, done, reason, ok, apply, acc;
};

__device__ inline unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ inline double warp_all_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sum_{i < cnt} f(i) in an order fixed by cnt alone: 32-element chunks summed
// by a warp butterfly, chunk sums added by warp 0 in a fixed pattern.  Every
// thread gets the result.
template <class F>
__device__ double cta_sum(int cnt, F f, double* part, double* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int nch = (cnt + 31) / 32;
  for (int c = warp; c < nch; c += nw) {
    const int i = c * 32 + lane;
    const double v = warp_all_sum(i < cnt ? f(i) : 0.0);
    if (lane == 0) part[c] = v;
  }
  __syncthreads();
  if (warp == 0) {
    double v = 0.0;
    for (int c = lane; c < nch; c += 32) v += part[c];
    v = warp_all_sum(v);
    if (lane == 0) sh[0] = v;
  }
  __syncthreads();
  const double r = sh[0];
  __syncthreads();
  return r;
}

// max_{i < cnt} f(i) (exact in any order).
template <class F>
__device__ double cta_max(int cnt, F f, double* sh) {
  double m = 0.0;
  for (int i = threadIdx.x; i < cnt; i += blockDim.x) m = fmax(m, f(i));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) r = fmax(r, sh[w]);
    sh[32] = r;
  }
  __syncthreads();
  const double r = sh[32];
  __syncthreads();
  return r;
}

// Work area of one warp in shared memory: the stages of pair operands, or the
// blocks of up to 32 edges on their way in or out.
template <int BC>
struct BatchCfg {
  static constexpr int LW = Layout<double, BC>::W;
  static constexpr int TD = BC / 3, LP = TD * TD;        // 3 x 3 tiles of a block
  static constexpr int G = 32 / LP;                      // pairs side by side
  static constexpr int ROUNDS = G >= 8 ? 1 : 2, PBT = G * ROUNDS;  // pairs per stage
  static constexpr int kStages = 3;
  static constexpr int kWarpDoubles = kStages * 2 * PBT * LW;
  static_assert(32 * LW <= kWarpDoubles, "edge blocks of a warp fit");
};

// the 16 doubles of a camera state (128-byte aligned) by 16-byte loads
__device__ __forceinline__ void load_cam(const double* c, double (&s)[16]) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const double2 v = reinterpret_cast<const double2*>(c)[i];
    s[2 * i] = v.x;
    s[2 * i + 1] = v.y;
  }
}

template <int BC>
__device__ double cost(const BProb& P, double* sh) {
  return cta_sum(
      P.ne,
      [&](int e) {
        double r0, r1;
        ba_project<double, BC, false, false>(P.cam + (size_t)P.e_cam[e] * 16, P.pt + (size_t)P.e_pt[e] * 3,
                                             P.e_obs[2 * e], P.e_obs[2 * e + 1], P.f, P.cx, P.cy, r0, r1, nullptr,
                                             nullptr);
        return P.e_w[e] * (r0 * r0 + r1 * r1);
      },
      P.part, sh);
}

// update(true) without the cost: U, bU, W (cameras) and V, bV (points).
template <int BC>
__device__ void jacobian_pass(const BProb& P) {
  constexpr int LW = BatchCfg<BC>::LW;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  for (int p = tid; p < P.npv; p += nt) {
    double v[6] = {0, 0, 0, 0, 0, 0}, b[3] = {0, 0, 0};
    const double X[3] = {P.pt[3 * (size_t)p], P.pt[3 * (size_t)p + 1], P.pt[3 * (size_t)p + 2]};
    for (int t = P.pt_ptr[p]; t < P.pt_ptr[p + 1]; t++) {
      const int e = P.p2e[t];
      double cs[16], r0, r1, Jp[6];
      load_cam(P.cam + (size_t)P.e_cam[e] * 16, cs);
      const double2 z = reinterpret_cast<const double2*>(P.e_obs)[e];
      ba_project<double, BC, false, true>(cs, X, z.x, z.y, P.f, P.cx, P.cy, r0, r1, nullptr, Jp);
      const double w = P.e_w[e];
      int q = 0;
#pragma unroll
      for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int j = i; j < 3; j++) v[q++] += w * (Jp[i] * Jp[j] + Jp[3 + i] * Jp[3 + j]);
        b[i] += w * (Jp[i] * r0 + Jp[3 + i] * r1);
      }
    }
    double* Vp = P.V + (size_t)p * 9;
    Vp[0] = v[0]; Vp[1] = v[1]; Vp[2] = v[2];
    Vp[3] = v[1]; Vp[4] = v[3]; Vp[5] = v[4];
    Vp[6] = v[2]; Vp[7] = v[4]; Vp[8] = v[5];
    P.bV[3 * (size_t)p] = b[0];
    P.bV[3 * (size_t)p + 1] = b[1];
    P.bV[3 * (size_t)p + 2] = b[2];
  }
  constexpr int NUU = BC * (BC + 1) / 2;
  double* const stage = smem + (size_t)warp * BatchCfg<BC>::kWarpDoubles;
  for (int c = warp; c < P.ncv; c += nw) {
    const double* cs = P.cam + (size_t)P.cam_slot[c] * 16;
    double u[NUU], b[BC];
#pragma unroll
    for (int i = 0; i < NUU; i++) u[i] = 0.0;
#pragma unroll
    for (int i = 0; i < BC; i++) b[i] = 0.0;
    const int e1 = P.cam_ptr[c + 1];
    for (int eb = P.cam_ptr[c]; eb < e1; eb += 32) {
      const int e = eb + lane;
      double Jc[2 * BC], Jp[6], w = 0.0;
      if (e < e1) {
        double r0, r1;
        const double2 z = reinterpret_cast<const double2*>(P.e_obs)[e];
        ba_project<double, BC, true, true>(cs, P.pt + (size_t)P.e_pt[e] * 3, z.x, z.y, P.f, P.cx, P.cy, r0, r1, Jc, Jp);
        w = P.e_w[e];
        int q = 0;
#pragma unroll
        for (int i = 0; i < BC; i++) {
#pragma unroll
          for (int j = i; j < BC; j++) u[q++] += w * (Jc[i] * Jc[j] + Jc[BC + i] * Jc[BC + j]);
          b[i] += w * (Jc[i] * r0 + Jc[BC + i] * r1);
        }
      }
      // W of the 32 edges (consecutive in memory) through shared memory
      if (e < e1) {
        double* We = stage + lane * LW;
#pragma unroll
        for (int i = 0; i < BC; i++)
#pragma unroll
          for (int j = 0; j < 3; j++) We[i * 3 + j] = w * (Jc[i] * Jp[j] + Jc[BC + i] * Jp[3 + j]);
      }
      __syncwarp();
      const int nv = min(32, e1 - eb) * LW / 2;
      double2* out = reinterpret_cast<double2*>(P.W + (size_t)eb * LW);
      for (int i = lane; i < nv; i += 32) out[i] = reinterpret_cast<const double2*>(stage)[i];
      __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < NUU; i++) u[i] = warp_all_sum(u[i]);
#pragma unroll
    for (int i = 0; i < BC; i++) b[i] = warp_all_sum(b[i]);
    if (lane == 0) {
      double* Uc = P.U + (size_t)c * BC * BC;
      int q = 0;
#pragma unroll
      for (int i = 0; i < BC; i++)
#pragma unroll
        for (int j = i; j < BC; j++) {
          Uc[i * BC + j] = u[q];
          Uc[j * BC + i] = u[q];
          q++;
        }
#pragma unroll
      for (int i = 0; i < BC; i++) P.bU[(size_t)c * BC + i] = b[i];
    }
  }
}

// (V_p + mu I)^-1 by Cholesky; false if not positive definite.
__device__ inline bool spd3_inverse(const double* A, double mu, double* X) {
  const double a00 = A[0] + mu, a10 = A[3], a11 = A[4] + mu, a20 = A[6], a21 = A[7], a22 = A[8] + mu;
  if (!(a00 > 0.0)) return false;
  const double l00 = sqrt(a00);
  const double l10 = a10 / l00, l20 = a20 / l00;
  const double d1 = a11 - l10 * l10;
  if (!(d1 > 0.0)) return false;
  const double l11 = sqrt(d1);
  const double l21 = (a21 - l20 * l10) / l11;
  const double d2 = a22 - l20 * l20 - l21 * l21;
  if (!(d2 > 0.0) || !isfinite(d2)) return false;
  const double l22 = sqrt(d2);
  // inv(L)
  const double i00 = 1.0 / l00, i11 = 1.0 / l11, i22 = 1.0 / l22;
  const double i10 = -l10 * i00 * i11;
  const double i21 = -l21 * i11 * i22;
  const double i20 = -(l20 * i00 + l21 * i10) * i22;
  // X = inv(L)' inv(L)
  X[0] = i00 * i00 + i10 * i10 + i20 * i20;
  X[1] = i10 * i11 + i20 * i21;
  X[2] = i20 * i22;
  X[4] = i11 * i11 + i21 * i21;
  X[5] = i21 * i22;
  X[8] = i22 * i22;
  X[3] = X[1];
  X[6] = X[2];
  X[7] = X[5];
  return true;
}

// One block of S (i <= j) by one warp: M = U_ij - sum_pairs Y_a W_b' (mu on the
// diagonal of diagonal blocks), written to the lower triangle.  Operands come
// through kStages stages of 16-byte asynchronous copies; a lane owns a 3 x 3 tile
// of one of G pairs side by side.
template <int BC>
__device__ void schur_block(const BProb& P, int b, double mu, int warp, int lane) {
  using Cfg = BatchCfg<BC>;
  constexpr int LW = Cfg::LW, LP = Cfg::LP, TD = Cfg::TD, G = Cfg::G, PBT = Cfg::PBT, VB = LW / 2,
                kStages = Cfg::kStages;
  double* const stage = smem + (size_t)warp * Cfg::kWarpDoubles;
  const uint32_t sa = (uint32_t)__cvta_generic_to_shared(stage);
  const int t0 = P.s_ptr[b], cnt = P.s_ptr[b + 1] - t0, nbatch = (cnt + PBT - 1) / PBT;
  const int q = lane / LP, tile = lane % LP, r0 = 3 * (tile / TD), c0 = 3 * (tile % TD);
  int ua = 0, ub = 0;
  auto load_ids = [&](int t) {
    if (lane < PBT && t * PBT + lane < cnt) {
      ua = P.pa[t0 + t * PBT + lane];
      ub = P.pb[t0 + t * PBT + lane];
    }
  };
  auto copy_batch = [&](int t) {
    const int n = min(PBT, cnt - t * PBT);
    const uint32_t dst = sa + (uint32_t)((t % kStages) * 2 * PBT * LW * 8);
#pragma unroll
    for (int v0 = 0; v0 < 2 * PBT * VB; v0 += 32) {
      const int v = v0 + lane, blk = v / VB, part = v - blk * VB, pair = blk < PBT ? blk : blk - PBT;
      const int y = __shfl_sync(0xffffffffu, ua, pair & 31), w = __shfl_sync(0xffffffffu, ub, pair & 31);
      if (blk < 2 * PBT && pair < n)
        cp_async16(dst + 16u * (uint32_t)v, (blk < PBT ? P.Y + (size_t)y * LW : P.W + (size_t)w * LW) + 2 * part);
    }
  };
  double acc[3][3] = {};
  load_ids(0);
#pragma unroll
  for (int t = 0; t < kStages - 1; t++) {
    if (t < nbatch) {
      copy_batch(t);
      load_ids(t + 1);
    }
    cp_async_commit();
  }
  for (int t = 0; t < nbatch; t++) {
    if (t + kStages - 1 < nbatch) {
      copy_batch(t + kStages - 1);
      load_ids(t + kStages);
    }
    cp_async_commit();
    cp_async_wait<kStages - 1>();
    __syncwarp();
    const double* st = stage + (t % kStages) * 2 * PBT * LW;
#pragma unroll
    for (int r = 0; r < Cfg::ROUNDS; r++) {
      const int pair = r * G + q;
      if (q < G && t * PBT + pair < cnt) {
        const double* y = st + pair * LW + 3 * r0;
        const double* w = st + (PBT + pair) * LW + 3 * c0;
        double yv[3][3], wv[3][3];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int m = 0; m < 3; m++) {
            yv[i][m] = y[3 * i + m];
            wv[i][m] = w[3 * i + m];
          }
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int j = 0; j < 3; j++)
#pragma unroll
            for (int m = 0; m < 3; m++) acc[i][j] += yv[i][m] * wv[j][m];
      }
    }
    __syncwarp();
  }
  if (G == 3) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const double x = __shfl_down_sync(0xffffffffu, acc[i][j], LP), z = __shfl_down_sync(0xffffffffu, acc[i][j], 2 * LP);
        acc[i][j] += x + z;
      }
  } else {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) acc[i][j] += __shfl_down_sync(0xffffffffu, acc[i][j], o * LP);
  }
  if (lane < LP) {
    const int bi = P.s_i[b], bj = P.s_j[b], n = P.n;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        double m = -acc[i][j];
        if (bi == bj) {
          m += P.U[(size_t)bi * BC * BC + (r0 + i) * BC + c0 + j];
          if (r0 + i == c0 + j) m += mu;
        }
        // block (i, j) of the upper S at lower (j BC + c, i BC + r)
        const int row = bj * BC + c0 + j, col = bi * BC + r0 + i;
        if (col <= row) P.S[(size_t)row * n + col] = m;
      }
  }
}

// 16 rows x 16 columns of the panel's product by one warp: acc = rows rr .. of
// the panel times rows cc .. of it, over columns [k0, k1); rows past `last` are
// read from row `last` (their results are not used).  Lane 4 g + t holds rows
// rr + g + 8 i, columns cc + 8 j + 2 t (+ 1).
__device__ __forceinline__ void panel_mma(Sh<double> sp, int rr, int cc, int last, int k0, int k1, int lane,
                                          double (&acc)[2][2][2]) {
  const int g = lane >> 2, t = lane & 3;
  Sh<double> pa[2], pb[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    pa[i] = sp + (min(rr + 8 * i + g, last) * kPLd + t);
    pb[i] = sp + (min(cc + 8 * i + g, last) * kPLd + t);
  }
#pragma unroll 4
  for (int k = k0; k < k1; k += 4) {
    const double a0 = load_one(pa[0] + k), a1 = load_one(pa[1] + k), b0 = load_one(pb[0] + k), b1 = load_one(pb[1] + k);
    mma_f64(acc[0][0], a0, b0);
    mma_f64(acc[0][1], a0, b1);
    mma_f64(acc[1][0], a1, b0);
    mma_f64(acc[1][1], a1, b1);
  }
}

// Cholesky of S with the row n (bS) carried along, which ends as the solution
// y of L y = bS.  A panel of 32 columns (identity on the columns past n) and all
// its rows stay in shared memory; the row bS is panel row 32 of the last panel
// and the last row of the others.  Per 16 columns: one warp factors the diagonal
// block, every thread solves rows below it.
__device__ void factor(const BProb& P, double* ucs, int* flag) {
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int n = P.n;
  const Sh<double> sp{(uint32_t)__cvta_generic_to_shared(smem)}, uc{(uint32_t)__cvta_generic_to_shared(ucs)};
  const Sh<double> inv_s = uc + PB * PB;
  for (int k0 = 0; k0 < n; k0 += kPW) {
    const int kb = min(kPW, n - k0), m = max(n - k0, kPW) + 1;
    for (int i = tid; i < m * kPW; i += nt) {
      const int r = i / kPW, c = i % kPW;
      const int row = r == m - 1 ? n : k0 + r;
      double v = r == c ? 1.0 : 0.0;
      if (c < kb && row <= n && (row < n || r == m - 1)) v = c <= r ? P.S[(size_t)row * n + k0 + c] : 0.0;
      smem[r * kPLd + c] = v;
    }
    __syncthreads();
#pragma unroll 1
    for (int sb = 0; sb < 2; sb++) {
      if (warp == 0) {
        const Sh<double> row = sp + ((sb * PB + (lane & (PB - 1))) * kPLd + sb * PB);
        double a[PB];
        load_row16(row, a);
        if (!pivot_block<double, false>(a, uc, inv_s, lane) && lane == 0) *flag = 1;
        if (lane < PB) {
#pragma unroll
          for (int c = 0; c < PB; c++)
            if (c > lane) a[c] = 0.0;
          store_row16(row, a);
        }
      }
      __syncthreads();
      for (int r = (sb + 1) * PB + tid; r < m; r += nt) {
        const Sh<double> row = sp + (r * kPLd + sb * PB);
        double a[PB];
        load_row16(row, a);
        follow_block<double, false>(a, uc, inv_s);
        store_row16(row, a);
      }
      __syncthreads();
      if (sb == 0) {
        for (int u = warp; u * 16 < m - PB; u += nw) {
          double acc[2][2][2] = {};
          panel_mma(sp, PB + 16 * u, PB, m - 1, 0, PB, lane, acc);
#pragma unroll
          for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
              const int r = PB + 16 * u + 8 * i + (lane >> 2);
              if (r >= m) continue;
              const Sh<double> c = sp + (r * kPLd + PB + 8 * j + 2 * (lane & 3));
              double x, y;
              load_two(c, x, y);
              store_two(c, x - acc[i][j][0], y - acc[i][j][1]);
            }
        }
        __syncthreads();
      }
    }
    for (int i = tid; i < m * kPW; i += nt) {
      const int r = i / kPW, c = i % kPW;
      const int row = r == m - 1 ? n : k0 + r;
      if (c < kb && (r == m - 1 || (row < n && c <= r))) P.S[(size_t)row * n + k0 + c] = smem[r * kPLd + c];
    }
    // trailing rows 32 .. m - 1 (bS last) and columns 32 .. n - k0 - 1, 16 x 16 tiles
    const int nc = n - k0 - kPW;
    if (nc > 0) {
      const int T = (m - kPW + 15) / 16, ntile = T * (T + 1) / 2;
      for (int q = warp; q < ntile; q += nw) {
        int I = (int)((sqrtf(8.0f * q + 1.0f) - 1.0f) * 0.5f);
        while ((I + 1) * (I + 2) / 2 <= q) I++;
        while (I * (I + 1) / 2 > q) I--;
        const int J = q - I * (I + 1) / 2;
        if (16 * J >= nc) continue;
        double c[2][2][2];
        auto at = [&](int i, int j, int h, bool& in) {
          const int r = 16 * I + 8 * i + (lane >> 2), cc = 16 * J + 8 * j + 2 * (lane & 3) + h;
          in = r < m - kPW && cc < nc && cc <= r;
          return P.S + (size_t)(k0 + kPW + r) * n + k0 + kPW + cc;
        };
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int j = 0; j < 2; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
              bool in;
              const double* s = at(i, j, h, in);
              c[i][j][h] = in ? *s : 0.0;
            }
        double acc[2][2][2] = {};
        panel_mma(sp, kPW + 16 * I, kPW + 16 * J, m - 1, 0, kPW, lane, acc);
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int j = 0; j < 2; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
              bool in;
              double* s = at(i, j, h, in);
              if (in) *s = c[i][j][h] - acc[i][j][h];
            }
      }
    }
    __syncthreads();
  }
}

// computeIncrement(H, b, 0, mu): inc = [xU; xV].  Returns false when a damped
// point block or S is not positive definite (the increment is then zero).
template <int BC>
__device__ bool compute_increment(const BProb& P, double mu, double* ucs, int* flag) {
  constexpr int LW = BatchCfg<BC>::LW;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int n = P.n;
  double* const stage = smem + (size_t)warp * BatchCfg<BC>::kWarpDoubles;
  const uint32_t stage_a = (uint32_t)__cvta_generic_to_shared(stage);
  if (tid == 0) *flag = 0;
  __syncthreads();
  // V^-1 and xV0 per point
  for (int p = tid; p < P.npv; p += nt) {
    double Vi[9];
    if (!spd3_inverse(P.V + (size_t)p * 9, mu, Vi)) {
      *flag = 1;
      for (int i = 0; i < 9; i++) Vi[i] = 0.0;
    }
    const double* b = P.bV + (size_t)p * 3;
    double x[3];
#pragma unroll
    for (int i = 0; i < 3; i++) x[i] = -(Vi[i * 3] * b[0] + Vi[i * 3 + 1] * b[1] + Vi[i * 3 + 2] * b[2]);
    double2* o = reinterpret_cast<double2*>(P.Vinv + (size_t)p * 10);
    o[0] = make_double2(Vi[0], Vi[1]);
    o[1] = make_double2(Vi[2], Vi[4]);
    o[2] = make_double2(Vi[5], Vi[8]);
    o[3] = make_double2(x[0], x[1]);
    o[4] = make_double2(x[2], 0.0);
  }
  // the lower triangle of S starts from zero
  for (size_t i = tid; i < (size_t)n * n; i += nt) P.S[i] = 0.0;
  __syncthreads();
  // Y = W V^-1 per edge and bS = -bU - W xV0 per camera: one warp per camera, a
  // lane per edge, the blocks in and out through shared memory
  for (int c = warp; c < P.ncv; c += nw) {
    double s[BC];
#pragma unroll
    for (int i = 0; i < BC; i++) s[i] = 0.0;
    const int e1 = P.cam_ptr[c + 1];
    for (int eb = P.cam_ptr[c]; eb < e1; eb += 32) {
      const int nv = min(32, e1 - eb) * LW / 2, e = eb + lane;
      for (int i = lane; i < nv; i += 32) cp_async16(stage_a + 16u * (uint32_t)i, P.W + (size_t)eb * LW + 2 * i);
      cp_async_commit();
      double2 v[5];
      const int ps = e < e1 ? P.e_pt[e] : P.npv;
      const bool in = ps < P.npv;
      if (in) {
        const double2* r = reinterpret_cast<const double2*>(P.Vinv + (size_t)ps * 10);
#pragma unroll
        for (int i = 0; i < 5; i++) v[i] = r[i];
      }
      cp_async_wait<0>();
      __syncwarp();
      if (in) {
        double* b = stage + lane * LW;
#pragma unroll
        for (int i = 0; i < BC; i++) {
          const double w0 = b[3 * i], w1 = b[3 * i + 1], w2 = b[3 * i + 2];
          b[3 * i] = w0 * v[0].x + w1 * v[0].y + w2 * v[1].x;
          b[3 * i + 1] = w0 * v[0].y + w1 * v[1].y + w2 * v[2].x;
          b[3 * i + 2] = w0 * v[1].x + w1 * v[2].x + w2 * v[2].y;
          s[i] += w0 * v[3].x + w1 * v[3].y + w2 * v[4].x;
        }
      }
      __syncwarp();
      double2* out = reinterpret_cast<double2*>(P.Y + (size_t)eb * LW);
      for (int i = lane; i < nv; i += 32) out[i] = reinterpret_cast<const double2*>(stage)[i];
      __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < BC; i++) s[i] = warp_all_sum(s[i]);
    if (lane == 0)
#pragma unroll
      for (int i = 0; i < BC; i++)
        P.S[(size_t)n * n + (size_t)c * BC + i] = -P.bU[(size_t)c * BC + i] - s[i];
  }
  __syncthreads();
  for (int b = warp; b < P.nS; b += nw)
    schur_block<BC>(P, b, mu, warp, lane);
  __syncthreads();
  factor(P, ucs, flag);
  // backward solve L' x = y
  double* x = P.inc;
  for (int i = tid; i < n; i += nt) x[i] = P.S[(size_t)n * n + i];
  __syncthreads();
  for (int k0 = ((n - 1) / kPW) * kPW; k0 >= 0 && n > 0; k0 -= kPW) {
    const int kb = min(kPW, n - k0);
    if (warp == 0) {
      // lane i holds column k0 + i of the diagonal block: L[k0 + j][k0 + i], j >= i
      double lcol[kPW];
#pragma unroll
      for (int j = 0; j < kPW; j++)
        lcol[j] = (lane < kb && j < kb && j >= lane) ? P.S[(size_t)(k0 + j) * n + k0 + lane] : 0.0;
      double yi = lane < kb ? x[k0 + lane] : 0.0;
      const double ri = lane < kb ? 1.0 / P.S[(size_t)(k0 + lane) * n + k0 + lane] : 0.0;
#pragma unroll
      for (int j = kPW - 1; j >= 0; j--) {
        if (j < kb) {
          const double xj = __shfl_sync(0xffffffffu, yi * ri, j);
          if (lane == j) yi = xj;
          if (lane < j) yi -= lcol[j] * xj;
        }
      }
      if (lane < kb) x[k0 + lane] = yi;
    }
    __syncthreads();
    for (int r = tid; r < k0; r += nt) {
      double s = x[r];
#pragma unroll 8
      for (int j = 0; j < kb; j++) s -= P.S[(size_t)(k0 + j) * n + r] * x[k0 + j];
      x[r] = s;
    }
    __syncthreads();
  }
  // back-substitution: W' xU per edge (into Y, 4 doubles an edge; a lane per
  // edge, blocks through shared memory), then xV = V^-1 (-bV - sum W' xU) per point
  {
    const int ne = P.cam_ptr[P.ncv];
    for (int eb = 32 * warp; eb < ne; eb += 32 * nw) {
      const int nv = min(32, ne - eb) * LW / 2, e = eb + lane;
      for (int i = lane; i < nv; i += 32) cp_async16(stage_a + 16u * (uint32_t)i, P.W + (size_t)eb * LW + 2 * i);
      cp_async_commit();
      double xu[BC];
      if (e < ne) {
        const double* xc = x + (size_t)P.slot2int[P.e_cam[e]] * BC;
#pragma unroll
        for (int i = 0; i < BC; i++) xu[i] = xc[i];
      }
      cp_async_wait<0>();
      __syncwarp();
      if (e < ne) {
        double t[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < BC; i++)
#pragma unroll
          for (int j = 0; j < 3; j++) t[j] += stage[lane * LW + 3 * i + j] * xu[i];
        double2* o = reinterpret_cast<double2*>(P.Y + (size_t)e * 4);
        o[0] = make_double2(t[0], t[1]);
        o[1] = make_double2(t[2], 0.0);
      }
      __syncwarp();
    }
  }
  __syncthreads();
  for (int p = tid; p < P.npv; p += nt) {
    double t[3] = {-P.bV[3 * (size_t)p], -P.bV[3 * (size_t)p + 1], -P.bV[3 * (size_t)p + 2]};
    const int nev = P.cam_ptr[P.ncv];  // edges of variable cameras come first
    for (int q = P.pt_ptr[p]; q < P.pt_ptr[p + 1]; q++) {
      const int e = P.p2e[q];
      if (e >= nev) continue;
      const double2* te = reinterpret_cast<const double2*>(P.Y + (size_t)e * 4);
      const double2 a = te[0], b = te[1];
      t[0] -= a.x;
      t[1] -= a.y;
      t[2] -= b.x;
    }
    const double* v = P.Vinv + (size_t)p * 10;
    x[n + 3 * (size_t)p] = v[0] * t[0] + v[1] * t[1] + v[2] * t[2];
    x[n + 3 * (size_t)p + 1] = v[1] * t[0] + v[3] * t[1] + v[4] * t[2];
    x[n + 3 * (size_t)p + 2] = v[2] * t[0] + v[4] * t[1] + v[5] * t[2];
  }
  __syncthreads();
  const bool ok = *flag == 0;
  if (!ok)  // SolverCholeskySchur.hpp:151-154
    for (int i = tid; i < n + 3 * P.npv; i += nt) x[i] = 0.0;
  __syncthreads();
  return ok;
}

template <int BC>
__device__ void oplus(const BProb& P) {
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int c = tid; c < P.ncv; c += nt) {
    double* s = P.cam + (size_t)P.cam_slot[c] * 16;
    const double* d = P.inc + (size_t)c * BC;
    double dR[9], R[9];
    so3_exp(d, dR);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) R[i * 3 + j] = dR[i * 3] * s[j] + dR[i * 3 + 1] * s[3 + j] + dR[i * 3 + 2] * s[6 + j];
#pragma unroll
    for (int i = 0; i < 9; i++) s[i] = R[i];
#pragma unroll
    for (int i = 0; i < 3; i++) s[9 + i] += d[3 + i];
    if (BC == 9)
#pragma unroll
      for (int i = 0; i < 3; i++) s[12 + i] += d[6 + i];
  }
  for (int i = tid; i < 3 * P.npv; i += nt) P.pt[i] += P.inc[P.n + i];
}

__device__ inline void copy_params(const BProb& P, bool to_backup) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const size_t nc = (size_t)P.nc_all * 16, np = (size_t)P.np_all * 3;
  double* cd = to_backup ? P.cam_bck : P.cam;
  const double* cs = to_backup ? P.cam : P.cam_bck;
  double* pd = to_backup ? P.pt_bck : P.pt;
  const double* ps = to_backup ? P.pt : P.pt_bck;
  for (size_t i = tid; i < nc; i += nt) cd[i] = cs[i];
  for (size_t i = tid; i < np; i += nt) pd[i] = ps[i];
}

template <int BC>
__device__ double max_abs_b(const BProb& P, double* sh) {
  const int nb = P.n, nv = 3 * P.npv;
  return cta_max(nb + nv, [&](int i) { return fabs(i < nb ? P.bU[i] : P.bV[i - nb]); }, sh);
}

template <int BC>
__device__ double max_abs_hdiag(const BProb& P, double* sh) {
  const int nb = P.n, nv = 3 * P.npv;
  return cta_max(
      nb + nv,
      [&](int i) {
        return fabs(i < nb ? P.U[(size_t)(i / BC) * BC * BC + (i % BC) * (BC + 1)] : P.V[(size_t)((i - nb) / 3) * 9 + ((i - nb) % 3) * 4]);
      },
      sh);
}

// The LM solve of one problem (nelson/LevenbergMarquardt.hpp:36-146; the
// decisions on thread 0, as lm_kernels.cuh orders them).
template <int BC>
__device__ void solve_problem(const BProb& P, const BSettings& s, BReport* rep, double* ucs, LmS& st,
                              double* sh, int* flag) {
  const int tid = threadIdx.x;
  if (tid == 0) rep->t_start = global_ns();
  double c0 = cost<BC>(P, sh);
  jacobian_pass<BC>(P);
  __syncthreads();
  const double mb = max_abs_b<BC>(P, sh);
  if (tid == 0) {
    st.chi2 = st.oldChi2 = c0;
    st.maxAbsB = mb;
    st.done = 0;
    st.iter = -1;
    st.subiter = 0;
    st.nsub = 0;
    st.mu = 0.0;
    if (mb <= s.epsBVector) {
      st.done = 1;
      st.reason = NL_SUCCESS_AT_START;
    }
  }
  __syncthreads();
  if (!st.done) {
    copy_params(P, true);
    const double hd = max_abs_hdiag<BC>(P, sh);
    if (tid == 0) {
      st.mu = s.tau * hd;  // LevenbergMarquardt.hpp:58
      st.curV = s.initV;
      st.iter = 0;
      if (s.maxNumIt <= 0) {
        st.done = 1;
        st.reason = NL_MAX_ITERATION_REACHED;
      }
    }
    __syncthreads();
  }
  while (!st.done) {
    const bool ok = compute_increment<BC>(P, st.mu, ucs, flag);
    const double mu = st.mu;
    const int nn = P.n + 3 * P.npv;
    const double a = cta_sum(nn, [&](int i) { return P.inc[i] * P.inc[i]; }, P.part, sh);
    const double den = cta_sum(
        nn,
        [&](int i) {
          const double x = P.inc[i], g = i < P.n ? P.bU[i] : P.bV[i - P.n];
          return x * (mu * x - g);
        },
        P.part, sh);
    if (tid == 0) {
      st.ok = ok && isfinite(a);
      st.incSq = st.ok ? a : 0.0;
      st.den = den;
      st.apply = 0;
      if (st.ok && st.iter >= s.minNumIt && st.incSq <= s.epsIncSquare) {  // LevenbergMarquardt.hpp:73-75
        st.done = 1;
        st.reason = NL_SUCCESS_SMALL_INCREMENT;
      } else {
        st.apply = st.ok;
      }
    }
    __syncthreads();
    if (st.done) break;
    double cn = 0.0;
    if (st.apply) {
      oplus<BC>(P);
      __syncthreads();
      cn = cost<BC>(P, sh);
    }
    if (tid == 0) {
      // LevenbergMarquardt.hpp:78-129
      double rho = -1.0;
      if (st.apply) {
        st.chi2_new = cn;
        rho = (st.oldChi2 - cn) / st.den;
      }
      st.rho = rho;
      st.acc = st.apply && rho > 0.0;
      st.nsub++;
      if (st.acc) {
        st.chi2 = cn;
        if (st.iter > s.minNumIt && st.maxAbsB <= s.epsBVector) {
          st.done = 1;
          st.reason = NL_SUCCESS_EPS_B;
        } else if (st.iter > s.minNumIt && cn < s.epsChi2) {
          st.done = 1;
          st.reason = NL_SUCCESS_SMALL_RESIDUALS;
        } else {
          const double fc = 2.0 * rho - 1.0;
          double alpha = fmin(s.maxScale, 1.0 - fc * fc * fc);
          alpha = fmax(s.minScale, alpha);
          st.mu = st.mu * alpha;
          st.curV = s.initV;
        }
      } else {
        st.mu = st.mu * st.curV;
        st.curV = st.curV * s.penaltyV;
      }
      if (!st.done) {
        st.subiter++;
        if (st.subiter >= s.maxNumSubIt) {
          st.done = 1;
          st.reason = NL_MAX_SUBITERATION_REACHED;
        }
      }
    }
    __syncthreads();
    if (!st.acc) {
      copy_params(P, false);  // rollbackSolution
      __syncthreads();
    }
    if (st.done) break;
    if (st.acc) {
      // update(true) at the accepted point (its cost is cn), backupSolution
      jacobian_pass<BC>(P);
      __syncthreads();
      const double mb2 = max_abs_b<BC>(P, sh);
      copy_params(P, true);
      if (tid == 0) {
        st.chi2 = cn;
        st.oldChi2 = cn;
        st.maxAbsB = mb2;
        st.iter++;
        st.subiter = 0;
        if (st.iter >= s.maxNumIt) {
          st.done = 1;
          st.reason = NL_MAX_ITERATION_REACHED;
        }
      }
      __syncthreads();
    }
  }
  __syncthreads();
  if (tid == 0) {
    rep->reason = st.reason;
    rep->iterations = st.iter;
    rep->subiterations = st.nsub;
    rep->chi2 = st.chi2;
    rep->mu = st.mu;
    rep->t_end = global_ns();
  }
  __syncthreads();
}

// One instantiation for every launch shape (up to 512 threads): the same
// machine code gives the same bits.
template <int BC>
__global__ void __launch_bounds__(512) batch_lm_kernel(const BProb* __restrict__ probs, const int* __restrict__ order,
                                                      int nprob, int* __restrict__ queue, BSettings s,
                                                      BReport* __restrict__ reps) {
  __shared__ BProb Ps;
  __shared__ LmS st;
  __shared__ double sh[40];
  __shared__ __align__(16) double ucs[PB * PB + 2 * PB];
  __shared__ int q_s, flag;
  for (;;) {
    if (threadIdx.x == 0) q_s = atomicAdd(queue, 1);
    __syncthreads();
    const int q = q_s;
    if (q >= nprob) return;
    const int pi = order[q];
    if (threadIdx.x == 0) Ps = probs[pi];
    __syncthreads();
    solve_problem<BC>(Ps, s, reps + pi, ucs, st, sh, &flag);
    __syncthreads();
  }
}

using BatchKernel = void (*)(const BProb*, const int*, int, int*, BSettings, BReport*);

}  // namespace
}  // namespace nl

// ===========================================================================
// Host side.
struct nl_batch {
  int n = 0, bc = 0, device = 0, max_n = 0;
  std::vector<nl_problem*> hs;
  nl::DevBuf arena, probs, order, queue, reps, params;
  std::vector<nl::BProb> hp;            // host copies of the descriptors
  std::vector<size_t> off_cam, off_pt;  // state offsets in the arena (doubles)
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int tuned_nt = 0, tuned_cps = 0;  // autotuner's choice (0: not tuned)
  float tune_ms[6] = {0, 0, 0, 0, 0, 0};
  ~nl_batch() {
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (st) cudaStreamDestroy(st);
  }
};

extern "C" {

nl_status nl_batch_create(nl_problem** hs, int n, nl_batch** out) {
  using namespace nl;
  if (!hs || n <= 0 || !out) return NL_ERR_ARG;
  *out = nullptr;
  std::unique_ptr<nl_batch> b(new nl_batch());
  b->n = n;
  b->hs.assign(hs, hs + n);
  std::vector<nl_problem_view> vs(n);
  for (int i = 0; i < n; i++) {
    if (!hs[i]) return NL_ERR_ARG;
    for (int j = 0; j < i; j++)
      if (hs[j] == hs[i]) return NL_ERR_ARG;
    nl_status s = nl_problem_get_view(hs[i], &vs[i]);
    if (s != NL_OK) return s;
    if (!vs[i].ready) return NL_ERR_STATE;
    if (vs[i].bc != vs[0].bc) return NL_ERR_UNSUPPORTED;
    if ((long long)vs[i].ncv * vs[i].bc > kMaxN) return NL_ERR_UNSUPPORTED;
  }
  b->bc = vs[0].bc;
  const int bc = b->bc;
  int dev = 0;
  NL_CUDA(cudaGetDevice(&dev));
  b->device = dev;
  NL_CUDA(cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking));
  NL_CUDA(cudaEventCreate(&b->e0));
  NL_CUDA(cudaEventCreate(&b->e1));
  // ---- host structure of every problem, then one arena for all of it ----
  struct HostProb {
    std::vector<int> e_cam, e_pt, cam_ptr, cam_slot, slot2int, pt_ptr, p2e, s_i, s_j, s_ptr, pa, pb;
    std::vector<double> e_obs, e_w;
  };
  std::vector<HostProb> H(n);
  std::vector<double> work(n, 0.0);
  size_t total = 0;  // bytes
  auto al = [](size_t x) { return (x + 255) / 256 * 256; };
  std::vector<std::vector<size_t>> offs(n);
  for (int i = 0; i < n; i++) {
    const nl_problem_view& v = vs[i];
    HostProb& h = H[i];
    const int ne = (int)v.e_cam->size(), ncv = v.ncv, npv = v.npv;
    const std::vector<int>& eo = *v.eorder;
    std::vector<int> epos(ne);
    for (int t = 0; t < ne; t++) epos[eo[t]] = t;
    h.e_cam.resize(ne);
    h.e_pt.resize(ne);
    h.e_obs.resize(2 * (size_t)ne);
    h.e_w.resize(ne);
    h.cam_ptr.assign(ncv + 1, 0);
    for (int t = 0; t < ne; t++) {
      const int e = eo[t];
      const bool cf = (*v.e_camfix)[e] != 0, pf = (*v.e_ptfix)[e] != 0;
      h.e_cam[t] = cf ? ncv + (*v.e_cam)[e] : (*v.e_cam)[e];
      h.e_pt[t] = pf ? npv + (*v.e_pt)[e] : (*v.e_pt)[e];
      h.e_obs[2 * t] = (*v.e_obs)[2 * (size_t)e];
      h.e_obs[2 * t + 1] = (*v.e_obs)[2 * (size_t)e + 1];
      h.e_w[t] = (*v.e_w)[e];
      if (!cf) h.cam_ptr[(*v.perm)[(*v.e_cam)[e]] + 1]++;
    }
    for (int c = 0; c < ncv; c++) h.cam_ptr[c + 1] += h.cam_ptr[c];
    h.cam_slot.resize(ncv);
    h.slot2int.assign(ncv + v.ncf, -1);
    for (int u = 0; u < ncv; u++) {
      h.cam_slot[(*v.perm)[u]] = u;
      h.slot2int[u] = (*v.perm)[u];
    }
    const std::vector<int>& po = *v.porder;
    h.p2e.resize(po.size());
    h.pt_ptr.assign(npv + 1, 0);
    for (size_t t = 0; t < po.size(); t++) {
      h.p2e[t] = epos[po[t]];
      h.pt_ptr[(*v.e_pt)[po[t]] + 1]++;
    }
    for (int p = 0; p < npv; p++) h.pt_ptr[p + 1] += h.pt_ptr[p];
    // S blocks (i <= j) and their pairs, points ascending (MatrixWWtMultiplier::prepare order)
    std::vector<int> bid((size_t)ncv * ncv, -1);
    for (int c = 0; c < ncv; c++) {
      bid[(size_t)c * ncv + c] = (int)h.s_i.size();
      h.s_i.push_back(c);
      h.s_j.push_back(c);
    }
    std::vector<std::vector<std::pair<int, int>>> blist;
    blist.resize(ncv);
    std::vector<int> ve;
    for (int p = 0; p < npv; p++) {
      ve.clear();
      for (int t = h.pt_ptr[p]; t < h.pt_ptr[p + 1]; t++)
        if (h.e_cam[h.p2e[t]] < ncv) ve.push_back(h.p2e[t]);
      for (int a : ve)
        for (int bb : ve) {
          const int ci = (*v.perm)[h.e_cam[a]], cj = (*v.perm)[h.e_cam[bb]];
          if (ci > cj) continue;
          int& id = bid[(size_t)ci * ncv + cj];
          if (id < 0) {
            id = (int)h.s_i.size();
            h.s_i.push_back(ci);
            h.s_j.push_back(cj);
            blist.emplace_back();
          }
          blist[id].push_back({a, bb});
        }
    }
    h.s_ptr.assign(h.s_i.size() + 1, 0);
    for (size_t q = 0; q < h.s_i.size(); q++) {
      h.s_ptr[q + 1] = h.s_ptr[q] + (int)blist[q].size();
      for (auto& pr : blist[q]) {
        h.pa.push_back(pr.first);
        h.pb.push_back(pr.second);
      }
    }
    const int nn = ncv * bc;
    work[i] = (double)h.pa.size() * bc * bc * 3 + (double)nn * nn * nn / 6.0 + 60.0 * ne * bc;
    // arena layout (bytes)
    const size_t nc_all = (size_t)ncv + v.ncf, np_all = (size_t)npv + v.npf;
    const size_t lw = bc == 9 ? Layout<double, 9>::W : Layout<double, 6>::W;
    const size_t sizes[] = {
        sizeof(int) * ne, sizeof(int) * ne, sizeof(double) * 2 * ne, sizeof(double) * ne,                  // 0-3
        sizeof(int) * (ncv + 1), sizeof(int) * ncv, sizeof(int) * (ncv + v.ncf), sizeof(int) * (npv + 1),  // 4-7
        sizeof(int) * h.p2e.size(), sizeof(int) * h.s_i.size(), sizeof(int) * h.s_j.size(),                 // 8-10
        sizeof(int) * h.s_ptr.size(), sizeof(int) * h.pa.size(), sizeof(int) * h.pb.size(),                 // 11-13
        sizeof(double) * nc_all * 16, sizeof(double) * np_all * 3,                                          // 14-15
        sizeof(double) * nc_all * 16, sizeof(double) * np_all * 3,                                          // 16-17
        sizeof(double) * ne * lw, sizeof(double) * ne * lw,                                                 // 18-19 W, Y
        sizeof(double) * ncv * bc * bc, sizeof(double) * ncv * bc,                                          // 20-21 U, bU
        sizeof(double) * npv * 9, sizeof(double) * npv * 10, sizeof(double) * npv * 3,                       // 22-24
        sizeof(double) * (nn + 1) * nn, sizeof(double) * (nn + 3 * npv),                                   // 25-26
        sizeof(double) * ((size_t)std::max(ne, nn + 3 * npv) / 32 + 64)};                                   // 27
    for (size_t s : sizes) {
      offs[i].push_back(total);
      total += al(std::max<size_t>(s, 8));
    }
    b->max_n = std::max(b->max_n, nn);
  }
  nl_status s;
  if ((s = b->arena.alloc(total)) != NL_OK) return s;
  char* base = static_cast<char*>(b->arena.p);
  b->hp.resize(n);
  b->off_cam.resize(n);
  b->off_pt.resize(n);
  for (int i = 0; i < n; i++) {
    const nl_problem_view& v = vs[i];
    HostProb& h = H[i];
    const std::vector<size_t>& o = offs[i];
    BProb& P = b->hp[i];
    P = BProb{};
    P.ncv = v.ncv;
    P.nc_all = v.ncv + v.ncf;
    P.npv = v.npv;
    P.np_all = v.npv + v.npf;
    P.ne = (int)h.e_cam.size();
    P.n = v.ncv * bc;
    P.nS = (int)h.s_i.size();
    P.f = v.f;
    P.cx = v.cx;
    P.cy = v.cy;
    auto put = [&](int k, const void* src, size_t bytes) -> nl_status {
      if (bytes) NL_CUDA(cudaMemcpyAsync(base + o[k], src, bytes, cudaMemcpyHostToDevice, b->st));
      return NL_OK;
    };
#define NL_PUT(k, vec)                                                                              \
  if ((s = put(k, vec.data(), vec.size() * sizeof(vec[0]))) != NL_OK) return s;
    NL_PUT(0, h.e_cam) NL_PUT(1, h.e_pt) NL_PUT(2, h.e_obs) NL_PUT(3, h.e_w) NL_PUT(4, h.cam_ptr)
    NL_PUT(5, h.cam_slot) NL_PUT(6, h.slot2int) NL_PUT(7, h.pt_ptr) NL_PUT(8, h.p2e) NL_PUT(9, h.s_i)
    NL_PUT(10, h.s_j) NL_PUT(11, h.s_ptr) NL_PUT(12, h.pa) NL_PUT(13, h.pb)
#undef NL_PUT
    P.e_cam = reinterpret_cast<const int*>(base + o[0]);
    P.e_pt = reinterpret_cast<const int*>(base + o[1]);
    P.e_obs = reinterpret_cast<const double*>(base + o[2]);
    P.e_w = reinterpret_cast<const double*>(base + o[3]);
    P.cam_ptr = reinterpret_cast<const int*>(base + o[4]);
    P.cam_slot = reinterpret_cast<const int*>(base + o[5]);
    P.slot2int = reinterpret_cast<const int*>(base + o[6]);
    P.pt_ptr = reinterpret_cast<const int*>(base + o[7]);
    P.p2e = reinterpret_cast<const int*>(base + o[8]);
    P.s_i = reinterpret_cast<const int*>(base + o[9]);
    P.s_j = reinterpret_cast<const int*>(base + o[10]);
    P.s_ptr = reinterpret_cast<const int*>(base + o[11]);
    P.pa = reinterpret_cast<const int*>(base + o[12]);
    P.pb = reinterpret_cast<const int*>(base + o[13]);
    double* d[14];
    for (int k = 14; k < 28; k++) d[k - 14] = reinterpret_cast<double*>(base + o[k]);
    P.cam = d[0];
    P.pt = d[1];
    P.cam_bck = d[2];
    P.pt_bck = d[3];
    P.W = d[4];
    P.Y = d[5];
    P.U = d[6];
    P.bU = d[7];
    P.V = d[8];
    P.Vinv = d[9];
    P.bV = d[10];
    P.S = d[11];
    P.inc = d[12];
    P.part = d[13];
    b->off_cam[i] = o[14];
    b->off_pt[i] = o[15];
  }
  // W / Y of edges without a variable camera or point are never read; zero all once
  if ((s = upload(b->probs, b->hp, b->st)) != NL_OK) return s;
  std::vector<int> ord(n);
  std::iota(ord.begin(), ord.end(), 0);
  std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return work[x] > work[y]; });
  if ((s = upload(b->order, ord, b->st)) != NL_OK) return s;
  if ((s = b->queue.alloc(sizeof(int) * 8)) != NL_OK) return s;
  if ((s = b->reps.alloc(sizeof(BReport) * n)) != NL_OK) return s;
  if ((s = b->params.alloc(sizeof(ParamCopy) * n)) != NL_OK) return s;
  NL_CUDA(cudaStreamSynchronize(b->st));
  *out = b.release();
  return NL_OK;
}

nl_status nl_batch_destroy(nl_batch* b) {
  if (!b) return NL_ERR_ARG;
  cudaSetDevice(b->device);
  cudaStreamSynchronize(b->st);
  delete b;
  return NL_OK;
}

}  // extern "C"

namespace {

nl_status batch_launch(nl_batch* b, const nl::BSettings& s, int nt, int cps, float* ms) {
  using namespace nl;
  // the Cholesky panel (its rows, bS, at least one block) or the warps' work areas
  const size_t warp_d = b->bc == 9 ? BatchCfg<9>::kWarpDoubles : BatchCfg<6>::kWarpDoubles;
  const size_t smem = sizeof(double) * std::max((size_t)(std::max(b->max_n, kPW) + 1) * kPLd, warp_d * (size_t)(nt / 32));
  BatchKernel k = b->bc == 9 ? batch_lm_kernel<9> : batch_lm_kernel<6>;
  NL_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int sms = 0, occ = 0;
  NL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device));
  NL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, nt, smem));
  if (occ <= 0) return NL_ERR_UNSUPPORTED;
  const int grid = std::max(1, std::min(b->n, sms * std::min(cps, occ)));
  NL_CUDA(cudaMemsetAsync(b->queue.p, 0, sizeof(int), b->st));
  NL_CUDA(cudaEventRecord(b->e0, b->st));
  k<<<grid, nt, smem, b->st>>>(b->probs.as<BProb>(), b->order.as<int>(), b->n, b->queue.as<int>(), s,
                               b->reps.as<BReport>());
  NL_CUDA(cudaGetLastError());
  NL_CUDA(cudaEventRecord(b->e1, b->st));
  NL_CUDA(cudaEventSynchronize(b->e1));
  NL_CUDA(cudaEventElapsedTime(ms, b->e0, b->e1));
  return NL_OK;
}

__global__ void batch_params_kernel(const nl::ParamCopy* __restrict__ pc, int to_arena) {
  const nl::ParamCopy c = pc[blockIdx.x];
  const double* cs = to_arena ? c.h_cam : c.a_cam;
  double* cd = to_arena ? c.a_cam : c.h_cam;
  const double* ps = to_arena ? c.h_pt : c.a_pt;
  double* pd = to_arena ? c.a_pt : c.h_pt;
  const int t = blockIdx.y * blockDim.x + threadIdx.x, nt = gridDim.y * blockDim.x;
  for (int i = t; i < c.nc; i += nt) cd[i] = cs[i];
  for (int i = t; i < c.np; i += nt) pd[i] = ps[i];
}

// parameters: handles <-> arena, one launch for all problems (two copies a
// problem took 2 x 128 launches of ~1.7 us for 128 problems)
nl_status batch_params(nl_batch* b, bool to_arena) {
  using namespace nl;
  if (to_arena) {  // the copy back of the same call uses this table
    char* base = static_cast<char*>(b->arena.p);
    std::vector<ParamCopy> pc(b->n);
    for (int i = 0; i < b->n; i++) {
      nl_problem_view v;
      nl_status s = nl_problem_get_view(b->hs[i], &v);
      if (s != NL_OK) return s;
      pc[i] = {v.d_cam, v.d_pt, reinterpret_cast<double*>(base + b->off_cam[i]),
               reinterpret_cast<double*>(base + b->off_pt[i]), (v.ncv + v.ncf) * 16, (v.npv + v.npf) * 3};
    }
    NL_CUDA(cudaMemcpyAsync(b->params.p, pc.data(), sizeof(ParamCopy) * b->n, cudaMemcpyHostToDevice, b->st));
  }
  batch_params_kernel<<<dim3(b->n, 4), 256, 0, b->st>>>(b->params.as<ParamCopy>(), to_arena ? 1 : 0);
  NL_CUDA(cudaGetLastError());
  return NL_OK;
}

}  // namespace

extern "C" {

nl_status nl_batch_autotune(nl_batch* b, const nl_lm_settings* st, int* nt_out, int* cps_out) {
  using namespace nl;
  if (!b || !st) return NL_ERR_ARG;
  NL_CUDA(cudaSetDevice(b->device));
  BSettings s{st->maxNumIt, st->maxNumSubIt, st->minNumIt, 0, st->epsBVector, st->epsIncSquare, st->epsChi2,
              st->tau, st->penaltyV, st->initV, st->maxScaleFactor, st->minScaleFactor};
  const int cand_nt[3] = {128, 256, 512};
  const int cand_cps[2] = {1, 2};
  float best = 1e30f;
  int bn = 256, bcps = 1, q = 0;
  for (int a = 0; a < 3; a++)
    for (int c = 0; c < 2; c++, q++) {
      nl_status r = batch_params(b, true);  // every candidate starts from the handles' parameters
      if (r != NL_OK) return r;
      float ms = 0;
      r = batch_launch(b, s, cand_nt[a], cand_cps[c], &ms);
      if (r == NL_ERR_UNSUPPORTED) {
        b->tune_ms[q] = -1;
        continue;
      }
      if (r != NL_OK) return r;
      b->tune_ms[q] = ms;
      if (ms < best) {
        best = ms;
        bn = cand_nt[a];
        bcps = cand_cps[c];
      }
    }
  b->tuned_nt = bn;
  b->tuned_cps = bcps;
  if (nt_out) *nt_out = bn;
  if (cps_out) *cps_out = bcps;
  return NL_OK;
}

nl_status nl_batch_lm_solve(nl_batch* b, const nl_lm_settings* st, int threads, int ctas_per_sm,
                            nl_solve_report* reps, double* latency_ms, double* device_ms) {
  using namespace nl;
  if (!b || !st) return NL_ERR_ARG;
  if (threads != 0 && threads != 128 && threads != 256 && threads != 512) return NL_ERR_ARG;
  if (ctas_per_sm < 0 || ctas_per_sm > 4) return NL_ERR_ARG;
  NL_CUDA(cudaSetDevice(b->device));
  BSettings s{st->maxNumIt, st->maxNumSubIt, st->minNumIt, 0, st->epsBVector, st->epsIncSquare, st->epsChi2,
              st->tau, st->penaltyV, st->initV, st->maxScaleFactor, st->minScaleFactor};
  // untuned: 512 threads (128 problems of 8 .. 64 cameras, 6 iterations: 10.4 ms against
  // 17.5 ms with 256 and 30.4 with 128; 9 parameters 20.1, 27.9, 47.7)
  const int nt = threads ? threads : (b->tuned_nt ? b->tuned_nt : 512);
  const int cps = ctas_per_sm ? ctas_per_sm : (b->tuned_cps ? b->tuned_cps : 1);
  nl_status r = batch_params(b, true);
  if (r != NL_OK) return r;
  float ms = 0;
  if ((r = batch_launch(b, s, nt, cps, &ms)) != NL_OK) return r;
  if ((r = batch_params(b, false)) != NL_OK) return r;
  std::vector<BReport> hr(b->n);
  NL_CUDA(cudaMemcpyAsync(hr.data(), b->reps.p, sizeof(BReport) * b->n, cudaMemcpyDeviceToHost, b->st));
  NL_CUDA(cudaStreamSynchronize(b->st));
  unsigned long long t0 = ~0ull;
  for (auto& x : hr) t0 = std::min(t0, x.t_start);
  for (int i = 0; i < b->n; i++) {
    if (reps) {
      reps[i].reason = hr[i].reason;
      reps[i].iterations = hr[i].iterations;
      reps[i].subiterations = hr[i].subiterations;
      reps[i].n_trace = 0;
      reps[i].chi2 = hr[i].chi2;
      reps[i].mu = hr[i].mu;
      reps[i].device_ms = 1e-6 * (double)(hr[i].t_end - hr[i].t_start);
    }
    if (latency_ms) latency_ms[i] = 1e-6 * (double)(hr[i].t_end - t0);
  }
  if (device_ms) *device_ms = ms;
  return NL_OK;
}

}  // extern "C"
