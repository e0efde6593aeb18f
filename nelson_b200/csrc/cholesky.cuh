// cholesky.cuh -- blocked right-looking Cholesky of the reduced camera system.
//
// Replaces the dense LDLT factorisation + solve of SolverCholeskySchur
// (SolverCholeskyEigenDense::factorize/solve, nelson/SolverCholeskyDense.hpp:15-24,
// used at nelson/SolverCholeskySchur.hpp:136-140).  S is stored dense,
// row-major, lower triangle, n padded to a multiple of NB = 128 (identity on
// the padding).  Per 128-wide panel k:
//   potrf_diag_kernel  factor of the diagonal tile (one CTA) and the inverses
//                      of its 16 x 16 diagonal blocks
//   trsm_kernel        L_ik = A_ik L_kk^-T by substitution with those
//   syrk update        A_ij -= L_ik L_jk' on the trailing lower triangle
//                      (tensor-core kernel in tc_syrk.cu for the mixed path,
//                      cuBLAS DSYRK for the FP64 comparison path)
// After the last panel inv_tiles_kernel forms the inverses of all diagonal
// tiles; solves use them: trsv_fwd/bwd_kernel with a ticketed
// look-back between CTAs of one launch, each wait bounded.
#pragma once

#include "nl_common.cuh"
#include "tc_pack_layout.cuh"

namespace nl {

constexpr int NB = 128;
constexpr long long kSpinLimit = 1LL << 24;  // default bound of the solves' waits (~1 s worst case)

// ---------------------------------------------------------------------------
// One CTA: factor the NB x NB diagonal tile of panel k in the storage
// precision T (FP64 for the FP64 path; FP32 for the mixed path, whose
// trailing updates and off-diagonal solves are FP32-accurate as well and whose
// factor only preconditions the FP64 refinement) and invert the 16 x 16 blocks
// on its diagonal (all that the panel solves need; inv_tiles_kernel completes
// the inverse of every tile at once, off the chain).
//
// The tile is bound by its 128 dependent pivots, so the kernel is laid out
// around that chain, in eight block columns of 16:
//   pivot warp    the diagonal block, a lane holding one row of 16 columns in
//       registers (lanes 16 .. 31 repeat lanes 0 .. 15).  With u = the unscaled
//       column, d its pivot and r = 1 / d, an entry becomes a_c -= (a_j r) u_c
//       (u and d times kPivScale, r over it).
//       Every lane carries the next pivot itself (d' = v - u1 (u1 r), u1 and v
//       fetched by shuffle while r is formed), so a column costs one reciprocal
//       and a few FMAs of latency; the columns further right are updated one
//       step late from the column published in shared memory.  It has its
//       scheduler to itself.
//   row warps     apply the published columns to the rows below, one per lane,
//       8 columns at a time behind the pivot warp (named barriers), so the
//       panel solve runs under the pivot chain; 16 rows of the identity beside
//       them become the inverse of the diagonal block.
//   helper warps  complete the block column under way (its last update, which
//       the row warps wait for) and apply all but the last update to the next
//       one: left-looking, so that the work is even over the block columns.
// Between two block columns only the last update of the next diagonal block is
// left on the chain.  Blocks of 16 keep the unrolled code of the roles that run
// side by side within the instruction cache (blocks of 32 did not: about 3
// cycles an instruction).  One tile after another on an idle B200: FP32 15.4 us
// against 30.0 us, FP64 22.6 against 67.5, for 32 rank-4 super-steps that
// formed the whole inverse as well (forming it here too: 20.5 and 28.7 us).
constexpr int PB = 16;
constexpr int kPBlocks = NB / PB;
constexpr int kPotLd = NB + 4;     // row stride of `sm` (conflict-free rows and MMA operands)
constexpr int kPotDld = PB + 4;    // of `dg`
constexpr int kRowWarps = 4;
constexpr int PT = 512, kHelpWarps = 8;
// Warp roles: a scheduler serves the warps of equal index mod 4, and warps 4,
// 8 and 12 stay off the pivot warp's.  0: pivot, 1 .. 4: row warps, 5 .. 12:
// helpers, -1: none.
__device__ __forceinline__ int potrf_role(int w) { return w == 0 ? 0 : (w & 3) == 0 ? -1 : w - (w >> 2); }
template <typename T>
constexpr size_t potrf_smem() {
  return sizeof(T) * ((size_t)NB * (kPotLd + kPotDld) + PB * PB + 2 * PB);
}

// four consecutive elements (16-byte aligned; any address space)
__device__ inline void store_row4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ inline void store_row4(double* p, double a, double b, double c, double d) {
  reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
  reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
}
__device__ inline void load_row4(const float* p, float v[4]) {
  const float4 x = *reinterpret_cast<const float4*>(p);
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ inline void load_row4(const double* p, double v[4]) {
  const double2 x = reinterpret_cast<const double2*>(p)[0], y = reinterpret_cast<const double2*>(p)[1];
  v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}
// Shared memory by 32-bit shared-window address (a pointer picked at run time
// between two shared arrays would be read through the generic path).
template <typename T>
struct Sh {
  uint32_t a;
  __device__ __forceinline__ Sh operator+(int i) const { return Sh{a + (uint32_t)(i * (int)sizeof(T))}; }
};
__device__ __forceinline__ void load_row4(Sh<float> p, float v[4]) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(p.a));
}
__device__ __forceinline__ void load_row4(Sh<double> p, double v[4]) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(p.a));
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "r"(p.a + 16));
}
__device__ __forceinline__ void store_row4(Sh<float> p, float a, float b, float c, float d) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(p.a), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void store_row4(Sh<double> p, double a, double b, double c, double d) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(p.a), "d"(a), "d"(b) : "memory");
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(p.a + 16), "d"(c), "d"(d) : "memory");
}
__device__ __forceinline__ void load_two(Sh<float> p, float& x, float& y) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(p.a));
}
__device__ __forceinline__ void load_two(Sh<double> p, double& x, double& y) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(p.a));
}
__device__ __forceinline__ void store_two(Sh<float> p, float x, float y) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(p.a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void store_two(Sh<double> p, double x, double y) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(p.a), "d"(x), "d"(y) : "memory");
}
__device__ __forceinline__ void store_one(Sh<float> p, float x) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(p.a), "f"(x) : "memory");
}
__device__ __forceinline__ void store_one(Sh<double> p, double x) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(p.a), "d"(x) : "memory");
}
__device__ __forceinline__ float load_one(Sh<float> p) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(p.a));
  return v;
}
__device__ __forceinline__ double load_one(Sh<double> p) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p.a));
  return v;
}
// 16-byte global -> shared copies that complete asynchronously: a kernel
// issues all of its staging before one wait, so the staging costs one L2 /
// HBM round trip however loaded the memory system is
__device__ inline void cp_async16(uint32_t sa, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ inline void cp_async16(void* smem, const void* gmem) {
  cp_async16((uint32_t)__cvta_generic_to_shared(smem), gmem);
}
__device__ inline void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ inline void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// A pivot d is carried as kPivScale d, and the published columns have the same
// factor.  FP32 takes a quarter: its reciprocal 4 / d is then a normal number up to the end
// of the range, where that of d is subnormal above 2^126 and the flushing rcp.approx
// would leave the column out of the elimination (the one that does not flush costs
// 0.6 us a tile in the chain).  A power of two changes no other bit.
template <typename T>
constexpr T kPivScale = sizeof(T) == 4 ? (T)0.25 : (T)1;
// 1 / dq and 1 / sqrt(d) of a pivot, dq = kPivScale d, clamped away from zero (a
// non-positive pivot is flagged separately)
__device__ __forceinline__ void pivot_inv(float dq, float& ri, float& rs) {
  dq = fmaxf(dq, 0.25e-30f);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ri) : "f"(dq));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(rs) : "f"(dq));
  rs *= 0.5f;
}
__device__ __forceinline__ void pivot_inv(double dq, double& ri, double& rs) {
  rs = rsqrt(fmax(dq, 1e-300));
  ri = rs * rs;
}

__device__ __forceinline__ void named_sync(int id, int n) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(n) : "memory");
}

// Eliminates the 16 x 16 block whose row lane % 16 is a[] (entries right of the
// diagonal are ignored), leaving the row of L in a[] and publishing every
// column (times kPivScale) in uc, (1 / (kPivScale d), 1 / sqrt(d)) in inv_s.  False
// on a non-positive pivot.
// kPaced: named barriers pace the row warps of the same CTA behind it.
template <typename T, bool kPaced = true>
__device__ __forceinline__ bool pivot_block(T (&a)[PB], Sh<T> uc, Sh<T> inv_s, int lane) {
  bool ok = true;
  constexpr T kQ = kPivScale<T>;
  T dq = kQ * __shfl_sync(0xffffffffu, a[0], 0);
  T up[PB];
  T tp = (T)0;
#pragma unroll
  for (int j = 0; j < PB; j++) {
    T ri, rs;
    pivot_inv(dq, ri, rs);
    T u1 = (T)0, u2 = (T)0, v = (T)0;
    if (j + 1 < PB) {
      u1 = kQ * __shfl_sync(0xffffffffu, a[j], j + 1);
      v = kQ * __shfl_sync(0xffffffffu, a[j + 1], j + 1);
    }
    if (j + 2 < PB) u2 = kQ * __shfl_sync(0xffffffffu, a[j], j + 2);
    if (lane < PB) store_one(uc + (j * PB + lane), kQ * a[j]);
    ok &= dq > (T)0 && isfinite(dq);
    // column j - 1 applied to the columns that its step left out
    if (j > 0) {
#pragma unroll
      for (int c = j + 2; c < PB; c++) a[c] -= tp * up[c];
    }
    if (lane == 0) store_two(inv_s + 2 * j, ri, rs);
    __syncwarp();
#pragma unroll
    for (int c = (j + 3) & ~3; c < PB; c += 4) {
      T q[4];
      load_row4(uc + (j * PB + c), q);
#pragma unroll
      for (int i = 0; i < 4; i++) up[c + i] = q[i];
    }
    const T t = a[j] * ri;
    if (j + 1 < PB) {
      dq = v - u1 * (u1 * ri);
      a[j + 1] -= t * u1;
    }
    if (j + 2 < PB) a[j + 2] -= t * u2;
    a[j] *= rs;
    tp = t;
    if (kPaced && (j & 7) == 7) named_arrive(1 + (j >> 3), 32 * (1 + kRowWarps));
  }
  return ok;
}

// The same elimination for a row outside the pivot block.
template <typename T, bool kPaced = true>
__device__ __forceinline__ void follow_block(T (&a)[PB], Sh<T> uc, Sh<T> inv_s) {
#pragma unroll
  for (int j = 0; j < PB; j++) {
    if (kPaced && (j & 7) == 0) named_sync(1 + (j >> 3), 32 * (1 + kRowWarps));
    T ri, rs;
    load_two(inv_s + 2 * j, ri, rs);
    const T t = a[j] * ri;
#pragma unroll
    for (int c = (j + 1) & ~3; c < PB; c += 4) {
      T q[4];
      load_row4(uc + (j * PB + c), q);
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (c + i > j) a[c + i] -= t * q[i];
    }
    a[j] *= rs;
  }
}

// 16 x 8 piece of one warp: C -= P Q' over k in [k0, k1) (multiples of 16), P
// and Q rows of `sm`.
// FP32: lane (g, t) = (lane / 4, lane % 4) owns rows g, g + 8, columns 2 t, 2 t + 1
__device__ __forceinline__ void help_block(Sh<float> C, Sh<float> P, Sh<float> Q, int k0, int k1, int lane) {
  const int g = lane >> 2, t = lane & 3;
  float acc[2][2] = {};
  P = P + g * kPotLd;
  Q = Q + 2 * t * kPotLd;
#pragma unroll 1
  for (int k = k0; k < k1; k += PB) {
#pragma unroll
    for (int kk = 0; kk < PB; kk += 4) {
      float p[2][4], q[2][4];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        load_row4(P + (8 * i * kPotLd + k + kk), p[i]);
        load_row4(Q + (i * kPotLd + k + kk), q[i]);
      }
#pragma unroll
      for (int m = 0; m < 4; m++)
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int j = 0; j < 2; j++) acc[i][j] += p[i][m] * q[j][m];
    }
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const Sh<float> c = C + ((g + 8 * i) * kPotLd + 2 * t);
    float x, y;
    load_two(c, x, y);
    store_two(c, x - acc[i][0], y - acc[i][1]);
  }
}
// FP64: mma.m8n8k4 (FP64 in and out, 1.6 times the rate of FMAs), lane = 4 g + t
__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}
__device__ __forceinline__ void help_block(Sh<double> C, Sh<double> P, Sh<double> Q, int k0, int k1, int lane) {
  const int g = lane >> 2, t = lane & 3;
  double acc[2][2][2] = {};
  P = P + (g * kPotLd + t);
  Q = Q + (g * kPotLd + t);
#pragma unroll 1
  for (int k = k0; k < k1; k += PB) {
#pragma unroll
    for (int kk = 0; kk < PB; kk += 4) {
      const double b = load_one(Q + (k + kk));
#pragma unroll
      for (int i = 0; i < 2; i++) mma_f64(acc[(kk >> 2) & 1][i], load_one(P + (8 * i * kPotLd + k + kk)), b);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const Sh<double> c = C + ((g + 8 * i) * kPotLd + 2 * t);
    double x, y;
    load_two(c, x, y);
    store_two(c, x - (acc[0][i][0] + acc[1][i][0]), y - (acc[0][i][1] + acc[1][i][1]));
  }
}

// 8 x 8 piece of the next diagonal block: C -= P Q' over 16 columns
__device__ __forceinline__ void diag_piece(Sh<float> C, Sh<float> P, Sh<float> Q, int lane) {
  const int r = lane >> 2, c = 2 * (lane & 3);
  float s0[2] = {0.f, 0.f}, s1[2] = {0.f, 0.f};
#pragma unroll
  for (int k = 0; k < PB; k += 4) {
    float x[4], y[4], z[4];
    load_row4(P + (r * kPotLd + k), x);
    load_row4(Q + (c * kPotLd + k), y);
    load_row4(Q + ((c + 1) * kPotLd + k), z);
#pragma unroll
    for (int m = 0; m < 4; m++) {
      s0[m & 1] += x[m] * y[m];
      s1[m & 1] += x[m] * z[m];
    }
  }
  const Sh<float> o = C + (r * kPotLd + c);
  float x, y;
  load_two(o, x, y);
  store_two(o, x - (s0[0] + s0[1]), y - (s1[0] + s1[1]));
}
__device__ __forceinline__ void diag_piece(Sh<double> C, Sh<double> P, Sh<double> Q, int lane) {
  const int g = lane >> 2, t = lane & 3;
  double acc[2] = {0.0, 0.0};
#pragma unroll
  for (int k = 0; k < PB; k += 4) mma_f64(acc, load_one(P + (g * kPotLd + k + t)), load_one(Q + (g * kPotLd + k + t)));
  const Sh<double> c = C + (g * kPotLd + 2 * t);
  double x, y;
  load_two(c, x, y);
  store_two(c, x - acc[0], y - acc[1]);
}

// Block column p of L (rows 16 p .., zeros above the diagonal) to the tile, and
// the inverse of its diagonal block (transposed rows in dg) to X.  Threads id, id + n, ...
template <typename T>
__device__ __forceinline__ void potrf_write(Sh<T> sm, Sh<T> dg, int p, T* __restrict__ A, int ld, T* __restrict__ X,
                                            int id, int n) {
  const int nl = (NB - p * PB) * 4;
#pragma unroll 1
  for (int e = id; e < nl; e += n) {
    const int r = p * PB + (e >> 2), c = p * PB + 4 * (e & 3);
    T v[4];
    load_row4(sm + (r * kPotLd + c), v);
    store_row4(A + (size_t)r * ld + c, v[0], v[1], v[2], v[3]);
  }
  if (id < PB) {  // 4 x 4 pieces
    const int b = 4 * (id & 3), c = 4 * (id >> 2);
    T v[4][4];
#pragma unroll
    for (int q = 0; q < 4; q++) load_row4(dg + ((p * PB + b + q) * kPotDld + c), v[q]);
#pragma unroll
    for (int q = 0; q < 4; q++)
      store_row4(X + (size_t)(p * PB + c + q) * NB + p * PB + b, v[0][q], v[1][q], v[2][q], v[3][q]);
  }
}

template <typename T>
__device__ __forceinline__ void load_row16(Sh<T> p, T (&a)[PB]) {
#pragma unroll
  for (int c = 0; c < PB; c += 4) {
    T q[4];
    load_row4(p + c, q);
#pragma unroll
    for (int i = 0; i < 4; i++) a[c + i] = q[i];
  }
}
template <typename T>
__device__ __forceinline__ void store_row16(Sh<T> p, const T (&a)[PB]) {
#pragma unroll
  for (int c = 0; c < PB; c += 4) store_row4(p + c, a[c], a[c + 1], a[c + 2], a[c + 3]);
}

template <typename T>
static __global__ void __launch_bounds__(PT, 1) potrf_diag_kernel(T* __restrict__ S, int ld, int k,
                                                               T* __restrict__ Linv, int* __restrict__ status,
                                                               const int* __restrict__ active) {
  constexpr int EPV = 16 / (int)sizeof(T);
  extern __shared__ float4 smf4[];
  const Sh<T> sm{(uint32_t)__cvta_generic_to_shared(smf4)};  // L on and below the diagonal 16-blocks
  const Sh<T> dg = sm + NB * kPotLd;     // inverses of the diagonal blocks, transposed
  const Sh<T> uc = dg + NB * kPotDld;    // published columns of the pivot block
  const Sh<T> inv_s = uc + PB * PB;    // (1 / (kPivScale d), 1 / sqrt(d)) per column
  chain_release();
  chain_wait();
  if (active && !*active) return;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, role = potrf_role(w);
  T* A = S + (size_t)k * NB * ld + (size_t)k * NB;
  T* X = Linv + (size_t)k * NB * NB;
  // the lower 16-blocks of the tile
#pragma unroll 4
  for (int e = tid; e < NB * (NB / EPV); e += PT) {
    const int r = e / (NB / EPV), c = EPV * (e % (NB / EPV));
    if (c <= (r | (PB - 1))) cp_async16((sm + (r * kPotLd + c)).a, A + (size_t)r * ld + c);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
#pragma unroll 1
  for (int kb = 0; kb < kPBlocks; kb++) {
    if (role == 0) {
      const Sh<T> row = sm + ((kb * PB + (lane & (PB - 1))) * kPotLd + kb * PB);
      T a[PB];
      load_row16(row, a);
      if (!pivot_block(a, uc, inv_s, lane) && lane == 0) atomicOr(status, ST_CHOL_FAIL);
      if (lane < PB) {
#pragma unroll
        for (int c = 0; c < PB; c++)
          if (c > lane) a[c] = (T)0;
        store_row16(row, a);
      }
    } else if (role > 0 && role <= kRowWarps) {
      // A row r below block kb, a row of the identity in it
      const int r = 32 * (role - 1) + lane;
      const bool unit = r / PB == kb;
      if (kb > 0) named_sync(3, 32 * (kHelpWarps + kRowWarps));
      T a[PB];
      load_row16(sm + (r * kPotLd + kb * PB), a);
#pragma unroll
      for (int c = 0; c < PB; c++)
        if (unit) a[c] = c == (r & (PB - 1)) ? (T)1 : (T)0;
      follow_block(a, uc, inv_s);
      if (r / PB >= kb) store_row16(unit ? dg + r * kPotDld : sm + (r * kPotLd + kb * PB), a);
    } else if (role > 0 && kb > 0) {
      // 16 x 8 pieces: block column kb with block column kb - 1 (rows below its
      // diagonal block, which is done), then block column kb + 1 with 0 .. kb - 1
      const int hw = role - 1 - kRowWarps, n = 2 * (kPBlocks - 1 - kb);
#pragma unroll 1
      for (int u = hw; u < n; u += kHelpWarps) {
        const int r = (kb + 1 + (u >> 1)) * PB, c = kb * PB + 8 * (u & 1);
        help_block(sm + (r * kPotLd + c), sm + r * kPotLd, sm + c * kPotLd, (kb - 1) * PB, kb * PB, lane);
      }
      named_arrive(3, 32 * (kHelpWarps + kRowWarps));
      // the warps without a piece above first
#pragma unroll 1
      for (int u = (hw + kHelpWarps - n % kHelpWarps) % kHelpWarps; u < n; u += kHelpWarps) {
        const int r = (kb + 1 + (u >> 1)) * PB, c = (kb + 1) * PB + 8 * (u & 1);
        help_block(sm + (r * kPotLd + c), sm + r * kPotLd, sm + c * kPotLd, 0, kb * PB, lane);
      }
      potrf_write(sm, dg, kb - 1, A, ld, X, hw * 32 + lane, 32 * kHelpWarps);
    }
    __syncthreads();
    if (kb + 1 < kPBlocks) {
      // the next diagonal block, 8 x 8 pieces on and below the diagonal
      if (w < 3) {
        const int i = w > 0, j = w > 1, b = (kb + 1) * PB;
        diag_piece(sm + ((b + 8 * i) * kPotLd + b + 8 * j), sm + ((b + 8 * i) * kPotLd + kb * PB),
                   sm + ((b + 8 * j) * kPotLd + kb * PB), lane);
      }
      __syncthreads();
    }
  }
  potrf_write(sm, dg, kPBlocks - 1, A, ld, X, tid, PT);
}

// ---------------------------------------------------------------------------
// Panel solve L_ik = A_ik inv(L_kk)' for rows [row_begin, row_begin + nrows)
// below the diagonal tile (absolute row indices), by substitution over the
// eight block columns of 16 with the inverses of L_kk's diagonal blocks: half
// the products of a multiplication by the whole inverse, and nothing waits for
// that one.  A CTA owns 16 RT rows; thread (ty, tx) holds rows ty RT .. of
// columns tx + 16 j, so a row lives in half a warp and the substitution needs
// no CTA barrier.  Step kb: y = t inv(L_kb,kb)' through shared memory, then
// the columns to the right (kept one block nearer in every step, so that the
// loop body is the same code) lose y L_j,kb'.
// RT = 1 while that leaves SMs idle; more rows a thread share L_kk's reads.
// 96 CTAs beside the chain: 8.0 us against 15.5 us for the product with the
// whole inverse by 64-row CTAs.
constexpr int kTrLd = NB + 4, kTrXld = PB + 4;
template <typename T, int RT>
constexpr size_t trsm_smem() {
  return sizeof(T) * ((size_t)NB * (kTrLd + kTrXld) + (size_t)16 * RT * (kTrLd + kTrXld));
}

template <typename T, int RT>
static __global__ void __launch_bounds__(256) trsm_kernel(T* __restrict__ S, int ld, int k, int row_begin, int nrows,
                                                          const T* __restrict__ Linv,
                                                          uint8_t* __restrict__ pack,
                                                          const int* __restrict__ active) {
  constexpr int ROWS = 16 * RT, EPV = 16 / (int)sizeof(T);
  extern __shared__ float4 smf4[];
  const Sh<T> sl{(uint32_t)__cvta_generic_to_shared(smf4)};  // L_kk, lower 16-blocks
  const Sh<T> sx = sl + NB * kTrLd;                          // inverses of its diagonal blocks
  const Sh<T> sy = sx + NB * kTrXld;                         // rows: A, then L
  const Sh<T> st = sy + ROWS * kTrLd;                        // t of one step
  chain_release();
  chain_wait();
  if (active && !*active) return;
  const int tid = threadIdx.x;
  const int r0 = row_begin + blockIdx.x * ROWS;
  const int nr = min(ROWS, row_begin + nrows - r0);
  if (nr <= 0) return;
  const T* D = S + (size_t)k * NB * ld + (size_t)k * NB;
  const T* X = Linv + (size_t)k * NB * NB;
  T* A = S + (size_t)r0 * ld + (size_t)k * NB;
#pragma unroll 4
  for (int e = tid; e < NB * (NB / EPV); e += 256) {
    const int r = e / (NB / EPV), c = EPV * (e % (NB / EPV));
    if (c < (r & ~(PB - 1)))
      cp_async16((sl + (r * kTrLd + c)).a, D + (size_t)r * ld + c);
    else if (c <= (r | (PB - 1)))
      cp_async16((sx + (r * kTrXld + (c & (PB - 1)))).a, X + (size_t)r * NB + c);
  }
#pragma unroll 4
  for (int e = tid; e < nr * (NB / EPV); e += 256) {
    const int r = e / (NB / EPV), c = EPV * (e % (NB / EPV));
    cp_async16((sy + (r * kTrLd + c)).a, A + (size_t)r * ld + c);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int tx = tid & 15, ty = tid >> 4;
  const Sh<T> y = sy + ty * RT * kTrLd, t = st + ty * RT * kTrXld;
  T acc[RT][kPBlocks];
#pragma unroll
  for (int r = 0; r < RT; r++)
#pragma unroll
    for (int j = 0; j < kPBlocks; j++) acc[r][j] = load_one(y + (r * kTrLd + tx + PB * j));
#pragma unroll 1
  for (int kb = 0; kb < kPBlocks; kb++) {
#pragma unroll
    for (int r = 0; r < RT; r++) store_one(t + (r * kTrXld + tx), acc[r][0]);
    __syncwarp();
    T v[RT];
#pragma unroll
    for (int r = 0; r < RT; r++) v[r] = (T)0;
#pragma unroll
    for (int c = 0; c < PB; c += 4) {
      T x[4];
      load_row4(sx + ((kb * PB + tx) * kTrXld + c), x);
#pragma unroll
      for (int r = 0; r < RT; r++) {
        T q[4];
        load_row4(t + (r * kTrXld + c), q);
#pragma unroll
        for (int m = 0; m < 4; m++) v[r] += q[m] * x[m];
      }
    }
#pragma unroll
    for (int r = 0; r < RT; r++) store_one(y + (r * kTrLd + kb * PB + tx), v[r]);
    __syncwarp();
    T q[RT][PB];
#pragma unroll
    for (int r = 0; r < RT; r++)
#pragma unroll
      for (int c = 0; c < PB; c += 4) {
        T w[4];
        load_row4(y + (r * kTrLd + kb * PB + c), w);
#pragma unroll
        for (int m = 0; m < 4; m++) q[r][c + m] = w[m];
      }
#pragma unroll
    for (int j = 0; j + 1 < kPBlocks; j++) {
      if (kb + 1 + j < kPBlocks) {
        const Sh<T> l = sl + (((kb + 1 + j) * PB + tx) * kTrLd + kb * PB);
        T s[RT];
#pragma unroll
        for (int r = 0; r < RT; r++) s[r] = (T)0;
#pragma unroll
        for (int c = 0; c < PB; c += 4) {
          T w[4];
          load_row4(l + c, w);
#pragma unroll
          for (int r = 0; r < RT; r++)
#pragma unroll
            for (int m = 0; m < 4; m++) s[r] += q[r][c + m] * w[m];
        }
#pragma unroll
        for (int r = 0; r < RT; r++) acc[r][j] = acc[r][j + 1] - s[r];
      }
    }
  }
  __syncthreads();
#pragma unroll 2
  for (int e = tid; e < nr * (NB / 4); e += 256) {
    const int r = e / (NB / 4), c = 4 * (e % (NB / 4));
    T v[4];
    load_row4(sy + (r * kTrLd + c), v);
    store_row4(A + (size_t)r * ld + c, v[0], v[1], v[2], v[3]);
  }
  if (sizeof(T) == 4 && pack) {
    // BF16 hi/lo pack of the rows for the tensor-core update, 8 consecutive columns per item
    const int rel0 = r0 - (k + 1) * NB;  // pack rows start below the diagonal tile
    for (int i = tid; i < nr * 16; i += 256) {
      const int rr = i >> 4, h = i & 15;
      float x[8];
#pragma unroll
      for (int q = 0; q < 8; q += 4) {
        T v[4];
        load_row4(sy + (rr * kTrLd + 8 * h + q), v);
#pragma unroll
        for (int m = 0; m < 4; m++) x[q + m] = (float)v[m];
      }
      tc_pack_store8(pack, tc_pack_offset(rel0 + rr, h), x);
    }
  }
}

// ---------------------------------------------------------------------------
// The same substitution for the row tile below panel j's diagonal tile, on the
// factorisation's critical path, as 32 CTAs of 4 rows: a row's 8 blocks are
// spread over four half-warps (half-warp group g holds blocks g and g + 4), so
// a step is one 16 x 16 product in the group that owns block kb, one barrier
// and at most two products in every other group.  Writes the rows and their
// BF16 pack.  6.0 us (8 CTAs of 16 rows through trsm_kernel: 8.0 us); what it
// adds to the 4 us of a product with the whole inverse is less than the
// diagonal factor saves by not forming that.
constexpr int kChainTrsmRows = 4;
template <typename T>
constexpr size_t trsm_tile_smem() {
  return sizeof(T) * ((size_t)NB * (kTrLd + kTrXld) + kChainTrsmRows * (kTrLd + kTrXld));
}
template <typename T>
static __global__ void __launch_bounds__(256) trsm_tile_kernel(T* __restrict__ S, int ld, int j,
                                                               const T* __restrict__ Linv,
                                                               uint8_t* __restrict__ pack,
                                                               const int* __restrict__ active) {
  constexpr int EPV = 16 / (int)sizeof(T), ROWS = kChainTrsmRows;
  extern __shared__ float4 smf4[];
  const Sh<T> sl{(uint32_t)__cvta_generic_to_shared(smf4)};  // L_jj, lower 16-blocks
  const Sh<T> sx = sl + NB * kTrLd;                          // inverses of its diagonal blocks
  const Sh<T> sy = sx + NB * kTrXld;                         // rows: A, then L
  const Sh<T> st = sy + ROWS * kTrLd;
  chain_release();
  chain_wait();
  if (active && !*active) return;
  const int tid = threadIdx.x, rel0 = blockIdx.x * ROWS;
  const T* D = S + (size_t)j * NB * ld + (size_t)j * NB;
  const T* X = Linv + (size_t)j * NB * NB;
  T* A = S + (size_t)((j + 1) * NB + rel0) * ld + (size_t)j * NB;
  for (int e = tid; e < ROWS * (NB / EPV); e += 256) {
    const int r = e / (NB / EPV), c = EPV * (e % (NB / EPV));
    cp_async16((sy + (r * kTrLd + c)).a, A + (size_t)r * ld + c);
  }
#pragma unroll 4
  for (int e = tid; e < NB * (NB / EPV); e += 256) {
    const int r = e / (NB / EPV), c = EPV * (e % (NB / EPV));
    if (c < (r & ~(PB - 1)))
      cp_async16((sl + (r * kTrLd + c)).a, D + (size_t)r * ld + c);
    else if (c <= (r | (PB - 1)))
      cp_async16((sx + (r * kTrXld + (c & (PB - 1)))).a, X + (size_t)r * NB + c);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  // warp w: row w / 2; half-warp (w & 1, lane / 16) is group g
  const int tx = tid & 15, g = (tid >> 4) & 3, row = tid >> 6;
  const Sh<T> y = sy + row * kTrLd, t = st + row * kTrXld;
  T acc[2] = {load_one(y + (g * PB + tx)), load_one(y + ((g + 4) * PB + tx))};
#pragma unroll
  for (int kb = 0; kb < kPBlocks; kb++) {
    if (g == (kb & 3)) {
      store_one(t + tx, acc[kb >> 2]);
      __syncwarp(0xffffu << (tid & 16));
      T v[4] = {(T)0, (T)0, (T)0, (T)0};
#pragma unroll
      for (int c = 0; c < PB; c += 4) {
        T x[4], q[4];
        load_row4(sx + ((kb * PB + tx) * kTrXld + c), x);
        load_row4(t + c, q);
#pragma unroll
        for (int m = 0; m < 4; m++) v[m] += q[m] * x[m];
      }
      store_one(y + (kb * PB + tx), (v[0] + v[1]) + (v[2] + v[3]));
    }
    __syncthreads();
    T q[PB];
    if (kb + 1 < kPBlocks) load_row16(y + kb * PB, q);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int b = g + 4 * h;
      if (b > kb) {
        const Sh<T> l = sl + ((b * PB + tx) * kTrLd + kb * PB);
        T v[4] = {(T)0, (T)0, (T)0, (T)0};
#pragma unroll
        for (int c = 0; c < PB; c += 4) {
          T w[4];
          load_row4(l + c, w);
#pragma unroll
          for (int m = 0; m < 4; m++) v[m] += q[c + m] * w[m];
        }
        acc[h] -= (v[0] + v[1]) + (v[2] + v[3]);
      }
    }
  }
  for (int e = tid; e < ROWS * (NB / 4); e += 256) {
    const int r = e / (NB / 4), c = 4 * (e % (NB / 4));
    T v[4];
    load_row4(sy + (r * kTrLd + c), v);
    store_row4(A + (size_t)r * ld + c, v[0], v[1], v[2], v[3]);
  }
  if (sizeof(T) == 4 && pack) {
    for (int e = tid; e < ROWS * 16; e += 256) {
      const int r = e >> 4, h = e & 15;
      float x[8];
#pragma unroll
      for (int q = 0; q < 8; q += 4) {
        T v[4];
        load_row4(sy + (r * kTrLd + 8 * h + q), v);
#pragma unroll
        for (int m = 0; m < 4; m++) x[q + m] = (float)v[m];
      }
      tc_pack_store8(pack, tc_pack_offset(rel0 + r, h), x);
    }
  }
}

// ---------------------------------------------------------------------------
// The inverse of every diagonal tile from the inverses of its diagonal
// 16-blocks (one CTA per tile, once per factorisation): X_ij = -X_ii sum_k
// L_ik X_kj for i > j.  Columns are independent: warp w owns 8 of them, from
// block column j = w / 2 on, and walks down the rows with L and its part of X
// in shared memory as packed lower 16-blocks.  The blocks of Linv above the
// diagonal are never written.  Bound by the chain of up to seven block rows:
// FP64 11.7 us (34.6 us with L read from global memory and FMAs).
constexpr int kInvBlk = PB * (PB + 4);
__device__ __forceinline__ int inv_blk(int i, int j) { return (i * (i + 1) / 2 + j) * kInvBlk; }
template <typename T>
constexpr size_t inv_tiles_smem() {
  return sizeof(T) * (size_t)(2 * (kPBlocks * (kPBlocks + 1) / 2) * kInvBlk + 16 * PB * (8 + 4));
}
// 16 x 8 product of one warp: C (row stride 12) = A B, A 16 x 16 (row stride 20),
// B 16 x 8 (row stride ldb), added to acc; out() stores it
__device__ __forceinline__ void inv_mac(float (&acc)[4], Sh<float> A, Sh<float> B, int ldb, int lane) {
  const int row = lane >> 1, col = 4 * (lane & 1);
#pragma unroll
  for (int c = 0; c < PB; c += 4) {
    float l[4];
    load_row4(A + (row * (PB + 4) + c), l);
#pragma unroll
    for (int m = 0; m < 4; m++) {
      float x[4];
      load_row4(B + ((c + m) * ldb + col), x);
#pragma unroll
      for (int q = 0; q < 4; q++) acc[q] += l[m] * x[q];
    }
  }
}
__device__ __forceinline__ void inv_out(const float (&acc)[4], float sign, Sh<float> C, int ldc, int lane) {
  store_row4(C + ((lane >> 1) * ldc + 4 * (lane & 1)), sign * acc[0], sign * acc[1], sign * acc[2], sign * acc[3]);
}
// FP64 on mma.m8n8k4: acc = rows (g, g + 8), columns (2 t, 2 t + 1)
__device__ __forceinline__ void inv_mac(double (&acc)[4], Sh<double> A, Sh<double> B, int ldb, int lane) {
  const int g = lane >> 2, t = lane & 3;
  double c0[2] = {acc[0], acc[1]}, c1[2] = {acc[2], acc[3]};
#pragma unroll
  for (int c = 0; c < PB; c += 4) {
    const double b = load_one(B + ((c + t) * ldb + g));
    mma_f64(c0, load_one(A + (g * (PB + 4) + c + t)), b);
    mma_f64(c1, load_one(A + ((g + 8) * (PB + 4) + c + t)), b);
  }
  acc[0] = c0[0]; acc[1] = c0[1]; acc[2] = c1[0]; acc[3] = c1[1];
}
__device__ __forceinline__ void inv_out(const double (&acc)[4], double sign, Sh<double> C, int ldc, int lane) {
  const int g = lane >> 2, t = lane & 3;
  store_two(C + (g * ldc + 2 * t), sign * acc[0], sign * acc[1]);
  store_two(C + ((g + 8) * ldc + 2 * t), sign * acc[2], sign * acc[3]);
}
template <typename T>
static __global__ void __launch_bounds__(512) inv_tiles_kernel(const T* __restrict__ S, int ld, T* __restrict__ Linv,
                                                              const int* __restrict__ active) {
  constexpr int EPV = 16 / (int)sizeof(T);
  extern __shared__ float4 smf4[];
  const Sh<T> sl{(uint32_t)__cvta_generic_to_shared(smf4)};
  const Sh<T> sx = sl + kPBlocks * (kPBlocks + 1) / 2 * kInvBlk;
  chain_start(S, active);
  if (active && !*active) return;
  const int k = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const Sh<T> st = sx + (kPBlocks * (kPBlocks + 1) / 2 * kInvBlk + w * PB * 12);
  const T* L = S + (size_t)k * NB * ld + (size_t)k * NB;
  T* X = Linv + (size_t)k * NB * NB;
#pragma unroll 4
  for (int e = threadIdx.x; e < NB * (NB / EPV); e += 512) {
    const int r = e / (NB / EPV), c = EPV * (e % (NB / EPV)), i = r / PB, j = c / PB;
    const int o = inv_blk(i, j) + (r % PB) * (PB + 4) + c % PB;
    if (j < i)
      cp_async16((sl + o).a, L + (size_t)r * ld + c);
    else if (j == i)
      cp_async16((sx + o).a, X + (size_t)r * NB + c);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int j = w >> 1, h = 8 * (w & 1);
#pragma unroll 1
  for (int i = j + 1; i < kPBlocks; i++) {
    T a[4] = {(T)0, (T)0, (T)0, (T)0}, b[4] = {(T)0, (T)0, (T)0, (T)0};
#pragma unroll 1
    for (int c = j; c < i; c++) inv_mac(a, sl + inv_blk(i, c), sx + (inv_blk(c, j) + h), PB + 4, lane);
    inv_out(a, (T)1, st, 12, lane);
    __syncwarp();
    inv_mac(b, sx + inv_blk(i, i), st, 12, lane);
    inv_out(b, (T)-1, sx + (inv_blk(i, j) + h), PB + 4, lane);
    __syncwarp();
  }
  __syncthreads();
#pragma unroll 2
  for (int e = threadIdx.x; e < NB * (NB / 4); e += 512) {
    const int r = e / (NB / 4), c = 4 * (e % (NB / 4)), i = r / PB, jj = c / PB;
    if (jj >= i) continue;
    T v[4];
    load_row4(sx + (inv_blk(i, jj) + (r % PB) * (PB + 4) + c % PB), v);
    store_row4(X + (size_t)r * NB + c, v[0], v[1], v[2], v[3]);
  }
}

// ---------------------------------------------------------------------------
// The trailing update of the next diagonal tile, on the factorisation's
// critical path (FP32): A_tt -= sum_p L_t,p L_t,p' over panels p in [p0, p0 +
// np), by 128 / RPC CTAs of 256 threads, CTA c owning an RPC-row slice (RPC =
// kChainRows below).  Both operands stay row-major in shared memory (row stride
// 132 floats) and are read as float4 along K.
// Rows per CTA, LM it/s at 1,500 9-parameter cameras with identical results:
// 16 rows (8 CTAs) 93.1, 8 rows 94.6, 4 rows 95.6 -- every CTA stages the
// whole panel, so more CTAs cut each one's FMAs, not its copies.
constexpr int kChainRows = 4;
static_assert(kChainRows == 16 || kChainRows == 8 || kChainRows == 4, "chain kernels: 4, 8 or 16 rows per CTA");
constexpr int kSlLd = NB + 4;                // 132
constexpr size_t kDiagUpdSmem = sizeof(float) * (size_t)NB * kSlLd;                 // 67,584 B per panel

// acc[h][m] += sum_l a_h[l] b[16 w + (lane & 3) + 4 m][l], l < NB
// A CTA of the chain kernels owns RPC rows of a 128 x 128 result as RPC / 2
// row pairs (a0, a1); warp w owns columns 16 w .. 16 w + 15.  Lane l: pair
// l / CG, columns 16 w + l % CG + CG m (m < 16 / CG), CG = 32 / (RPC / 2).
// Each output sums over l = 0 .. 127 in order (x, y, z, w of every float4).
template <int RPC>
__device__ inline void slice_mma(const float* __restrict__ a0, const float* __restrict__ a1,
                                 const float* __restrict__ sb, int lane, int w, float acc[2][16 / (64 / RPC)]) {
  constexpr int CG = 64 / RPC, M = 16 / CG;
  const float* pb = sb + (16 * w + (lane % CG)) * kSlLd;
#pragma unroll 4
  for (int l = 0; l < NB; l += 4) {
    float4 a[2], b[M];
    a[0] = *reinterpret_cast<const float4*>(a0 + l);
    a[1] = *reinterpret_cast<const float4*>(a1 + l);
#pragma unroll
    for (int m = 0; m < M; m++) b[m] = *reinterpret_cast<const float4*>(pb + CG * m * kSlLd + l);
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int m = 0; m < M; m++) {
        acc[h][m] = fmaf(a[h].x, b[m].x, acc[h][m]);
        acc[h][m] = fmaf(a[h].y, b[m].y, acc[h][m]);
        acc[h][m] = fmaf(a[h].z, b[m].z, acc[h][m]);
        acc[h][m] = fmaf(a[h].w, b[m].w, acc[h][m]);
      }
  }
}

// rows x 128 FP32 columns (row stride ld) into shared memory (stride kSlLd)
__device__ inline void stage_rows_f32(const float* __restrict__ src, size_t ld, int rows, float* __restrict__ dst,
                                      int tid) {
  for (int e = tid; e < rows * NB / 4; e += 256) {
    const int r = e >> 5, c4 = e & 31;
    cp_async16(dst + r * kSlLd + 4 * c4, src + (size_t)r * ld + 4 * c4);
  }
}

// Slice c of RPC rows owns tile rows P c .. P c + P - 1 and 127 - P c - P + 1
// .. 127 - P c (P = RPC / 2): equal shares of the lower triangle.  A_tt's
// lower triangle only is written.  np <= 4 panels through two staging
// buffers (min(np, 2) x kDiagUpdSmem bytes of shared memory): panel p + 2 is
// copied in while panel p + 1 is applied.
constexpr int kDiagUpdMaxPanels = 4;
template <int RPC>
__device__ inline int diag_slice_row(int c, int p) {
  constexpr int P = RPC / 2;
  return p < P ? P * c + p : NB - 1 - P * c - (p - P);
}

template <int RPC>
static __global__ void __launch_bounds__(256) diag_update_kernel(float* __restrict__ S, int ld, int t, int p0, int np,
                                                                 const int* __restrict__ active) {
  constexpr int P = RPC / 2, CG = 32 / P, M = 16 / CG;
  extern __shared__ float4 smf4[];
  float* sm = reinterpret_cast<float*>(smf4);  // L_t,p (all 128 rows) per panel
  chain_release();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, c = blockIdx.x;
  const int ra = diag_slice_row<RPC>(c, lane / CG), rb = diag_slice_row<RPC>(c, P + lane / CG);
  const float* T0 = S + (size_t)t * NB * ld + (size_t)p0 * NB;
  // all panels but the last were finished before the stream's preceding
  // kernel (the row-tile TRSM of the last one) started: fetch the first while
  // that kernel runs
  if (np > 1) stage_rows_f32(T0, ld, NB, sm, tid);
  cp_async_commit();
  chain_wait();
  if (active && !*active) {
    cp_async_wait<0>();
    return;
  }
  if (np > 1)
    stage_rows_f32(T0 + NB, ld, NB, sm + NB * kSlLd, tid);
  else
    stage_rows_f32(T0, ld, NB, sm, tid);
  cp_async_commit();
  float acc[2][M] = {};
  for (int p = 0; p < np; p++) {
    // committed groups so far: panels 0 .. min(p + 1, np - 1) (one empty
    // group when np == 1); panel p is complete once at most the newest is
    // still in flight
    if (p + 1 < np)
      cp_async_wait<1>();
    else
      cp_async_wait<0>();
    __syncthreads();
    const float* sb = sm + (p & 1) * NB * kSlLd;
    slice_mma<RPC>(sb + ra * kSlLd, sb + rb * kSlLd, sb, lane, w, acc);
    __syncthreads();  // every warp is done with buffer p & 1
    if (p + 2 < np) {
      stage_rows_f32(T0 + (size_t)(p + 2) * NB, ld, NB, sm + (p & 1) * NB * kSlLd, tid);
      cp_async_commit();
    }
  }
  float* D = S + (size_t)t * NB * ld + (size_t)t * NB;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int r = h ? rb : ra;
#pragma unroll
    for (int m = 0; m < M; m++) {
      const int i = 16 * w + (lane % CG) + CG * m;
      if (i <= r) D[(size_t)r * ld + i] -= acc[h][m];
    }
  }
}

// ---------------------------------------------------------------------------
// CUDA-core trailing update (FP32 or FP64), one CTA per 128 x 128 lower tile:
// C_IJ -= X_I X_J' with X = columns [k NB, (k+1) NB).  The reference of the
// tensor-core kernel's self-test.
template <typename T>
__device__ inline void syrk_cc_tile(T* __restrict__ S, int ld, int k, int gI, int gJ);

template <typename T>
static __global__ void __launch_bounds__(256) syrk_cc_kernel(T* __restrict__ S, int ld, int k, int t0, int nt,
                                                      const int* __restrict__ active) {
  if (active && !*active) return;
  const int q = blockIdx.x;
  int I = (int)((sqrt(8.0 * q + 1.0) - 1.0) * 0.5);
  while ((I + 1) * (I + 2) / 2 <= q) I++;
  while (I * (I + 1) / 2 > q) I--;
  const int J = q - I * (I + 1) / 2;
  syrk_cc_tile<T>(S, ld, k, t0 + I, t0 + J);
}

template <typename T>
__device__ inline void syrk_cc_tile(T* __restrict__ S, int ld, int k, int gI, int gJ) {
  constexpr int KC = 16;
  __shared__ T As[KC][NB + 4];
  __shared__ T Bs[KC][NB + 4];
  const int I = gI, J = gJ;
  const int rA = gI * NB, rB = gJ * NB, kc = k * NB;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  T acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) acc[i][j] = (T)0;
  for (int kk = 0; kk < NB; kk += KC) {
    for (int i = threadIdx.x; i < NB * KC; i += 256) {
      const int r = i / KC, c = i - r * KC;
      As[c][r] = S[(size_t)(rA + r) * ld + kc + kk + c];
      Bs[c][r] = S[(size_t)(rB + r) * ld + kc + kk + c];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < KC; c++) {
      T a[8], b[8];
#pragma unroll
      for (int i = 0; i < 8; i++) a[i] = As[c][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 8; j++) b[j] = Bs[c][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] += a[i] * b[j];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int r = ty + 16 * i;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int c = tx + 16 * j;
      if (I != J || c <= r) S[(size_t)(rA + r) * ld + rB + c] -= acc[i][j];
    }
  }
}

// The same for the FP64 factorisation, one panel: A_tt -= L_tp L_tp' on the lower
// triangle, a CTA per 16 x 16 block (36), its four warps a quarter of K each on
// the FP64 tensor cores.  Bound by its two copies (L2 latency).  With it and the
// row-tile TRSM the FP64 chain no longer waits for the rest of the panel: 55 us per
// panel (factor 21, TRSM of all rows 16, cuBLAS column update 12, gaps) before.
constexpr int kDiag64Ctas = (NB / 16) * (NB / 16 + 1) / 2;
static __global__ void __launch_bounds__(128) diag_update64_kernel(double* __restrict__ S, int ld, int t, int p,
                                                                   const int* __restrict__ active) {
  constexpr int LDA = NB + 4;
  __shared__ __align__(16) double sa[2][16 * LDA];
  chain_release();
  chain_wait();
  if (active && !*active) return;
  int bi = 0, bj = blockIdx.x;  // block row, block column
  while (bj > bi) bj -= ++bi;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* L = S + (size_t)t * NB * ld + (size_t)p * NB;
  for (int e = tid; e < 16 * (NB / 2); e += 128) {
    const int r = e / (NB / 2), c = 2 * (e % (NB / 2));
    cp_async16(&sa[0][r * LDA + c], L + (size_t)(16 * bi + r) * ld + c);
    if (bi != bj) cp_async16(&sa[1][r * LDA + c], L + (size_t)(16 * bj + r) * ld + c);
  }
  cp_async_commit();
  const int r = tid >> 3, c = 2 * (tid & 7);  // this thread's two entries of the block
  double2* C = reinterpret_cast<double2*>(S + (size_t)(t * NB + 16 * bi + r) * ld + (size_t)t * NB + 16 * bj + c);
  double2 v = *C;
  cp_async_wait<0>();
  __syncthreads();
  const int g = lane >> 2, q = lane & 3;
  const double* A = sa[0] + g * LDA + q;
  const double* B = sa[bi != bj] + g * LDA + q;
  double acc[2][2][2] = {};
#pragma unroll
  for (int k = 0; k < NB / 4; k += 4) {
    const int kk = warp * (NB / 4) + k;
    double a[2], b[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      a[i] = A[8 * i * LDA + kk];
      b[i] = B[8 * i * LDA + kk];
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) mma_f64(acc[i][j], a[i], b[j]);
  }
  __syncthreads();
  double* part = sa[0] + warp * 256;
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int m = 0; m < 2; m++) part[(8 * i + g) * 16 + 8 * j + 2 * q + m] = acc[i][j][m];
  __syncthreads();
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int w = 0; w < 4; w++) {
    s0 += sa[0][w * 256 + r * 16 + c];
    s1 += sa[0][w * 256 + r * 16 + c + 1];
  }
  if (bi != bj || c <= r) v.x -= s0;  // above the diagonal of the tile: as it was
  if (bi != bj || c + 1 <= r) v.y -= s1;
  *C = v;
}

// ---------------------------------------------------------------------------
// Triangular solves with the tile inverses, a chain of one hop per 128-row tile.
// kSolveCtas CTAs per tile, 32 rows (backward: columns) each: a hop is bounded by
// the product with a 128 x 128 matrix, which in FP64 arithmetic on one SM takes
// 1 us (16 conversions and 38 FMAs per clock), and by the way of the result to
// the next tile.  A CTA waits for earlier tiles (forward; later ones backward) and for
// the other CTAs of its own tile.  CTA r of each kSolveCtas consecutive ones takes its
// tile from ticket r, so that tiles are handed out in order, and every wait ends if
// the CTAs of a tile do get onto the chip, however many other solves share it:
// - in clusters of kSolveCtas they are there together (with m clusters placed, the
//   tickets hand out tiles 0 .. m - 1, each complete);
// - without, a launch holds at most kSolveCtas - 1 CTAs that wait for an unplaced one
//   (those of complete tiles end, by induction over the tiles), and the device at most
//   kMaxGrids launches: where the chip has room for many more CTAs than these, the
//   unplaced ones find it.
// solve_cluster takes clusters unless there is room for twice as many: systems of one
// tile (FP32 two) stage less and go without.  A cluster launch costs the host 1.4 us (scan
// alignment, one tile, 943 -> 959 us a solve).  Each wait is also bounded.
//
// A value is passed on with the tag of its solve as one 16-byte store and load:
// the reader that finds the tag has the value, without barrier, release, flag and
// second load.  A tag is never used twice (a call's number and the solve within
// it), so the packets are not cleared between calls.
//
// Per solve, one CTA per tile with flags -> now: 15 tiles FP32 33 -> 21.5 us, FP64
// 42 -> 22 us, band of 47 tiles 92 -> 53 us, 106 tiles 240 -> 205 us (1.4 us per
// hop at 15 and 31 tiles, of which 0.7 us are the packet's way through L2; 1.9 us at 106
// tiles, where a CTA also streams L's rows; three hop matrices instead of two
// change nothing).
constexpr int kSolveCtas = 4, SVR = NB / kSolveCtas, SVT = 128;
// rank of the CTA among the kSolveCtas consecutive ones of a cluster
__device__ __forceinline__ int solve_rank() { return (int)(blockIdx.x % kSolveCtas); }
static_assert(SVT == NB && SVR == 8 * (SVT / 32), "a thread fetches one row, a warp finishes eight");

__device__ inline void put_packet(ulonglong2* p, double v, unsigned long long tag) {
  asm volatile("{\n.reg .b128 t;\nmov.b128 t, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ ulonglong2 look_packet(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("{\n.reg .b128 t;\nld.relaxed.gpu.global.b128 t, [%2];\nmov.b128 {%0, %1}, t;\n}\n"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}

// The values of a tile in shared memory, read as double2 (load4)
struct __align__(16) TileValues {
  double v[NB];
};
static_assert(alignof(TileValues) == 16 && sizeof(TileValues) % 16 == 0, "load4 reads 16-byte pieces");

// Fetches the 128 values at pk into dst (shared), one per thread; every thread of
// the CTA calls it.  `seen`: what a look at the thread's packet gave earlier.
// False after a wait that ran out.
__device__ inline bool fetch_tile(const ulonglong2* __restrict__ pk, ulonglong2 seen, unsigned long long tag,
                                  TileValues& dst, int* __restrict__ status, long long limit) {
  long long it = 0;
  while (seen.y != tag && ++it <= limit) {
    if (it > 4096) __nanosleep(100);
    seen = look_packet(pk + threadIdx.x);
  }
  const bool bad = seen.y != tag;
  if (bad) atomicOr(status, ST_SPIN_TIMEOUT);
  dst.v[threadIdx.x] = __longlong_as_double(seen.x);
  return !__syncthreads_or(bad);
}

// Start of a call that solves without forming S: clears the solves' tickets (the
// first forward solve hands out tiles from `first` on) and numbers the call.
static __global__ void solve_begin_kernel(int* tickets, int n, int first, unsigned long long* call) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) tickets[i] = i < kSolveCtas ? first : 0;
  if (threadIdx.x == 0) (*call)++;
}

template <typename T>
__device__ inline void load4(const T* p, double* v) {
  if (sizeof(T) == 4) {
    const float4 f = *reinterpret_cast<const float4*>(p);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
    const double2 a = *reinterpret_cast<const double2*>(p);
    const double2 b = *reinterpret_cast<const double2*>(p + 2);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
}

constexpr int SV = 512;
// Four consecutive entries of an L row in the storage type (kept raw in
// registers, widened to FP64 at the product).
template <typename T>
struct Row4;
template <>
struct Row4<float> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) { v = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ double dot(const double* y) const {
    return (double)v.x * y[0] + (double)v.y * y[1] + (double)v.z * y[2] + (double)v.w * y[3];
  }
  __device__ __forceinline__ double at(int q) const {
    return q == 0 ? (double)v.x : q == 1 ? (double)v.y : q == 2 ? (double)v.z : (double)v.w;
  }
};
template <>
struct Row4<double> {
  double2 a, b;
  __device__ __forceinline__ void load(const double* p) {
    a = reinterpret_cast<const double2*>(p)[0];
    b = reinterpret_cast<const double2*>(p)[1];
  }
  __device__ __forceinline__ double dot(const double* y) const { return a.x * y[0] + a.y * y[1] + b.x * y[2] + b.y * y[3]; }
  __device__ __forceinline__ double at(int q) const { return q == 0 ? a.x : q == 1 ? a.y : q == 2 ? b.x : b.y; }
};

// Sums over the 32 lanes of eight per-lane values v[0..7] by recursive
// halving: at offsets 16, 8 and 4 each lane keeps half of its values and adds
// its partner's copy of them, then two butterfly steps finish.  Lane l ends
// with the full sum of v[4 b4 + 2 b3 + b2] (b4, b3, b2 = bits 4, 3, 2 of l;
// `reduce8_row` gives that index).  9 exchanges, 5 dependent levels; the
// order of the additions is fixed by the lane numbers.
__device__ __forceinline__ int reduce8_row(int lane) {
  return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
}
__device__ __forceinline__ double reduce8(const double (&v)[8], int lane) {
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
  double a[4], b[2];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const double send = h4 ? v[q] : v[4 + q];
    a[q] = (h4 ? v[4 + q] : v[q]) + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const double send = h3 ? a[q] : a[2 + q];
    b[q] = (h3 ? a[2 + q] : a[q]) + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  double c = (h2 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h2 ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}

// The hop matrices of the solves, formed once per factorisation.  For the
// d-th neighbour (d = 1 .. kHopDepth):
//   M_d,I = Linv_I L_I,I-d                 (forward, I >= d)
//   Q_d,I = (L_I+d,I Linv_I)'              (backward, I + d < ntiles)
// at hop + ((dir kHopDepth + d - 1) ntiles + I) NB^2, dir 0 forward / 1
// backward.  With them y_I = c_I - sum_d M_d,I y_I-d, where c_I = Linv_I (b_I
// - sum_{J < I - kHopDepth} L_IJ y_J) needs only tiles published kHopDepth
// hops earlier, and likewise x_I = c'_I - sum_d Q_d,I x_I+d: after the wait
// for its neighbour a solve CTA applies one matrix that it has at hand.  Products
// in T (FP32 for the mixed factor, FP64 for the FP64 one).  A tile L outside the
// envelope is zero, and so is its hop matrix.  Grid (ntiles - 1, 2 kHopDepth, 4):
// a 64 x 64 block per CTA, its operands staged in one go: with one CTA per
// product the chip was idle (15 tiles: 54 CTAs) and every k step waited for memory
// (15 tiles FP32 30 -> 11 us, FP64 45 -> 13 us, 106 tiles 78 -> 44 us).
constexpr int kHopDepth = 2;

// The eight rows x four columns of a matrix that a thread of a solve applies, in
// shared memory: copied and read by that thread alone (no barrier, no conflict).
template <typename T>
struct OwnBlock {
  static constexpr int kPieces = sizeof(T) / 4, kBytes = 8 * kPieces * SVT * 16;  // 16-byte pieces per row
  char* p;
  __device__ OwnBlock(void* smem, int i) : p((char*)smem + i * kBytes + threadIdx.x * 16) {}
  __device__ __forceinline__ void stage(const T* src, size_t row_step) const {
#pragma unroll
    for (int i = 0; i < 8 * kPieces; i++)
      cp_async16(p + i * SVT * 16, src + (i / kPieces) * row_step + (i % kPieces) * (16 / sizeof(T)));
  }
  __device__ __forceinline__ void row(int rr, double* v) const {
    if (sizeof(T) == 4) {
      const float4 f = *reinterpret_cast<const float4*>(p + rr * SVT * 16);
      v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
      const double2 a = *reinterpret_cast<const double2*>(p + 2 * rr * SVT * 16);
      const double2 b = *reinterpret_cast<const double2*>(p + (2 * rr + 1) * SVT * 16);
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
  }
  // rows in the lanes' eight values, summed over the warp: the value of row
  // reduce8_row(lane)
  __device__ __forceinline__ double times(const double* x4, int lane) const {
    double q[8];
#pragma unroll
    for (int rr = 0; rr < 8; rr++) {
      double v[4];
      row(rr, v);
      q[rr] = v[0] * x4[0] + v[1] * x4[1] + v[2] * x4[2] + v[3] * x4[3];
    }
    return reduce8(q, lane);
  }
};
template <typename T>
constexpr size_t trsv_smem(int ntiles) {  // Linv_I and the hop matrices
  return (size_t)(ntiles > kHopDepth ? 1 + kHopDepth : ntiles) * OwnBlock<T>::kBytes;
}
constexpr int kMaxGrids = 128;  // grids resident on a device at once, at most
// CTAs per cluster of a solve where `slots` of its CTAs fit on the chip
inline int solve_cluster(int slots) { return slots > 2 * (kSolveCtas - 1) * kMaxGrids ? 1 : kSolveCtas; }
constexpr int kHopB = 64, kHopLd = kHopB + 4;  // output block, row length of a staged block
template <typename T>
constexpr size_t hop_smem() {
  return 4 * sizeof(T) * kHopB * kHopLd;
}
template <typename T>
static __global__ void __launch_bounds__(256) hop_mat_kernel(const T* __restrict__ S, int ld, int ntiles,
                                                             const T* __restrict__ Linv, T* __restrict__ hop,
                                                             const int* __restrict__ active) {
  extern __shared__ float4 hop_stage[];
  T* sm = reinterpret_cast<T*>(hop_stage);  // [k half][A, B][kHopB][kHopLd]
  chain_start(S, Linv, active);
  if (active && !*active) return;
  const bool fwd = blockIdx.y < kHopDepth;
  const int d = (int)(blockIdx.y % kHopDepth) + 1;
  // forward: I = d + x, tile (I, I - d); backward: I = x, tile (I + d, I)
  const int I = fwd ? d + (int)blockIdx.x : (int)blockIdx.x;
  if ((fwd && I >= ntiles) || (!fwd && I + d >= ntiles)) return;
  const int br = (blockIdx.z >> 1) * kHopB, bc = (blockIdx.z & 1) * kHopB;  // first row, column of the product
  const T* Lt = fwd ? S + (size_t)I * NB * ld + (size_t)(I - d) * NB : S + (size_t)(I + d) * NB * ld + (size_t)I * NB;
  const T* A = fwd ? Linv + (size_t)I * NB * NB : Lt;
  const int lda = fwd ? NB : ld;
  const T* B = fwd ? Lt : Linv + (size_t)I * NB * NB;
  const int ldb = fwd ? ld : NB;
  // Linv is lower triangular: rows of A below 64 end at k = 64 (forward), columns
  // of B from 64 on start there (backward)
  const int h0 = !fwd && bc ? 1 : 0, h1 = fwd && !br ? 1 : 2;
  T* out = hop + ((size_t)blockIdx.y * ntiles + I) * NB * NB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int V = 16 / (int)sizeof(T), PV = kHopB / V;  // elements per copy, copies per row
#pragma unroll
  for (int h = 0; h < 2; h++) {
    if (h >= h0 && h < h1) {
      T* As = sm + (2 * h) * kHopB * kHopLd;
      T* Bs = As + kHopB * kHopLd;
      for (int e = tid; e < kHopB * PV; e += 256) {
        const int r = e / PV, c = (e % PV) * V;
        cp_async16(As + r * kHopLd + c, A + (size_t)(br + r) * lda + h * kHopB + c);
        cp_async16(Bs + r * kHopLd + c, B + (size_t)(h * kHopB + r) * ldb + bc + c);
      }
    }
    cp_async_commit();
  }
  auto staged = [&](int h) {
    if (h == 0)
      cp_async_wait<1>();
    else
      cp_async_wait<0>();
    __syncthreads();
  };
  if constexpr (sizeof(T) == 8) {
    // warp: 32 rows x 16 columns, tensor-core FP64
    const int wr = (warp >> 2) * 32, wc = (warp & 3) * 16, g = lane >> 2, t = lane & 3;
    double acc[4][2][2] = {};
    for (int h = h0; h < h1; h++) {
      staged(h);
      const T* As = sm + (2 * h) * kHopB * kHopLd + (wr + g) * kHopLd + t;
      const T* Bs = sm + (2 * h + 1) * kHopB * kHopLd + t * kHopLd + wc + g;
#pragma unroll 4
      for (int k = 0; k < kHopB; k += 4) {
        double a[4], b[2];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = As[8 * i * kHopLd + k];
#pragma unroll
        for (int j = 0; j < 2; j++) b[j] = Bs[k * kHopLd + 8 * j];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 2; j++) mma_f64(acc[i][j], a[i], b[j]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const int r = wr + 8 * i + g, c = wc + 8 * j + 2 * t + q;
          sm[fwd ? r * kHopLd + c : c * kHopLd + r] = acc[i][j][q];
        }
  } else {
    // thread: 4 rows x 4 columns
    const int tx = tid & 15, ty = tid >> 4;
    float acc[4][4] = {};
    for (int h = h0; h < h1; h++) {
      staged(h);
      const float4* As = reinterpret_cast<const float4*>(sm + (2 * h) * kHopB * kHopLd);
      const float4* Bs = reinterpret_cast<const float4*>(sm + (2 * h + 1) * kHopB * kHopLd);
#pragma unroll 4
      for (int k = 0; k < kHopB; k += 4) {
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = As[((ty + 16 * i) * kHopLd + k) / 4];
#pragma unroll
        for (int q = 0; q < 4; q++) b[q] = Bs[(k + q) * (kHopLd / 4) + tx];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float av[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
          for (int q = 0; q < 4; q++) {
            acc[i][0] += av[q] * b[q].x;
            acc[i][1] += av[q] * b[q].y;
            acc[i][2] += av[q] * b[q].z;
            acc[i][3] += av[q] * b[q].w;
          }
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int r = ty + 16 * i, c = 4 * tx + j;
        sm[fwd ? r * kHopLd + c : c * kHopLd + r] = acc[i][j];
      }
  }
  // rows of the result (backward: transposed), whole lines
  __syncthreads();
  out += fwd ? (size_t)br * NB + bc : (size_t)bc * NB + br;
  for (int e = tid; e < kHopB * PV; e += 256) {
    const int r = e / PV, c = (e % PV) * V;
    *reinterpret_cast<float4*>(out + (size_t)r * NB + c) = *reinterpret_cast<const float4*>(sm + r * kHopLd + c);
  }
}

// Forward solve L y = b.  A CTA of tile I streams the tiles J < I - kHopDepth of
// its rows as they are published, passes b_I - partial to the CTAs of its tile,
// subtracts M_d,I y_I-d for d = kHopDepth .. 2, adds c_I = Linv_I (b_I - partial)
// and ends with M_1,I y_I-1.  b = the vector b less, if given, the nch partials
// `part` of a refinement residual.  Warp w, lane l: rows 8 w .. 8 w + 7 of the
// CTA's, columns 4 l .. 4 l + 3.  pk: 2 x 128 ntiles packets (y, b - partial).
template <typename T>
static __global__ void __launch_bounds__(SVT) trsv_fwd_kernel(
    const T* __restrict__ L, int ld, int ntiles, const T* __restrict__ Linv, const T* __restrict__ hop,
    const double* __restrict__ b, const double* __restrict__ part, int nch, double* __restrict__ y,
    int* __restrict__ ticket, ulonglong2* __restrict__ pk, const unsigned long long* __restrict__ call, int sub,
    int* __restrict__ status, long long spin_limit, const int* __restrict__ env, const int* __restrict__ active) {
  extern __shared__ float4 own4[];
  __shared__ TileValues got[2];
  __shared__ int t_s;
  chain_start(L, Linv, hop, b, part, call, active);
  if (active && !*active) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long tag = (*call << 32) | (unsigned)sub;
  if (tid == 0) t_s = atomicAdd(ticket + solve_rank(), 1);
  __syncthreads();
  const int I = t_s, r0 = solve_rank() * SVR + warp * 8;
  const size_t own = (size_t)r0 * NB + 4 * lane;
  OwnBlock<T>(own4, 0).stage(Linv + (size_t)I * NB * NB + own, NB);
#pragma unroll
  for (int d = 1; d <= kHopDepth; d++)
    if (I >= d) OwnBlock<T>(own4, d).stage(hop + ((size_t)(d - 1) * ntiles + I) * NB * NB + own, NB);
  cp_async_commit();
  // the right-hand side of the row this lane finishes
  const size_t row = (size_t)I * NB + r0 + reduce8_row(lane);
  double b_own = b[row];
  if (part)
    for (int c = 0; c < nch; c++) b_own -= part[(size_t)c * ntiles * NB + row];
  // with an envelope, the tiles of row I before its first nonzero are zero
  const int J0 = env ? env[I] : 0;
  const int Jend = I - kHopDepth;  // tiles [J0, Jend) are streamed, the last kHopDepth go through M_d,I
  int par = 0;
  double x4[4];
  auto fetch = [&](const ulonglong2* p, ulonglong2 seen) -> bool {  // uniform
    const bool ok = fetch_tile(p, seen, tag, got[par], status, spin_limit);
    load4(got[par].v + 4 * lane, x4);
    par ^= 1;  // the other buffer is written only after the next barrier
    if (!ok) cp_async_wait<0>();  // the CTA gives up: no copy stays in flight
    return ok;
  };
  const ulonglong2 none = make_ulonglong2(0, 0);  // call numbers start at 1
  double dots[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (J0 < Jend) {
    const T* Lrow = L + (size_t)(I * NB + r0) * ld + 4 * lane;
    Row4<T> cur[8];
    ulonglong2 seen = none;
    for (int J = J0; J < Jend; J++) {
#pragma unroll
      for (int rr = 0; rr < 8; rr++) cur[rr].load(Lrow + (size_t)rr * ld + (size_t)J * NB);
      const ulonglong2* p = pk + (size_t)J * NB;
      const ulonglong2 now = seen;
      if (J + 1 < Jend) seen = look_packet(p + NB + tid);
      if (!fetch(p, now)) return;
#pragma unroll
      for (int rr = 0; rr < 8; rr++) dots[rr] += cur[rr].dot(x4);
    }
  }
  ulonglong2* pa = pk + (size_t)(ntiles + I) * NB;
  {
    const double sr = reduce8(dots, lane);
    if ((lane & 3) == 0) put_packet(pk + (size_t)ntiles * NB + row, b_own - sr, tag);
  }
  cp_async_wait<0>();
  double yr = 0.0;
#pragma unroll
  for (int d = kHopDepth; d >= 1; d--) {
    if (d == 1) {
      if (!fetch(pa, none)) return;
      yr = OwnBlock<T>(own4, 0).times(x4, lane) - yr;
    }
    const int J = I - d;
    if (J < 0 || J < J0) continue;  // outside the matrix or the envelope (uniform)
    if (!fetch(pk + (size_t)J * NB, none)) return;
    const double h = OwnBlock<T>(own4, d).times(x4, lane);
    yr = d > 1 ? yr + h : yr - h;
  }
  if ((lane & 3) == 0) {
    put_packet(pk + row, yr, tag);
    y[row] = yr;
  }
}

// Backward solve L' x = y.  A CTA of tile I streams the tiles J > I + kHopDepth of
// its columns (rows of L_J,I), passes y_I - partial to the CTAs of its tile and
// goes on as the forward solve with Q_d,I x_I+d (Q_d,I row-major: row c is column
// c of L_I+d,I Linv_I) and c'_I = Linv_I' (y_I - partial).  For L_J,I and Linv_I a
// thread holds rows 32 w + (l >> 3) + 4 i, columns 4 (l & 7) .. + 3 of the CTA's.
// `sum`, if given, gets x added (a refinement step).
template <typename T>
static __global__ void __launch_bounds__(SVT) trsv_bwd_kernel(
    const T* __restrict__ L, int ld, int ntiles, const T* __restrict__ Linv, const T* __restrict__ hop,
    const double* __restrict__ yv, double* __restrict__ x, double* __restrict__ sum, int* __restrict__ ticket,
    ulonglong2* __restrict__ pk, const unsigned long long* __restrict__ call, int sub, int* __restrict__ status,
    long long spin_limit, const int* __restrict__ env, const int* __restrict__ active) {
  extern __shared__ float4 own4[];
  __shared__ TileValues got[2];
  __shared__ double red[SVT / 32][SVR];
  __shared__ int t_s;
  chain_start(L, Linv, hop, yv, call, active);
  if (active && !*active) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned long long tag = (*call << 32) | (unsigned)sub;
  if (tid == 0) t_s = atomicAdd(ticket + solve_rank(), 1);
  __syncthreads();
  const int I = ntiles - 1 - t_s, q0 = solve_rank() * SVR;
  const int tr = 32 * warp + (lane >> 3), tc = q0 + 4 * (lane & 7);  // transposed blocks: first row, first column
  OwnBlock<T>(own4, 0).stage(Linv + (size_t)I * NB * NB + (size_t)tr * NB + tc, 4 * NB);
#pragma unroll
  for (int d = 1; d <= kHopDepth; d++)
    if (I + d < ntiles)
      OwnBlock<T>(own4, d).stage(
          hop + ((size_t)(kHopDepth + d - 1) * ntiles + I) * NB * NB + (size_t)(q0 + warp * 8) * NB + 4 * lane, NB);
  cp_async_commit();
  const double y_own = tid < SVR ? yv[(size_t)I * NB + q0 + tid] : 0.0;
  // with an envelope, the tiles of column I past its last nonzero are zero
  const int J1 = env ? env[ntiles + I] : ntiles - 1;
  const int Jend = I + kHopDepth;  // tiles (Jend, J1] are streamed, the nearest kHopDepth go through Q_d,I
  int par = 0;
  const double* v = nullptr;
  auto fetch = [&](const ulonglong2* p, ulonglong2 seen) -> bool {  // uniform
    const bool ok = fetch_tile(p, seen, tag, got[par], status, spin_limit);
    v = got[par].v;
    par ^= 1;
    if (!ok) cp_async_wait<0>();  // the CTA gives up: no copy stays in flight
    return ok;
  };
  // the sum over a column's rows: the lanes of a column, then the warps (thread < SVR)
  auto column_sum = [&](double (&p)[4]) -> double {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      p[q] += __shfl_xor_sync(0xffffffffu, p[q], 8);
      p[q] += __shfl_xor_sync(0xffffffffu, p[q], 16);
    }
    if (lane < 8) {
#pragma unroll
      for (int q = 0; q < 4; q++) red[warp][4 * lane + q] = p[q];
    }
    __syncthreads();
    double s = 0.0;
    if (tid < SVR) {
#pragma unroll
      for (int w = 0; w < SVT / 32; w++) s += red[w][tid];
    }
    return s;
  };
  const ulonglong2 none = make_ulonglong2(0, 0);  // call numbers start at 1
  double part[4] = {0, 0, 0, 0};
  if (J1 > Jend) {
    const T* Lcol = L + (size_t)tr * ld + (size_t)I * NB + tc;  // + J NB ld: tile (J, I)
    Row4<T> cur[8];
    ulonglong2 seen = none;
    for (int J = J1; J > Jend; J--) {
#pragma unroll
      for (int rr = 0; rr < 8; rr++) cur[rr].load(Lcol + (size_t)(J * NB + 4 * rr) * ld);
      const ulonglong2* p = pk + (size_t)J * NB;
      const ulonglong2 now = seen;
      if (J - 1 > Jend) seen = look_packet(p - NB + tid);
      if (!fetch(p, now)) return;
#pragma unroll
      for (int rr = 0; rr < 8; rr++) {
        const double xr = v[tr + 4 * rr];
#pragma unroll
        for (int q = 0; q < 4; q++) part[q] += cur[rr].at(q) * xr;
      }
    }
  }
  {
    const double s = column_sum(part);
    if (tid < SVR) put_packet(pk + (size_t)(ntiles + I) * NB + q0 + tid, y_own - s, tag);
  }
  cp_async_wait<0>();
  const int rsel = warp * 8 + reduce8_row(lane);
  double xr = 0.0;
#pragma unroll
  for (int d = kHopDepth; d >= 1; d--) {
    if (d == 1) {
      if (!fetch(pk + (size_t)(ntiles + I) * NB, none)) return;
      double p2[4] = {0, 0, 0, 0};
#pragma unroll
      for (int rr = 0; rr < 8; rr++) {
        const double ar = v[tr + 4 * rr];
        double lv[4];
        OwnBlock<T>(own4, 0).row(rr, lv);
#pragma unroll
        for (int q = 0; q < 4; q++) p2[q] += lv[q] * ar;
      }
      const double s = column_sum(p2);  // red: every thread has passed fetch's barrier since it was read
      if (warp == 0) red[0][lane] = s;  // thread i alone reads and writes red[0][i] from here
      __syncthreads();
      xr = red[0][rsel] - xr;
    }
    const int J = I + d;
    if (J >= ntiles || J > J1) continue;  // outside the matrix or the envelope (uniform)
    if (!fetch(pk + (size_t)J * NB, none)) return;
    double x4[4];
    load4(v + 4 * lane, x4);
    const double h = OwnBlock<T>(own4, d).times(x4, lane);
    xr = d > 1 ? xr + h : xr - h;
  }
  if ((lane & 3) == 0) {
    const size_t row = (size_t)I * NB + q0 + rsel;
    put_packet(pk + row, xr, tag);
    x[row] = xr;
    if (sum) sum[row] += xr;
  }
}

// ---------------------------------------------------------------------------
// Refinement residual r = b - S0 x from the lower storage of S0.  Grid
// (row tile I, chunk); a chunk covers a range of column tiles J.  For J < I
// the tile S0_IJ is read row-wise (y_I += S0_IJ x_J), for J > I the tile
// S0_JI is read row-wise and applied transposed (y_I += S0_JI' x_J); the
// diagonal tile uses both halves.  ENV: only the column tiles env[I] ..
// env[ntiles + I] of the chunk, the others are zero (band of 47 tiles: 35 -> 14 us);
// the dense form without these bounds is the faster code (106 tiles: 120 against
// 144 us).  Partials per chunk are summed in a fixed
// order by the forward solve that follows.
template <typename T, int NCH, bool ENV>
static __global__ void __launch_bounds__(SV) symv_partial_kernel(const T* __restrict__ S0, int ld, int ntiles,
                                                                 const double* __restrict__ x,
                                                                 double* __restrict__ part,
                                                                 const int* __restrict__ env,
                                                                 const int* __restrict__ active) {
  __shared__ double red[SV / 32][NB];
  chain_start(S0, x, active);
  if (active && !*active) return;
  const int I = blockIdx.x, ch = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (ntiles + NCH - 1) / NCH;
  int J0 = ch * per, J1 = min(ntiles, J0 + per);
  if (ENV) {
    J0 = max(J0, env[I]);
    J1 = min(J1, env[ntiles + I] + 1);
  }
  double rp[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // rows 8 warp + rr
  double cp[4] = {0, 0, 0, 0};              // columns 4 lane + q
  for (int J = J0; J < J1; J++) {
    if (J <= I) {
      const T* Ls = S0 + (size_t)(I * NB + warp * 8) * ld + (size_t)J * NB + 4 * lane;
      double xv[4];
      load4(x + (size_t)J * NB + 4 * lane, xv);
#pragma unroll
      for (int rr = 0; rr < 8; rr++) {
        double lv[4];
        load4(Ls + (size_t)rr * ld, lv);
        if (J == I) {  // lower half of the diagonal tile: c <= r
          const int r = warp * 8 + rr;
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (4 * lane + q > r) lv[q] = 0.0;
        }
        rp[rr] += lv[0] * xv[0] + lv[1] * xv[1] + lv[2] * xv[2] + lv[3] * xv[3];
      }
    }
    if (J >= I) {
      const T* Ls = S0 + (size_t)(J * NB + warp * 8) * ld + (size_t)I * NB + 4 * lane;
#pragma unroll
      for (int rr = 0; rr < 8; rr++) {
        const int r = warp * 8 + rr;  // row of tile J
        const double xr = x[(size_t)J * NB + r];
        double lv[4];
        load4(Ls + (size_t)rr * ld, lv);
        if (J == I) {  // strictly-lower entries (r > c) applied transposed
#pragma unroll
          for (int q = 0; q < 4; q++)
            if (r <= 4 * lane + q) lv[q] = 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) cp[q] += lv[q] * xr;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 4; q++) red[warp][4 * lane + q] = cp[q];
  __syncthreads();
  double rowsum[8];
#pragma unroll
  for (int rr = 0; rr < 8; rr++) rowsum[rr] = warp_sum(rp[rr]);
  if (lane == 0) {
#pragma unroll
    for (int rr = 0; rr < 8; rr++) {
      const int r = warp * 8 + rr;
      double c = 0.0;
#pragma unroll
      for (int w = 0; w < SV / 32; w++) c += red[w][r];
      part[(size_t)ch * ntiles * NB + (size_t)I * NB + r] = rowsum[rr] + c;
    }
  }
}

}  // namespace nl
