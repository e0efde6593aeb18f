// lm_kernels.cuh -- LevenbergMarquardt / GaussNewton control kept on the device.
//
// The state machine of LevenbergMarquardt::solve
// (nelson/LevenbergMarquardt.hpp:36-146) split into single-thread kernels
// that read and write an LmDev record in device memory, so one sub-iteration
// is a fixed launch sequence (capturable in a CUDA graph) whose kernels test
// flags instead of the host branching:
//   [computeIncrement kernels, predicated on `active`]
//   inc_dot_kernel     |inc|^2, den = inc'(mu inc - b); SuccessSmallIncrement test;
//                      `apply` = active && solve ok && !done
//   [oplus + cost kernels, predicated on `apply`]
//   lm_decide_kernel   rho, accept / reject, mu / v update, termination tests;
//                      `rollback` and `do_jac` flags
//   [rollback copies on `rollback`; Jacobian pass on `do_jac`]
//   lm_after_jac_kernel oldChi2 = chi2, iter++, MaxIterationReached test; the
//                      next sub-iteration's flags (active = !done, status 0)
#pragma once

#include "nl_common.cuh"

namespace nl {

struct LmDev {
  // settings (LevenbergMarquardtSettings / GaussNewtonSettings)
  int maxNumIt, maxNumSubIt, minNumIt, gn;
  double epsBVector, epsIncSquare, epsChi2, tau, penaltyV, initV, maxScale, minScale;
  double gnRel, gnAbs;
  // state
  double mu, curV, oldChi2, chi2, chi2_new, rho, incSq, den, maxAbsB, maxAbsHDiag;
  double lam[2];  // (relLambda, absLambda) read by the solver kernels
  int iter, subiter, nsub, done;  // read by the host in one copy
  int reason, solve_ok;
  int active, apply, rollback, do_jac, accepted;
  int trace_n, trace_cap;
  int status;     // solver status bits of the current sub-iteration
};

// The flags and the damping of the next sub-iteration: set on the host for the
// first one, at the end of lm_after_jac_kernel for the others.
__host__ __device__ inline void lm_begin(LmDev* s) {
  s->active = s->done ? 0 : 1;
  s->status = 0;
  s->apply = 0;
  s->rollback = 0;
  s->do_jac = 0;
  if (!s->done) {
    s->lam[0] = s->gn ? s->gnRel : 0.0;
    s->lam[1] = s->gn ? s->gnAbs : s->mu;
  }
}

__device__ inline void lm_trace(LmDev* s, double* trace, double it, double sub, double chi2, double mu, double rho,
                                double inc, double ok, double acc) {
  if (trace && s->trace_n < s->trace_cap) {
    double* t = trace + (size_t)s->trace_n * NL_TRACE_STRIDE;
    t[0] = it; t[1] = sub; t[2] = chi2; t[3] = mu; t[4] = rho; t[5] = inc; t[6] = ok; t[7] = acc;
  }
  s->trace_n++;
}

// |inc|^2 and inc'(mu inc - b), CTA partials added by the last CTA, which then
// takes the first decisions of the sub-iteration.
__device__ inline void lm_inc(LmDev* s, double a, double b, double* trace);
template <typename T, int NT>
static __global__ void __launch_bounds__(NT) inc_dot_kernel(const double* __restrict__ incU, const T* __restrict__ bU,
                                                     int nu, const double* __restrict__ incV,
                                                     const T* __restrict__ bV, int nv, LmDev* __restrict__ s,
                                                     double* __restrict__ part, int* __restrict__ count,
                                                     double* __restrict__ trace) {
  __shared__ double sh[NT / 32];
  chain_start(incU, bU, incV, bV);
  if (!s->active) return;
  const double mu = s->gn ? 0.0 : s->mu;
  double a = 0.0, b = 0.0;
  for (int i = blockIdx.x * NT + threadIdx.x; i < nu + nv; i += gridDim.x * NT) {
    double x, g;
    if (i < nu) {
      x = incU[i];
      g = (double)bU[i];
    } else {
      x = incV[i - nu];
      g = (double)bV[i - nu];
    }
    a += x * x;
    b += x * (mu * x - g);
  }
  a = block_sum<NT>(a, sh);
  b = block_sum<NT>(b, sh);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = a;
    part[2 * blockIdx.x + 1] = b;
  }
  if (!last_block(count)) return;
  a = b = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += NT) {
    a += __ldcg(part + 2 * i);
    b += __ldcg(part + 2 * i + 1);
  }
  a = block_sum<NT>(a, sh);
  b = block_sum<NT>(b, sh);
  if (threadIdx.x == 0) lm_inc(s, a, b, trace);
}

__device__ inline void lm_inc(LmDev* s, double a, double b, double* trace) {
  s->solve_ok = (s->status & (ST_VINV_FAIL | ST_CHOL_FAIL | ST_SPIN_TIMEOUT)) == 0;
  if (!isfinite(a)) s->solve_ok = 0;
  s->incSq = s->solve_ok ? a : 0.0;
  s->den = b;
  if (s->gn) {
    // GaussNewton::solve (nelson/GaussNewton.hpp:64-87)
    if (!s->solve_ok) {
      lm_trace(s, trace, s->iter, 0, -1, 0, 0, s->incSq, 0, 0);
      s->done = 1;
      s->reason = NL_SOLVER_FAILURE;
      return;
    }
    if (s->iter >= s->minNumIt && s->incSq <= s->epsIncSquare) {
      lm_trace(s, trace, s->iter, 0, s->chi2, 0, 0, s->incSq, 1, 0);
      s->done = 1;
      s->reason = NL_SUCCESS_SMALL_INCREMENT;
      return;
    }
    s->apply = 1;
    return;
  }
  // LevenbergMarquardt.hpp:73-75
  if (s->solve_ok && s->iter >= s->minNumIt && s->incSq <= s->epsIncSquare) {
    lm_trace(s, trace, s->iter, s->subiter, s->chi2, s->mu, 0, s->incSq, 1, 0);
    s->done = 1;
    s->reason = NL_SUCCESS_SMALL_INCREMENT;
    return;
  }
  s->apply = s->solve_ok;
}

// LevenbergMarquardt.hpp:78-129 (LM) / GaussNewton.hpp:89-123 (GN).
static __global__ void lm_decide_kernel(LmDev* s, double* trace) {
  chain_start();
  if (!s->active || s->done) return;
  if (s->gn) {
    // oplus + update(true) already ran: chi2_new and maxAbsB are current
    s->nsub++;
    s->do_jac = 1;  // the Jacobian pass runs on the accepted state
    return;
  }
  double rho = -1.0;
  if (s->apply) rho = (s->oldChi2 - s->chi2_new) / s->den;
  s->rho = rho;
  const bool acc = s->apply && rho > 0.0;
  s->accepted = acc ? 1 : 0;
  lm_trace(s, trace, s->iter, s->subiter, s->apply ? s->chi2_new : -1.0, s->mu, rho, s->incSq, s->solve_ok, acc);
  s->nsub++;
  if (acc) {
    s->chi2 = s->chi2_new;
    if (s->iter > s->minNumIt && s->maxAbsB <= s->epsBVector) {
      s->done = 1;
      s->reason = NL_SUCCESS_EPS_B;
      return;
    }
    if (s->iter > s->minNumIt && s->chi2_new < s->epsChi2) {
      s->done = 1;
      s->reason = NL_SUCCESS_SMALL_RESIDUALS;
      return;
    }
    const double fc = 2.0 * rho - 1.0;
    double alpha = fmin(s->maxScale, 1.0 - fc * fc * fc);
    alpha = fmax(s->minScale, alpha);
    s->mu = s->mu * alpha;
    s->curV = s->initV;
  } else {
    s->rollback = 1;
    s->mu = s->mu * s->curV;
    s->curV = s->curV * s->penaltyV;
  }
  s->subiter++;
  if (s->subiter >= s->maxNumSubIt) {
    s->done = 1;
    s->reason = NL_MAX_SUBITERATION_REACHED;
    return;
  }
  if (acc) s->do_jac = 1;
}

// The cost of update(true) is the accepted candidate's: the same parameters.
// chi2_out: the handle's cost.
__device__ inline void lm_after_jac(LmDev* s, double* chi2_out, double* trace) {
  s->chi2 = *chi2_out = s->chi2_new;
  s->oldChi2 = s->chi2;
  if (s->gn) {
    // GaussNewton.hpp:104-123
    lm_trace(s, trace, s->iter, 0, s->chi2, 0, 0, s->incSq, 1, 1);
    if (s->iter > s->minNumIt && s->maxAbsB <= s->epsBVector) {
      s->done = 1;
      s->reason = NL_SUCCESS_EPS_B;
      return;
    }
    if (s->iter > s->minNumIt && s->chi2 < s->epsChi2) {
      s->done = 1;
      s->reason = NL_SUCCESS_SMALL_RESIDUALS;
      return;
    }
  }
  s->iter++;
  s->subiter = 0;
  if (s->iter >= s->maxNumIt) {
    s->done = 1;
    s->reason = NL_MAX_ITERATION_REACHED;
  }
}
static __global__ void lm_after_jac_kernel(LmDev* s, double* chi2_out, double* trace) {
  chain_start();
  if (!s->active) return;
  if (s->do_jac) lm_after_jac(s, chi2_out, trace);
  lm_begin(s);
}

// Maximum over the block, then over the CTAs' partials by the last CTA.
template <int NT>
__device__ inline void max_out(double m, double* sh, double* __restrict__ part, int* __restrict__ count,
                               double* __restrict__ out) {
  auto block_max = [&](double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
      for (int i = 0; i < NT / 32; i++) r = fmax(r, sh[i]);
    __syncthreads();
    return r;
  };
  m = block_max(m);
  if (threadIdx.x == 0) part[blockIdx.x] = m;
  if (!last_block(count)) return;
  m = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += NT) m = fmax(m, __ldcg(part + i));
  m = block_max(m);
  if (threadIdx.x == 0) *out = m;
}

// max |x| over two arrays.
template <typename T, int NT>
static __global__ void __launch_bounds__(NT) maxabs_kernel(const T* __restrict__ a, int na, const T* __restrict__ b, int nb,
                                                    double* __restrict__ part, int* __restrict__ count,
                                                    double* __restrict__ out, const int* __restrict__ active) {
  __shared__ double sh[NT / 32];
  chain_start(a, b, active);
  if (active && !*active) return;
  double m = 0.0;
  for (int i = blockIdx.x * NT + threadIdx.x; i < na + nb; i += gridDim.x * NT) {
    const double v = fabs((double)(i < na ? a[i] : b[i - na]));
    m = fmax(m, v);
  }
  max_out<NT>(m, sh, part, count, out);
}

// max |diag| over the U diagonal blocks and the V blocks (SolverCholeskySchur::maxAbsHDiag).
template <typename T, int BC, int NT>
static __global__ void __launch_bounds__(NT) hdiag_kernel(const T* __restrict__ U, const int* __restrict__ u_diag_uid,
                                                   int nci, const T* __restrict__ V, const int* __restrict__ v_uid,
                                                   int np, double* __restrict__ part, int* __restrict__ count,
                                                   double* __restrict__ out) {
  __shared__ double sh[NT / 32];
  double m = 0.0;
  for (int i = blockIdx.x * NT + threadIdx.x; i < nci + np; i += gridDim.x * NT) {
    if (i < nci) {
      const int q = u_diag_uid[i];
      if (q >= 0)
        for (int r = 0; r < BC; r++) m = fmax(m, fabs((double)U[(size_t)q * Layout<T, BC>::U + r * BC + r]));
    } else {
      const int q = v_uid[i - nci];
      if (q >= 0)
        for (int r = 0; r < 3; r++) m = fmax(m, fabs((double)V[(size_t)q * Layout<T, BC>::V + r * 3 + r]));
    }
  }
  max_out<NT>(m, sh, part, count, out);
}

// copies predicated on a device flag (backup / rollback of parameters)
static __global__ void copy_if_kernel(double* __restrict__ dst, const double* __restrict__ src, size_t n,
                                      double* __restrict__ dst2, const double* __restrict__ src2, size_t n2,
                                      const int* __restrict__ flag) {
  chain_start(src, src2, flag);
  if (flag && !*flag) return;
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x, nt = (size_t)gridDim.x * blockDim.x;
  for (size_t i = t; i < n; i += nt) dst[i] = src[i];
  for (size_t i = t; i < n2; i += nt) dst2[i] = src2[i];
}

}  // namespace nl
