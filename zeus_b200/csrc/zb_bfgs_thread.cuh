// Fast BFGS for small D (the layout for D <= 8): one run per thread, or the
// same run on the 32 lanes of a warp.
//
// Everything a run owns lives in registers: x, g, p and the inverse Hessian
// H, stored as its upper triangle (D(D+1)/2 doubles).  The symmetric rank-2
// form of the reference's update (utils.cuh:245-287),
//   H+ = H + s w^T + w s^T,  u = H y,  w = -rho u + rho (1 + rho y.u)/2 s,
// costs O(D^2) instead of the reference's O(D^4) and keeps H exactly
// symmetric (each (i, j) pair is formed once).  The line search, the
// |s.y| < 1e-14 skip, accept-if-better and the termination protocol are the
// reference's (utils.cuh:376-412, bfgs_sequential.cuh:99-219); f at the
// accepted trial point is reused as f(x_new) and f(x) at termination is
// the tracked best value, both identical to what the reference recomputes.
#pragma once

#include "zb_common.cuh"

namespace zb {

  template <int D>
  __host__ __device__ constexpr int
  tri(int i, int j) // packed upper-triangle index, i <= j
  {
    return i * D - (i * (i - 1)) / 2 + (j - i);
  }
  template <int D>
  __host__ __device__ constexpr int
  sym(int i, int j)
  {
    return i <= j ? tri<D>(i, j) : tri<D>(j, i);
  }

  // f(x) through the objective's fast path when it has one.
  template <class F, int D>
  __device__ __forceinline__ double
  fast_value(const F& f, const double* x)
  {
    if constexpr (HasValue<F>) {
      return f.value(x);
    } else {
      std::array<double, D> a;
#pragma unroll
      for (int i = 0; i < D; ++i)
        a[i] = x[i];
      return f(a);
    }
  }

  // Gradient by D forward dual passes (the plain form), or by the
  // objective's adjoint.
  template <class F, int D, bool Adjoint>
  __device__ __forceinline__ void
  fast_gradient(const F& f, const double* x, double* g)
  {
    if constexpr (Adjoint && HasAdjoint<F>) {
      (void)f.adjoint(x, g);
    } else {
      std::array<dual::DualNumber, D> xd;
#pragma unroll
      for (int j = 0; j < D; ++j)
        xd[j] = dual::DualNumber(x[j], 0.0);
#pragma unroll
      for (int i = 0; i < D; ++i) {
        xd[i].dual = 1.0;
        g[i] = f(xd).dual;
        xd[i].dual = 0.0;
      }
    }
  }

  // Whether a thread of the standalone kernel takes ||g|| = sqrt(g.g) only where
  // it decides something (far above tol^2, g.g cannot pass the test), as a warp
  // does, and a thread of the batch kernel (the mixed batch 16.1 against 16.6 ms
  // with a root an iteration).  Here the branch costs more than the root
  // (8192 Ackley-10 runs 484 us with the root, 517 with the branch; 4096
  // likelihood fits with dual gradients 60.6 and 65.2 ms; Rosenbrock-4 95
  // registers and 104), but for the likelihood's adjoint (16384 fits of 300
  // iterations 74 and 56 ms).
  template <class F, bool Adjoint>
  constexpr bool
  root_rarely()
  {
    if constexpr (requires { F::kind; })
      return Adjoint && F::kind == 4;
    return false;
  }

  // One run, start x0[D], results to slot idx of `out`, on the calling thread
  // alone (G = 1) or on its warp (G = 32).  On a warp every lane holds the
  // whole run -- x, g, p, H and each scalar, the same bits in all of them --
  // and they differ only in the line search: lane l evaluates trial l, a
  // ballot picks the first that passes.  The values are those of the
  // one-thread form bit for bit, trial by trial and sum by sum.
  template <class F, int D, bool Adjoint, bool kTimed = false, int G = 1, bool Rarely = true>
  __device__ __forceinline__ void
  thread_run(const F& f, const BfgsParams& prm, const double* __restrict__ x0,
             int64_t idx, const RunOut& out, Control* ctl)
  {
    static_assert(G == 1 || !kTimed, "the cycle timers are per thread");
    static_assert(G == 1 || G == 32, "a thread or a warp");
    constexpr int NT = D * (D + 1) / 2;
    const int lane = G > 1 ? (int)(threadIdx.x & 31) : 0;
    double x[D], g[D], p[D], H[NT];
#pragma unroll
    for (int i = 0; i < D; ++i)
      x[i] = x0[i];
#pragma unroll
    for (int i = 0; i < D; ++i)
#pragma unroll
      for (int j = i; j < D; ++j)
        H[tri<D>(i, j)] = (i == j) ? 1.0 : 0.0;

    const CycleTimer<kTimed> tm(out, idx, true);
    double best = fast_value<F, D>(f, x);
    tm.start_grad();
    fast_gradient<F, D, Adjoint>(f, x, g);
    tm.stop_grad();
    long long n_eval = 1, n_grad = 1;
#pragma unroll
    for (int i = 0; i < D; ++i)
      p[i] = -g[i];

    int status = kUnset, iter, executed = -1;
    double fout = best, gout = 0.0;
    const double tol_sq4 = 4.0 * prm.tol * prm.tol;
    // the stop flag: a warp tests it every kStopEvery iterations, on the value
    // read at the previous test; a thread reads it one iteration ahead
    constexpr int every = G > 1 ? kStopEvery : 1;
    int stop = load_stop(ctl);
    for (iter = 0; iter < prm.max_iter; ++iter) {
      if (iter % every == 0) {
        if constexpr (G > 1)
          stop = __shfl_sync(0xffffffffu, stop, 0);
        if (stop) {
          status = kStopped;
          break;
        }
        stop = load_stop(ctl);
      }
      double ddir = 0.0;
#pragma unroll
      for (int i = 0; i < D; ++i)
        ddir = fma(g[i], p[i], ddir);
      double xn[D], alpha = 1.0, fnew = 0.0;
      if constexpr (G > 1) {
        // lanes past trial 20 judge nothing: trial 20 (alpha = 2^-20, taken
        // when no other passes) always passes before them
        const double ak = pow2neg(lane);
#pragma unroll
        for (int i = 0; i < D; ++i)
          xn[i] = fma(ak, p[i], x[i]);
        const double f1 = fast_value<F, D>(f, xn);
        const bool pass = lane >= kLineSearchTrials ||
                          (f1 <= best + kArmijoC1 * ak * ddir && f1 < best);
        const int found = __ffs((int)__ballot_sync(0xffffffffu, pass)) - 1;
        fnew = __shfl_sync(0xffffffffu, f1, found);
        n_eval += found + 1;
        alpha = pow2neg(found);
#pragma unroll
        for (int i = 0; i < D; ++i)
          xn[i] = fma(alpha, p[i], x[i]);
      } else {
        bool ok = false;
        for (int k = 0; k < kLineSearchTrials; ++k) {
#pragma unroll
          for (int i = 0; i < D; ++i)
            xn[i] = fma(alpha, p[i], x[i]);
          const double f1 = fast_value<F, D>(f, xn);
          ++n_eval;
          if (f1 <= best + kArmijoC1 * alpha * ddir && f1 < best) {
            ok = true;
            fnew = f1;
            break;
          }
          alpha *= 0.5;
        }
        if (!ok) {
#pragma unroll
          for (int i = 0; i < D; ++i)
            xn[i] = fma(alpha, p[i], x[i]);
          fnew = fast_value<F, D>(f, xn);
          ++n_eval;
        }
      }
      double gn[D], s[D], y[D];
      tm.start_grad();
      fast_gradient<F, D, Adjoint>(f, xn, gn);
      tm.stop_grad();
      ++n_grad;
      tm.start_update();
      double sy = 0.0;
#pragma unroll
      for (int i = 0; i < D; ++i) {
        s[i] = xn[i] - x[i];
        y[i] = gn[i] - g[i];
        sy = fma(s[i], y[i], sy);
      }
      // u = H y and y.u ahead of the division, which they do not need
      double u[D], yu = 0.0;
#pragma unroll
      for (int i = 0; i < D; ++i) {
        double a = 0.0;
#pragma unroll
        for (int j = 0; j < D; ++j)
          a = fma(H[sym<D>(i, j)], y[j], a);
        u[i] = a;
        yu = fma(y[i], a, yu);
      }
      const bool skipped = fabs(sy) < kMinCurvature;
      if (!skipped) {
        const double rho = 1.0 / sy;
        const double half_beta = 0.5 * rho * fma(rho, yu, 1.0);
        double w[D];
#pragma unroll
        for (int i = 0; i < D; ++i)
          w[i] = fma(half_beta, s[i], -rho * u[i]);
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
          for (int j = i; j < D; ++j)
            H[tri<D>(i, j)] += s[i] * w[j] + w[i] * s[j];
      }
      tm.stop_update();
      const bool take = fnew < best;
      if (take) {
        best = fnew;
#pragma unroll
        for (int i = 0; i < D; ++i) {
          x[i] = xn[i];
          g[i] = gn[i];
        }
      }
      double gg = 0.0;
#pragma unroll
      for (int i = 0; i < D; ++i)
        gg = fma(g[i], g[i], gg);
      const double size = Rarely ? gg : sqrt(gg);
      if (!isfinite(size) || !isfinite(fnew)) {
        status = kNonFinite;
        fout = fnew;
        gout = sqrt(gg);
        break;
      }
      if (Rarely ? gg <= tol_sq4 && sqrt(gg) < prm.tol : size < prm.tol) {
        if (lane == 0)
          note_converged(ctl, prm.required);
        status = kConverged;
        fout = best;
        gout = sqrt(gg);
        break;
      }
      if (!take && skipped && !(prm.flags & kFlagNoFixedPoint)) {
        executed = iter + 1; // fixed point: the rest would repeat this
        iter = prm.max_iter;
        break;
      }
#pragma unroll
      for (int i = 0; i < D; ++i) {
        double a = 0.0;
#pragma unroll
        for (int j = 0; j < D; ++j)
          a = fma(H[sym<D>(i, j)], g[j], a);
        p[i] = -a;
      }
    }
    if (status == kUnset || status == kStopped) {
      if (status == kUnset)
        status = kSurrender;
      fout = best;
      double gg = 0.0;
#pragma unroll
      for (int i = 0; i < D; ++i)
        gg = fma(g[i], g[i], gg);
      gout = sqrt(gg);
    }
    if (lane != 0)
      return;
    if (out.fval)
      out.fval[idx] = fout;
    if (out.status)
      out.status[idx] = status;
    if (out.iter)
      out.iter[idx] = iter;
    if (out.gnorm)
      out.gnorm[idx] = gout;
    if (out.x)
#pragma unroll
      for (int i = 0; i < D; ++i)
        out.x[idx * D + i] = x[i];
    if (out.counters) {
      out.counters[3 * idx + 0] = executed >= 0 ? executed : iter;
      out.counters[3 * idx + 1] = n_eval;
      out.counters[3 * idx + 2] = n_grad;
    }
    tm.finish();
  }

  template <class F, int D, bool Adjoint, bool kTimed = false>
  __global__ void __launch_bounds__(128)
    bfgs_thread_kernel(F f, BfgsParams prm, const double* __restrict__ starts,
                       RunOut out, Control* ctl)
  {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < prm.n)
      thread_run<F, D, Adjoint, kTimed, 1, root_rarely<F, Adjoint>()>(f, prm, starts + idx * D,
                                                                      idx, out, ctl);
  }

  // A run to a warp.  A launch lasts as long as its slowest runs, those
  // that iterate to MAX_ITER: there no trial passes, and one thread
  // evaluates 21 of them one after another while its warp's other lanes
  // wait.  All 21 at once leave the chain of one evaluation, one gradient
  // and the update, 0.35 us an iteration at D = 2 against 1.04 and 0.59
  // against 3.7 at D = 8, one run alone (B200, 1965 MHz; a good part of the
  // latter is the objective's unrolling, see Rosenbrock::adjoint).  1024
  // Rosenbrock-2 runs 10.5 -> 3.9 ms, 4099 Rosenbrock-8 runs 40.2 -> 8.8 or
  // 12.9 (by which SM partitions the 44 that iterate to MAX_ITER share), 16384
  // Rastrigin-2 runs 54 -> 6.4, 16384 Ackley-2 runs 72 -> 14; widths of 16 and 8
  // lanes measured slower throughout (10.0 and 12.4 ms for 16384 Rosenbrock-2
  // runs, 8.1 on 32).
  inline constexpr int kThreadGroupBlock = 64;

  template <class F, int D, bool Adjoint>
  __global__ void __launch_bounds__(kThreadGroupBlock)
    bfgs_thread_warp_kernel(F f, BfgsParams prm, const double* __restrict__ starts,
                            RunOut out, Control* ctl)
  {
    const int64_t idx =
      ((int64_t)blockIdx.x * kThreadGroupBlock + threadIdx.x) / 32;
    if (idx < prm.n) // uniform within the warp
      thread_run<F, D, Adjoint, false, 32>(f, prm, starts + idx * D, idx, out, ctl);
  }

} // namespace zb
