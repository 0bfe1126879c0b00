// Exact-mode BFGS: the reference's arithmetic, one run per CTA.
//
// Reproduces bfgs::sequential::optimize (bfgs_sequential.cuh:46-234) value
// for value: same line search (utils.cuh:376-412), same inverse update
// (utils.cuh:245-287), same dual-number gradient (duals.cuh:241-266), same
// accept / termination order (bfgs_common.cuh:110-238).  The translation
// unit that instantiates this header is compiled with -fmad=false, so with
// the reference's own operation order every +,-,*,/ and sqrt rounds exactly
// as in the reference built for the host; only CUDA's transcendental
// functions may differ from the host libm by an ulp.
//
// The CTA spreads the work that the reference does serially but whose
// per-element arithmetic is independent, without changing any summation
// order:
//   * the D dual passes of the gradient, one per thread;
//   * the 20 line-search trials alpha = 2^-k, one per thread, taking the
//     first k that passes (the sequential loop returns exactly that alpha);
//   * p_i = -sum_j H_ij g_j, one row per thread (j ascending);
//   * the update's inner sums T_kj = sum_m H_km B_mj, computed once per
//     (k, j) instead of once per (i, k, j) -- the reference recomputes the
//     same value D times -- then H_ij = sum_k A_ik T_kj + rho s_i s_j.
// Dot products and the gradient norm stay on thread 0 in index order.
// H and T (2 D^2 doubles) live in a global workspace slice per CTA.
//
// Up to D = 32 a run has a warp instead (bfgs_exact_warp_kernel): H and T in
// shared memory, no block barriers, the same sums in the same order.
#pragma once

#include "zb_common.cuh"

namespace zb {

  struct ExactShared {
    double best, f1, fnew, ddir, sy, gnorm;
    int accepted, done, status, stop, executed;
  };

  template <class F, int D>
  __device__ __forceinline__ double
  eval_array(const F& f, const double* x)
  {
    std::array<double, D> a;
#pragma unroll 1
    for (int i = 0; i < D; ++i)
      a[i] = x[i];
    return f(a);
  }

  // g_i = d f / d x_i by a forward pass seeded with e_i, i = tid, tid+bs, ...
  template <class F, int D>
  __device__ __forceinline__ void
  exact_dual_gradient(const F& f, const double* x, double* g)
  {
    for (int i = threadIdx.x; i < D; i += blockDim.x) {
      std::array<dual::DualNumber, D> xd;
#pragma unroll 1
      for (int j = 0; j < D; ++j)
        xd[j] = dual::DualNumber(x[j], 0.0);
      xd[i].dual = 1.0;
      g[i] = f(xd).dual;
    }
  }

  template <class F, int D, bool Traj>
  __global__ void __launch_bounds__(128)
    bfgs_exact_kernel(F f, BfgsParams prm, const double* __restrict__ starts,
                      RunOut out, Control* ctl, double* __restrict__ scratch)
  {
    extern __shared__ __align__(16) double sm[];
    double* x = sm;
    double* xn = x + D;
    double* g = xn + D;
    double* gn = g + D;
    double* p = gn + D;
    double* s = p + D;
    double* y = s + D;
    __shared__ ExactShared sh;
    __shared__ int trial_ok[kLineSearchTrials];
    __shared__ double trial_f[kLineSearchTrials];

    double* H = scratch + (size_t)blockIdx.x * 2 * D * D;
    double* T = H + (size_t)D * D;
    const int tid = threadIdx.x, bs = blockDim.x;
    const int N = (int)prm.n;

    for (int64_t run = blockIdx.x; run < prm.n; run += gridDim.x) {
      const int idx = (int)run;
      for (int d = tid; d < D; d += bs) {
        x[d] = starts[(size_t)idx * D + d];
        g[d] = 0.0;
      }
      for (int e = tid; e < D * D; e += bs)
        H[e] = (e / D == e % D) ? 1.0 : 0.0;
      long long n_eval = 0, n_grad = 0;
      __syncthreads();
      const CycleTimer<true> tm(out, idx, tid == 0);
      if (tid == 0) {
        sh.best = eval_array<F, D>(f, x);
        sh.done = 0;
        sh.status = kUnset;
      }
      tm.start_grad();
      exact_dual_gradient<F, D>(f, x, g);
      ++n_eval;
      ++n_grad;
      __syncthreads();
      tm.stop_grad();

      int iter;
      for (iter = 0; iter < prm.max_iter; ++iter) {
        if constexpr (Traj) {
          for (int d = tid; d < D; d += bs)
            out.traj_x[(size_t)iter * D * N + (size_t)d * N + idx] = x[d];
          if (tid == 0) {
            double gg = 0.0;
            for (int i = 0; i < D; ++i)
              gg += g[i] * g[i];
            out.traj_f[(size_t)iter * N + idx] = sh.best;
            out.traj_g[(size_t)iter * N + idx] = ::sqrt(gg);
            out.traj_status[(size_t)iter * N + idx] = -1;
          }
        }
        if (tid == 0)
          sh.stop = load_stop(ctl);
        __syncthreads();
        if (sh.stop) {
          if (tid == 0) {
            sh.status = kStopped;
            double gg = 0.0;
            for (int i = 0; i < D; ++i)
              gg += g[i] * g[i];
            sh.gnorm = ::sqrt(gg);
            sh.fnew = sh.best; // f(x_arr) == bestVal by construction
            if constexpr (Traj)
              out.traj_status[(size_t)iter * N + idx] = kStopped;
          }
          __syncthreads();
          break;
        }
        // p = -H g (utils.cuh:148-161)
        for (int i = tid; i < D; i += bs) {
          double sum = 0.0;
          for (int j = 0; j < D; ++j)
            sum += H[(size_t)i * D + j] * g[j];
          p[i] = -sum;
        }
        __syncthreads();
        if (tid == 0) {
          double dd = 0.0;
          for (int i = 0; i < D; ++i)
            dd += g[i] * p[i];
          sh.ddir = dd;
        }
        __syncthreads();
        // line search trials alpha_k = 2^-k, k = 0..19
        for (int k = tid; k < kLineSearchTrials; k += bs) {
          double alpha = 1.0;
          for (int h = 0; h < k; ++h)
            alpha *= 0.5;
          std::array<double, D> xt;
#pragma unroll 1
          for (int j = 0; j < D; ++j)
            xt[j] = x[j] + alpha * p[j];
          const double f1 = f(xt);
          const double f0 = sh.best;
          trial_ok[k] = (f1 <= f0 + kArmijoC1 * alpha * sh.ddir && f1 < f0);
          trial_f[k] = f1;
        }
        __syncthreads();
        if (tid == 0) {
          int k = 0;
          while (k < kLineSearchTrials && !trial_ok[k])
            ++k;
          sh.accepted = k;
          sh.f1 = k < kLineSearchTrials ? trial_f[k] : 0.0;
          n_eval += (k < kLineSearchTrials ? k + 1 : kLineSearchTrials);
        }
        __syncthreads();
        {
          const int k = sh.accepted;
          double alpha = 1.0;
          for (int h = 0; h < k; ++h)
            alpha *= 0.5; // k == 20 gives the reference's 2^-20
          for (int i = tid; i < D; i += bs) {
            xn[i] = x[i] + alpha * p[i];
            s[i] = xn[i] - x[i];
          }
        }
        __syncthreads();
        if (tid == 0) {
          if (sh.accepted < kLineSearchTrials) {
            sh.fnew = sh.f1; // same point, same arithmetic as f(x_new)
          } else {
            sh.fnew = eval_array<F, D>(f, xn);
            ++n_eval;
          }
        }
        tm.start_grad();
        exact_dual_gradient<F, D>(f, xn, gn);
        ++n_grad;
        __syncthreads();
        tm.stop_grad();
        for (int i = tid; i < D; i += bs)
          y[i] = gn[i] - g[i];
        __syncthreads();
        if (tid == 0) {
          double sy = 0.0;
          for (int i = 0; i < D; ++i)
            sy += s[i] * y[i];
          sh.sy = sy;
        }
        __syncthreads();
        tm.start_update();
        if (!(::fabs(sh.sy) < kMinCurvature)) {
          const double rho = 1.0 / sh.sy;
          for (int e = tid; e < D * D; e += bs) {
            const int k = e / D, j = e % D;
            double inner = 0.0;
            for (int m = 0; m < D; ++m) {
              const double B_mj = ((m == j) ? 1.0 : 0.0) - rho * y[m] * s[j];
              inner += H[(size_t)k * D + m] * B_mj;
            }
            T[e] = inner;
          }
          __syncthreads();
          for (int e = tid; e < D * D; e += bs) {
            const int i = e / D, j = e % D;
            double sum = 0.0;
            for (int k = 0; k < D; ++k) {
              const double A_ik = ((i == k) ? 1.0 : 0.0) - rho * s[i] * y[k];
              sum += A_ik * T[(size_t)k * D + j];
            }
            H[e] = sum + rho * s[i] * s[j];
          }
        }
        const bool skipped = ::fabs(sh.sy) < kMinCurvature;
        __syncthreads();
        tm.stop_update();
        const bool take = sh.fnew < sh.best;
        if (take)
          for (int i = tid; i < D; i += bs) {
            x[i] = xn[i];
            g[i] = gn[i];
          }
        __syncthreads();
        if (tid == 0) {
          if (take)
            sh.best = sh.fnew;
          double gg = 0.0;
          for (int i = 0; i < D; ++i)
            gg += g[i] * g[i];
          const double gnrm = ::sqrt(gg);
          sh.gnorm = gnrm;
          if (!::isfinite(gnrm) || !::isfinite(sh.fnew)) {
            sh.status = kNonFinite; // fval = fnew (bfgs_common.cuh:156-157)
            sh.done = 1;
          } else if (gnrm < prm.tol) {
            note_converged(ctl, prm.required);
            sh.status = kConverged;
            sh.fnew = sh.best;
            sh.done = 1;
          } else if (!Traj && !take && skipped &&
                     !(prm.flags & kFlagNoFixedPoint)) {
            sh.done = 2; // fixed point: the rest would repeat this iteration
          }
          if constexpr (Traj)
            if (sh.done)
              out.traj_status[(size_t)iter * N + idx] = (int8_t)sh.status;
        }
        __syncthreads();
        if (sh.done == 2) {
          sh.executed = iter + 1;
          iter = prm.max_iter;
          break;
        }
        if (sh.done)
          break;
      }
      if (sh.done != 2)
        sh.executed = iter;
      if (tid == 0) {
        if (sh.status == kUnset) { // bfgs_common.cuh:213-238
          sh.status = kSurrender;
          sh.fnew = sh.best;
          double gg = 0.0;
          for (int i = 0; i < D; ++i)
            gg += g[i] * g[i];
          sh.gnorm = ::sqrt(gg);
          if constexpr (Traj)
            if (prm.max_iter > 0)
              out.traj_status[(size_t)(prm.max_iter - 1) * N + idx] = 0;
        }
        if (out.fval)
          out.fval[idx] = sh.fnew;
        if (out.status)
          out.status[idx] = sh.status;
        if (out.iter)
          out.iter[idx] = iter;
        if (out.gnorm)
          out.gnorm[idx] = sh.gnorm;
        if (out.counters) {
          out.counters[3 * (size_t)idx + 0] = sh.executed;
          out.counters[3 * (size_t)idx + 1] = n_eval;
          out.counters[3 * (size_t)idx + 2] = n_grad;
        }
        tm.finish();
      }
      if (out.x)
        for (int d = tid; d < D; d += bs)
          out.x[(size_t)idx * D + d] = x[d];
      __syncthreads();
    }
  }

  // ---------------------------------------------------------------- warp
  // One run per warp.  The lanes are DP columns (D rounded up to a power of
  // two) times G groups of rows:
  //   * gradient pass i on lane i; line-search trial k on lane k, alpha =
  //     2^-20 on lane 20, the first that passes found by a ballot;
  //   * lane (j, g) holds column j of B in registers and forms T_kj for the
  //     rows k = g, g + G, ..., then with column j of T the rows of H;
  //     A_ik is formed once per (i, k) in shared memory, so an inner step is
  //     one multiply and one add (five operations, as the CTA form computes
  //     A or B within it);
  //   * dot products and norms: every lane, in index order, from shared
  //     memory.
  // What bounds a run is the chain of those steps' latencies: the CTA form
  // adds fifteen block barriers an iteration, thread 0's sums while the others
  // wait, and H and T in L2.  512 Rosenbrock runs of 300 recorded iterations:
  // D = 2 850 -> 276 us, D = 10 1394 -> 612, D = 32 6266 -> 4412; 16384 runs at
  // D = 10 12.2 -> 2.5 ms (B200).
  inline constexpr int kExactWarpMaxDim = 32;
  inline constexpr int kExactWarpBlock = 64;

  template <int D>
  struct ExactWarpShape {
    // columns, a power of two, and groups of rows
    static constexpr int DP = D <= 2 ? 2 : D <= 4 ? 4 : D <= 8 ? 8 : D <= 16 ? 16 : 32;
    static constexpr int G = 32 / DP;
    static constexpr int SD = D | 1;             // row stride: rows on different banks
    static constexpr int NR = (D + G - 1) / G;   // rows of a lane
    static constexpr int RB = NR < 8 ? NR : 8;   // ... formed at a time
    static constexpr int doubles = 7 * D + 3 * D * SD; // per warp
  };

  // Row k, or the last row where the last block of a lane's rows runs past it
  // (its sums are not kept).
  template <int D, class S>
  __device__ __forceinline__ int
  exact_row(int k)
  {
    return S::NR % S::RB == 0 && D % S::G == 0 ? k : (k < D ? k : D - 1);
  }

  // f at x + alpha p, coordinate by coordinate as the reference forms it
  template <class F, int D>
  __device__ __forceinline__ double
  exact_trial(const F& f, const double* x, const double* p, double alpha)
  {
    std::array<double, D> a;
#pragma unroll
    for (int j = 0; j < D; ++j)
      a[j] = x[j] + alpha * p[j];
    return f(a);
  }

  template <class F, int D>
  __device__ __forceinline__ double
  exact_dual_entry(const F& f, const double* x, int i)
  {
    std::array<dual::DualNumber, D> xd;
#pragma unroll
    for (int j = 0; j < D; ++j)
      xd[j] = dual::DualNumber(x[j], j == i ? 1.0 : 0.0);
    return f(xd).dual;
  }

  // sum_i a_i b_i in index order
  template <int D>
  __device__ __forceinline__ double
  exact_dot(const double* a, const double* b)
  {
    double v = 0.0;
#pragma unroll 8
    for (int i = 0; i < D; ++i)
      v += a[i] * b[i];
    return v;
  }

  template <class F, int D, bool Traj>
  __global__ void __launch_bounds__(kExactWarpBlock)
    bfgs_exact_warp_kernel(F f, BfgsParams prm, const double* __restrict__ starts,
                           RunOut out, Control* ctl)
  {
    using S = ExactWarpShape<D>;
    constexpr int DP = S::DP, G = S::G, SD = S::SD, NR = S::NR, RB = S::RB;
    extern __shared__ __align__(16) double sm[];
    const int lane = threadIdx.x & 31;
    double* x = sm + (threadIdx.x >> 5) * S::doubles;
    double* xn = x + D;
    double* g = xn + D;
    double* gn = g + D;
    double* p = gn + D;
    double* s = p + D;
    double* y = s + D;
    double* H = y + D;
    double* T = H + D * SD;
    double* A = T + D * SD;
    const int N = (int)prm.n;
    const int idx = (int)(blockIdx.x * (kExactWarpBlock / 32) + (threadIdx.x >> 5));
    if (idx >= N)
      return; // the whole warp leaves together
    const int j = lane % DP, grp = lane / DP; // column and group of rows
    const bool col = j < D;
    if (lane < D)
      x[lane] = starts[(size_t)idx * D + lane];
    for (int e = lane; e < D * D; e += 32)
      H[e / D * SD + e % D] = (e / D == e % D) ? 1.0 : 0.0;
    __syncwarp();
    const CycleTimer<true> tm(out, idx, lane == 0);
    long long n_eval = 1, n_grad = 1;
    int status = kUnset, executed = -1;
    double best = 0.0;
    if (lane == 0)
      best = eval_array<F, D>(f, x);
    best = __shfl_sync(0xffffffffu, best, 0);
    tm.start_grad();
    if (lane < D)
      g[lane] = exact_dual_entry<F, D>(f, x, lane);
    __syncwarp();
    tm.stop_grad();
    double gnorm = ::sqrt(exact_dot<D>(g, g)); // of the gradient at x
    double fout = best;
    // the stop flag, read one iteration ahead of the test
    int stop = load_stop(ctl);

    int iter;
    for (iter = 0; iter < prm.max_iter; ++iter) {
      if constexpr (Traj) {
        if (lane < D)
          out.traj_x[(size_t)iter * D * N + (size_t)lane * N + idx] = x[lane];
        if (lane == 0) {
          out.traj_f[(size_t)iter * N + idx] = best;
          out.traj_g[(size_t)iter * N + idx] = gnorm;
        }
      }
      stop = __shfl_sync(0xffffffffu, stop, 0);
      if (stop) {
        status = kStopped;
        fout = best; // f(x_arr) == bestVal by construction
        if constexpr (Traj)
          if (lane == 0)
            out.traj_status[(size_t)iter * N + idx] = kStopped;
        break;
      }
      stop = load_stop(ctl);
      // p = -H g (utils.cuh:148-161)
      if (lane < D)
        p[lane] = -exact_dot<D>(H + lane * SD, g);
      __syncwarp();
      const double ddir = exact_dot<D>(g, p);
      // line search trials alpha_k = 2^-k, k = 0..19; alpha = 2^-20 when none
      // passes
      double f1 = 0.0;
      bool pass = false;
      if (lane <= kLineSearchTrials) {
        const double alpha = pow2neg(lane);
        f1 = exact_trial<F, D>(f, x, p, alpha);
        pass = lane == kLineSearchTrials ||
               (f1 <= best + kArmijoC1 * alpha * ddir && f1 < best);
      }
      const int found = __ffs((int)__ballot_sync(0xffffffffu, pass)) - 1;
      const double fnew = __shfl_sync(0xffffffffu, f1, found);
      n_eval += found + 1;
      if (lane < D) {
        const double alpha = pow2neg(found);
        const double v = x[lane] + alpha * p[lane];
        xn[lane] = v;
        s[lane] = v - x[lane];
      }
      __syncwarp();
      tm.start_grad();
      if (lane < D) {
        const double v = exact_dual_entry<F, D>(f, xn, lane);
        gn[lane] = v;
        y[lane] = v - g[lane];
      }
      ++n_grad;
      __syncwarp();
      tm.stop_grad();
      const double sy = exact_dot<D>(s, y);
      const bool skipped = ::fabs(sy) < kMinCurvature;
      tm.start_update();
      if (!skipped) {
        const double rho = 1.0 / sy;
        {
          double b[D]; // column j of B
          const double sj = col ? s[j] : 0.0;
#pragma unroll
          for (int m = 0; m < D; ++m) {
            const double ry = rho * y[m];
            b[m] = ((m == j) ? 1.0 : 0.0) - ry * sj;
          }
          if (col)
#pragma unroll 1
            for (int r0 = 0; r0 < NR; r0 += RB) {
              double acc[RB];
#pragma unroll
              for (int r = 0; r < RB; ++r)
                acc[r] = 0.0;
#pragma unroll
              for (int m = 0; m < D; ++m)
#pragma unroll
                for (int r = 0; r < RB; ++r)
                  acc[r] += H[exact_row<D, S>(grp + G * (r0 + r)) * SD + m] * b[m];
#pragma unroll
              for (int r = 0; r < RB; ++r) {
                const int k = grp + G * (r0 + r);
                if (k < D)
                  T[k * SD + j] = acc[r];
              }
            }
          // A_ik, row i, column k = j
          if (col) {
            const double yj = y[j];
#pragma unroll 4
            for (int i = grp; i < D; i += G) {
              const double rs = rho * s[i];
              A[i * SD + j] = ((i == j) ? 1.0 : 0.0) - rs * yj;
            }
          }
        }
        __syncwarp();
        if (col) {
          double tc[D]; // column j of T
#pragma unroll
          for (int k = 0; k < D; ++k)
            tc[k] = T[k * SD + j];
          const double sj = s[j];
#pragma unroll 1
          for (int r0 = 0; r0 < NR; r0 += RB) {
            double acc[RB];
#pragma unroll
            for (int r = 0; r < RB; ++r)
              acc[r] = 0.0;
#pragma unroll
            for (int k = 0; k < D; ++k)
#pragma unroll
              for (int r = 0; r < RB; ++r)
                acc[r] += A[exact_row<D, S>(grp + G * (r0 + r)) * SD + k] * tc[k];
#pragma unroll
            for (int r = 0; r < RB; ++r) {
              const int i = grp + G * (r0 + r);
              if (i < D)
                H[i * SD + j] = acc[r] + rho * s[i] * sj;
            }
          }
        }
        __syncwarp();
      }
      tm.stop_update();
      const bool take = fnew < best;
      if (take) {
        if (lane < D) {
          x[lane] = xn[lane];
          g[lane] = gn[lane];
        }
        __syncwarp();
        best = fnew;
        gnorm = ::sqrt(exact_dot<D>(g, g));
      }
      int done = 0;
      if (!::isfinite(gnorm) || !::isfinite(fnew)) {
        status = kNonFinite; // fval = fnew (bfgs_common.cuh:156-157)
        fout = fnew;
        done = 1;
      } else if (gnorm < prm.tol) {
        if (lane == 0)
          note_converged(ctl, prm.required);
        status = kConverged;
        fout = best;
        done = 1;
      } else if (!Traj && !take && skipped && !(prm.flags & kFlagNoFixedPoint)) {
        done = 2; // fixed point: the rest would repeat this iteration
      }
      if constexpr (Traj)
        if (lane == 0)
          out.traj_status[(size_t)iter * N + idx] = (int8_t)status;
      if (done == 2) {
        executed = iter + 1;
        iter = prm.max_iter;
      }
      if (done)
        break;
    }
    if (status == kUnset) { // bfgs_common.cuh:213-238
      status = kSurrender;
      fout = best;
      if constexpr (Traj)
        if (lane == 0 && prm.max_iter > 0)
          out.traj_status[(size_t)(prm.max_iter - 1) * N + idx] = 0;
    }
    if (lane == 0) {
      if (out.fval)
        out.fval[idx] = fout;
      if (out.status)
        out.status[idx] = status;
      if (out.iter)
        out.iter[idx] = iter;
      if (out.gnorm)
        out.gnorm[idx] = gnorm;
      if (out.counters) {
        out.counters[3 * (size_t)idx + 0] = executed >= 0 ? executed : iter;
        out.counters[3 * (size_t)idx + 1] = n_eval;
        out.counters[3 * (size_t)idx + 2] = n_grad;
      }
      tm.finish();
    }
    if (out.x && lane < D)
      out.x[(size_t)idx * D + lane] = x[lane];
  }

  template <int D>
  inline size_t
  exact_smem_bytes()
  {
    return sizeof(double) * 7 * D;
  }

} // namespace zb
