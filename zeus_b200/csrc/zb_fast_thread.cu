// Thread-layout fast BFGS launcher (D <= 10).
#include "zb_bfgs_coop.cuh"
#include "zb_bfgs_thread.cuh"
#include "zb_objective_visit.cuh"

namespace zb {

  namespace {
    constexpr int kThreadBlock = 128;
    constexpr int kMaxThreadDim = 10;

    // Runs up to which a run gets a warp of its own: `sure` whatever they do,
    // above that `per_iter` for each iteration they may take, up to `most`.
    //
    // A warp costs a run up to 32 times the lane work (a dual gradient is
    // formed whole in every lane) and spares one that iterates to MAX_ITER most
    // of its chain of trials.  While the warps hide each other's latencies the
    // first costs nothing: that is `sure`, lower where f and its gradient are
    // longer.  Above it the warp form is the faster one only if some run
    // iterates long, and by more the more iterations it may take.  A warp a run
    // against a thread a run (B200):
    //   Rosenbrock-2   3072 runs, 5 iterations 57 us both; 16384 runs, 10000
    //                  iterations 8.1 and 10.6 ms, 50 iterations 203 and 126 us;
    //                  32768 runs, 1000 iterations 1.41 and 1.26 ms
    //   Rosenbrock-8   1024, 50: 0.12 and 0.18 ms; 4096, 50: 0.28 and 0.18;
    //                  4096, 1000: 0.43 of the thread form's time; 32768, 1000:
    //                  1.15 of it; 65536, 10000: 0.45
    //   Ackley-2       6144, 5: 0.96; 32768, 50: 0.78; 32768, 10000: 0.26
    //   Ackley-10      4096: 0.76 to 1.0; 8192: 1.2 to 1.5, however many
    //                  iterations they may take (no run takes 100)
    //   likelihood     12288: 0.75 to 0.95; 16384: 1.0 to 1.2; 65536: 2.2 to 2.9
    //   dual gradients Rosenbrock-8 4096, 50: 1.8, 10000: 0.58; Ackley-10 1024:
    //                  0.88, 2048: 1.6; the likelihood 1024: 0.82 to 0.9, 4096: 2.2
    // Runs that all converge within tens of iterations pay above `sure` (65536
    // Rosenbrock-8 runs that start 0.05 from the minimum: 0.2 -> 1.6 ms); which
    // do is not known at the launch.
    // A quadratic form stays a thread a run: its first trial passes and its runs
    // converge at once (Gaussian-8, 200 runs: 35.5 us a thread, 38.3 a warp).
    struct WarpRule {
      int64_t sure, per_iter, most;
    };

    template <class F>
    constexpr WarpRule
    warp_rule(bool adjoint)
    {
      constexpr int D = (int)F::arity;
      if (F::kind == ZEUS_OBJ_POISSON_NLL)
        return adjoint ? WarpRule{12288, 0, 0} : WarpRule{1024, 0, 0};
      if (F::kind == ZEUS_OBJ_ROSENBROCK) {
        const int64_t slope = 160 / D < 40 ? 160 / D : 40;
        return {8192 / D < 3072 ? 8192 / D : 3072, adjoint ? slope : slope * 3 / 4,
                D == 2 ? 16384 : 16384 * D};
      }
      // transcendental terms: longer trials
      if (F::kind == ZEUS_OBJ_ACKLEY && D > 2)
        return adjoint ? WarpRule{4096, 0, 0} : WarpRule{1024, 0, 0};
      return adjoint ? WarpRule{D <= 2 ? 6144 : 4096, 1600 / D, 16384 * D}
                     : WarpRule{D <= 2 ? 2048 : 1024, 960 / (D * D), D <= 2 ? 32768 : 65536};
    }

    template <class F>
    bool
    warp_per_run(bool adjoint, int max_iter, int64_t n)
    {
      if constexpr (QuadraticForm<F>)
        return false;
      constexpr WarpRule adj = warp_rule<F>(true), dual = warp_rule<F>(false);
      const WarpRule& r = adjoint ? adj : dual;
      return n <= r.sure || (n <= r.most && n <= r.per_iter * max_iter);
    }

    template <class F, int D, bool Adjoint>
    int
    launch_warp(const F& f, const BfgsParams& prm, const double* starts, const RunOut& out,
                Control* ctl, cudaStream_t st)
    {
      constexpr int per = kThreadGroupBlock / 32; // runs a block
      bfgs_thread_warp_kernel<F, D, Adjoint>
        <<<(unsigned)((prm.n + per - 1) / per), kThreadGroupBlock, 0, st>>>(f, prm, starts,
                                                                           out, ctl);
      return cuda_fail(cudaGetLastError(), "warp-per-run BFGS launch");
    }
  } // namespace

  bool
  thread_layout_warps(int kind, int dim, int gradient, int max_iter, int64_t n)
  {
    Objective o{kind, dim, nullptr, nullptr, 0, 0, nullptr};
    return visit_objective(o, [&](auto f) -> int {
             using F = decltype(f);
             if constexpr ((int)F::arity <= kMaxThreadDim)
               return warp_per_run<F>(gradient == ZEUS_GRAD_ADJOINT, max_iter, n) ? 1 : 0;
             return 0;
           }) == 1;
  }

  extern "C" int
  zeus_internal_thread_layout_warps(int kind, int dim, int gradient, int max_iter, int64_t n)
  {
    return thread_layout_warps(kind, dim, gradient, max_iter, n);
  }

  bool
  thread_layout_supported(int kind, int dim)
  {
    return builtin_supported(kind, dim) && dim <= kMaxThreadDim;
  }

  int
  launch_thread(const Objective& o, const zeus_bfgs_config& c,
                const BfgsParams& prm, const double* starts, const RunOut& out,
                Control* ctl, cudaStream_t st)
  {
    const bool adjoint = c.gradient == ZEUS_GRAD_ADJOINT;
    return visit_objective(o, [&](auto f) -> int {
      using F = decltype(f);
      constexpr int D = (int)F::arity;
      if constexpr (D <= kMaxThreadDim) {
        const int block = c.block > 0 ? c.block : kThreadBlock;
        const unsigned grid = (unsigned)((prm.n + block - 1) / block);
        // the cycle timers are compiled in only where they are asked for
        const bool timed = out.cycles != nullptr;
        // (a block size asked for names the thread form)
        if constexpr (!QuadraticForm<F>)
          if (!timed && (c.block == kBlockWarps ||
                         (c.block <= 0 && warp_per_run<F>(adjoint, prm.max_iter, prm.n))))
            return adjoint ? launch_warp<F, D, true>(f, prm, starts, out, ctl, st)
                           : launch_warp<F, D, false>(f, prm, starts, out, ctl, st);
        if (adjoint && timed)
          bfgs_thread_kernel<F, D, true, true>
            <<<grid, block, 0, st>>>(f, prm, starts, out, ctl);
        else if (adjoint)
          bfgs_thread_kernel<F, D, true>
            <<<grid, block, 0, st>>>(f, prm, starts, out, ctl);
        else if (timed)
          bfgs_thread_kernel<F, D, false, true>
            <<<grid, block, 0, st>>>(f, prm, starts, out, ctl);
        else
          bfgs_thread_kernel<F, D, false>
            <<<grid, block, 0, st>>>(f, prm, starts, out, ctl);
        return cuda_fail(cudaGetLastError(), "thread-layout BFGS launch");
      } else {
        set_error("thread layout: dim %d not built", D);
        return ZEUS_E_UNSUPPORTED;
      }
    });
  }

} // namespace zb
