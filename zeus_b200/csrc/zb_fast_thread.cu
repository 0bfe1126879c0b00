// Thread-layout fast BFGS launcher (D <= 10).
#include "zb_bfgs_coop.cuh"
#include "zb_bfgs_thread.cuh"
#include "zb_objective_visit.cuh"

namespace zb {

  namespace {
    constexpr int kThreadBlock = 128;
    constexpr int kMaxThreadDim = 10;

    // Runs up to which a run gets a warp of its own.  The bulk of the runs,
    // which converge within tens of iterations, costs a warp form up to 32
    // times the lane work, the runs that iterate to MAX_ITER a fraction of the
    // time; at D = 2 the two balance near 60 000 runs (Rosenbrock: 8.1 against
    // 10.6 ms at 16384 runs, 19.1 against 17.8 at 65536), and the line moves
    // up with D, as trials and gradients grow (D = 4: 18.4 against 33.0 ms at
    // 65536; D = 8: 53 against 141 at 131072).  A quadratic form stays a
    // thread per run: its first trial passes and its runs converge at once
    // (Gaussian-8, 200 runs: 35.5 us a thread, 38.3 a warp).
    template <class F>
    bool
    warp_per_run(int64_t n)
    {
      return n <= (int64_t)16384 * (int)F::arity;
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
          if (!timed && c.block <= 0 && warp_per_run<F>(prm.n))
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
