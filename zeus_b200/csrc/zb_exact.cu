// Exact-mode BFGS and PSO launchers.  Compiled with -fmad=false (see
// zeus_b200/build.py): no multiply-add contraction, so every basic
// operation rounds as in the reference built for the host.
#include "zb_bfgs_exact.cuh"
#include "zb_objective_visit.cuh"
#include "zb_pso.cuh"
#include "zb_pso_dmma.cuh"
#include "zb_pso_swarm.cuh"

namespace zb {

  namespace {
    constexpr int kExactBlock = 128;

    int
    exact_grid(int64_t n)
    {
      const int64_t g = (int64_t)sm_count() * 4;
      return (int)(n < g ? n : g);
    }

    // A warp per run up to D = 16; above, where a run's O(D^3) update is most
    // of its time, only with more runs than two to an SM: below that a block's
    // four warps on a run are the faster ones (Gaussian-32, 32 runs: 310 us
    // against 350; 512 runs: 782 against 474).  The same line for the Poisson
    // likelihood, whose evaluations take the same time in either form (100
    // runs: 20.9 ms a block, 21.4 a warp).
    bool
    exact_warp_form(int kind, int dim, int64_t n)
    {
      if (dim > kExactWarpMaxDim)
        return false;
      return (dim <= 16 && kind != ZEUS_OBJ_POISSON_NLL) || n > 2 * (int64_t)sm_count();
    }
  } // namespace

  bool
  exact_supported(int kind, int dim)
  {
    return builtin_supported(kind, dim);
  }

  size_t
  exact_workspace_bytes(const Objective& o, int64_t n)
  {
    if (n <= 0)
      return 0;
    // what the block form takes, in either form's range: a workspace sized
    // for many runs serves a later launch of few
    return sizeof(double) * 2 * (size_t)o.dim * o.dim * exact_grid(n);
  }

  int
  launch_exact(const Objective& o, const BfgsParams& prm,
               const double* starts, const RunOut& out, Control* ctl,
               void* ws, size_t ws_bytes, cudaStream_t st)
  {
    if (prm.n <= 0)
      return ZEUS_OK;
    const size_t need = exact_workspace_bytes(o, prm.n);
    if (ws_bytes < need || !ws) {
      set_error("exact BFGS needs %zu workspace bytes, got %zu", need,
                ws_bytes);
      return ZEUS_E_WORKSPACE;
    }
    const bool traj = out.traj_x && out.traj_f && out.traj_g &&
                      out.traj_status;
    return visit_objective(o, [&](auto f) -> int {
      using F = decltype(f);
      constexpr int D = (int)F::arity;
      if constexpr (D <= kExactWarpMaxDim) {
        if (exact_warp_form(F::kind, D, prm.n)) {
          constexpr int per = kExactWarpBlock / 32; // runs a block
          constexpr size_t wsm = sizeof(double) * per * ExactWarpShape<D>::doubles;
          auto kern = traj ? bfgs_exact_warp_kernel<F, D, true>
                           : bfgs_exact_warp_kernel<F, D, false>;
          if constexpr (wsm > 48 * 1024)
            if (int rc = cuda_fail(cudaFuncSetAttribute(
                                     kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)wsm),
                                   "exact BFGS shared memory attribute"))
              return rc;
          kern<<<(unsigned)((prm.n + per - 1) / per), kExactWarpBlock, wsm, st>>>(
            f, prm, starts, out, ctl);
          return cuda_fail(cudaGetLastError(), "exact BFGS launch");
        }
      }
      const int grid = exact_grid(prm.n);
      const size_t smem = exact_smem_bytes<D>();
      double* scratch = static_cast<double*>(ws);
      if (traj)
        bfgs_exact_kernel<F, D, true>
          <<<grid, kExactBlock, smem, st>>>(f, prm, starts, out, ctl, scratch);
      else
        bfgs_exact_kernel<F, D, false>
          <<<grid, kExactBlock, smem, st>>>(f, prm, starts, out, ctl, scratch);
      return cuda_fail(cudaGetLastError(), "exact BFGS launch");
    });
  }

  bool
  pso_supported(int kind, int dim)
  {
    return builtin_supported(kind, dim);
  }

  size_t
  pso_workspace_bytes(int64_t n, int dim)
  {
    const int64_t blocks = pso_blocks(n, dim);
    size_t b = 0;
    b += align_up(sizeof(double) * (size_t)n * dim); // X
    b += align_up(sizeof(double) * (size_t)n * dim); // V
    b += align_up(sizeof(unsigned long long) * (size_t)blocks);
    b += align_up(sizeof(int) * (size_t)blocks);
    b += align_up(sizeof(unsigned int));
    return b;
  }

  namespace {
    // Particles a block of the one-launch PSO takes; 0: the swarm does not fit,
    // and each iteration is a launch.  A block holds at least kSwarmElems (particle, coordinate)
    // elements, so a small swarm is one block and needs no meeting, and a
    // large one is spread over the SMs.
    constexpr int64_t kSwarmElems = 1024;
    // bins up to which a likelihood's swarm is one launch: the blocks that wait
    // for the slowest evaluation (some 10 ms) are then far from their limit,
    // and a launch an iteration is nothing beside longer ones
    constexpr int kSwarmMaxBins = 8192;

    template <class F, int D>
    int
    swarm_per_block(const F& f, int64_t n, int iters, cudaStream_t st)
    {
      constexpr int64_t limit = kSwarmSmem / sizeof(double);
      if (!swarm_built<F, D>() || iters < 1)
        return 0; // nothing to meet for
      if constexpr (F::kind == ZEUS_OBJ_POISSON_NLL)
        if (f.nbins > kSwarmMaxBins)
          return 0;
      const int64_t least = (kSwarmElems + D - 1) / D;
      // the blocks wait for one another, so there are no more than the stream
      // has SMs (a graph that records the launch has no other check)
      const int64_t has = n > least ? stream_sm_count(st) : 1;
      const int64_t sms = has < kSwarmMaxBlocks ? has : kSwarmMaxBlocks;
      int64_t per = (n + sms - 1) / sms;
      per = per > least ? per : least;
      per = per < n ? per : n;
      if constexpr (swarm_dmma<F, D>()) {
        per = (per + kPsoDmmaParticles - 1) / kPsoDmmaParticles * kPsoDmmaParticles;
        // eight particles and C to a block: with C in L2 the blocks of a
        // launch an iteration hide its latency better, several to an SM
        // (4096 particles at D = 150: 213 us that way, 234 this way)
        if (per > kPsoDmmaParticles)
          return 0;
      }
      if (per > swarm_threads<F, D>() || (int64_t)swarm_doubles<F, D>(per) > limit)
        return 0;
      return (int)per;
    }

    template <class F, int D>
    int
    launch_swarm(const F& f, const SwarmArgs& a, unsigned blocks, cudaStream_t st)
    {
      auto kern = pso_swarm_kernel<F, D>;
      const size_t smem = sizeof(double) * swarm_doubles<F, D>(a.per_block);
      int rc = ZEUS_OK;
      // the most a swarm takes, not what this one takes: the attribute is the
      // kernel's, and a smaller swarm on another thread would lower it between
      // this call's setting it and its launch
      if (smem > 40 * 1024 &&
          (rc = cuda_fail(cudaFuncSetAttribute(
                            kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)kSwarmSmem),
                          "PSO shared memory attribute")))
        return rc;
      if (blocks > 1 &&
          (rc = cuda_fail(cudaMemsetAsync(a.slots, 0,
                                          sizeof(unsigned long long) * 8 * blocks, st),
                          "PSO slot reset")))
        return rc;
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeCooperative;
      attr.val.cooperative = 1;
      cudaLaunchConfig_t lc{};
      lc.gridDim = dim3(blocks);
      lc.blockDim = dim3(swarm_threads<F, D>());
      lc.dynamicSmemBytes = smem;
      lc.stream = st;
      lc.attrs = &attr;
      lc.numAttrs = blocks > 1 ? 1 : 0;
      const cudaError_t e = cudaLaunchKernelEx(&lc, kern, f, a);
      if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError(); // no room for all blocks at once after all
        return kPsoNotOne;
      }
      return cuda_fail(e, "PSO launch");
    }
  } // namespace

  extern "C" int*
  zeus_internal_swarm_wait(void)
  {
    static thread_local int wait = kSwarmWait;
    return &wait;
  }

  int
  launch_pso(const Objective& o, uint64_t seed, int64_t n, double lower,
             double upper, int iters, double w, double c1, double c2,
             double* pbx, double* pbf, double* gbest, void* ws,
             size_t ws_bytes, cudaStream_t st, const uint32_t* sobol, PsoPath path)
  {
    if (n <= 0)
      return ZEUS_OK;
    const size_t need = pso_workspace_bytes(n, o.dim);
    if (!ws || ws_bytes < need) {
      set_error("PSO needs %zu workspace bytes, got %zu", need, ws_bytes);
      return ZEUS_E_WORKSPACE;
    }
    const int64_t blocks = pso_blocks(n, o.dim);
    char* p = static_cast<char*>(ws);
    PsoWork wk;
    wk.X = reinterpret_cast<double*>(p);
    p += align_up(sizeof(double) * (size_t)n * o.dim);
    wk.V = reinterpret_cast<double*>(p);
    p += align_up(sizeof(double) * (size_t)n * o.dim);
    wk.part_key = reinterpret_cast<unsigned long long*>(p);
    p += align_up(sizeof(unsigned long long) * (size_t)blocks);
    wk.part_idx = reinterpret_cast<int*>(p);
    p += align_up(sizeof(int) * (size_t)blocks);
    wk.counter = reinterpret_cast<unsigned int*>(p);
    wk.gbest = gbest;
    wk.sobol = sobol;
    return visit_objective(o, [&](auto f) -> int {
      using F = decltype(f);
      constexpr int D = (int)F::arity;
      if constexpr (swarm_built<F, D>())
        if (const int per = path == PsoPath::steps ? 0
                                                   : swarm_per_block<F, D>(f, n, iters, st)) {
          // the slots lie in the workspace: 2 x (32 + 8 D) bytes a block of
          // at least 1024 / D particles, within the positions' and velocities'
          // 16 D n bytes
          const unsigned nb = (unsigned)((n + per - 1) / per);
          SwarmArgs a{n,     per, iters, lower, upper, w, c1, c2, seed, sobol, pbx, pbf, gbest,
                      static_cast<unsigned long long*>(ws), nullptr,
                      *zeus_internal_swarm_wait()};
          a.slot_x = reinterpret_cast<double*>(a.slots + 8 * (size_t)nb);
          const int rc = launch_swarm<F, D>(f, a, nb, st);
          if (rc != kPsoNotOne)
            return rc;
        }
      if (path == PsoPath::one)
        return kPsoNotOne;
      pso_reset_kernel<D><<<1, 256, 0, st>>>(wk);
      if constexpr (D >= kPsoCoopMinDim && D <= kPsoDmmaMaxDim &&
                    F::kind == ZEUS_OBJ_GAUSSIAN) {
        // f = 0.5 x^T C x for 8 particles per warp on the FP64 tensor cores
        const unsigned b8 = (unsigned)pso_dmma_blocks(n);
        pso_init_dmma_kernel<D><<<b8, kPsoBlock, 0, st>>>(f, n, lower, upper, seed,
                                                          wk, pbx, pbf);
        for (int t = 1; t <= iters; ++t)
          pso_iter_dmma_kernel<D><<<b8, kPsoBlock, 0, st>>>(f, n, w, c1, c2, seed, t,
                                                            wk, pbx, pbf);
      } else if constexpr (D >= kPsoCoopMinDim) {
        pso_init_coop_kernel<F, D><<<(unsigned)blocks, kPsoBlock, 0, st>>>(
          f, n, lower, upper, seed, wk, pbx, pbf);
        for (int t = 1; t <= iters; ++t)
          pso_iter_coop_kernel<F, D><<<(unsigned)blocks, kPsoBlock, 0, st>>>(
            f, n, w, c1, c2, seed, t, wk, pbx, pbf);
      } else {
        pso_init_kernel<F, D><<<(unsigned)blocks, kPsoBlock, 0, st>>>(
          f, n, lower, upper, seed, wk, pbx, pbf);
        for (int t = 1; t <= iters; ++t)
          pso_iter_kernel<F, D><<<(unsigned)blocks, kPsoBlock, 0, st>>>(
            f, n, w, c1, c2, seed, t, wk, pbx, pbf);
      }
      return cuda_fail(cudaGetLastError(), "PSO launch");
    });
  }

} // namespace zb
