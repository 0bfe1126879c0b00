// C ABI (include/zeus_b200.h): validation, workspace layout, PSO graph
// capture, reductions and the host-buffer orchestration of zeus_optimize.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>
#include <cuda.h>

#include "zb_internal.h"
#include "zb_objective_visit.cuh"
#include "zb_philox.cuh"
#include "zb_sobol.cuh"
#include "zb_reduce.cuh"

namespace zb {

  namespace {
    thread_local char g_err[1024] = "";
  }

  void
  set_error(const char* fmt, ...)
  {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
  }

  int
  cuda_fail(cudaError_t e, const char* what)
  {
    if (e == cudaSuccess)
      return ZEUS_OK;
    set_error("%s: %s", what, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? ZEUS_E_NOMEM : ZEUS_E_CUDA;
  }

  int
  stream_sm_count(cudaStream_t st)
  {
    struct Driver {
      decltype(&cuStreamGetGreenCtx) green = nullptr;
      decltype(&cuGreenCtxGetDevResource) green_sms = nullptr;
      decltype(&cuCtxGetCurrent) current = nullptr;
      decltype(&cuCtxGetDevResource) sms = nullptr;
      Driver()
      {
        const auto get = [](const char* name, auto& fn) {
          cudaDriverEntryPointQueryResult q;
          void* p = nullptr;
          if (cudaGetDriverEntryPointByVersion(name, &p, 12040, cudaEnableDefault, &q) ==
                cudaSuccess &&
              q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(p);
          else
            cudaGetLastError();
        };
        get("cuStreamGetGreenCtx", green);
        get("cuGreenCtxGetDevResource", green_sms);
        get("cuCtxGetCurrent", current);
        get("cuCtxGetDevResource", sms);
      }
    };
    static const Driver d;
    int n = sm_count();
    const auto least = [&](CUresult r, const CUdevResource& res) {
      if (r == CUDA_SUCCESS && (int)res.sm.smCount > 0 && (int)res.sm.smCount < n)
        n = (int)res.sm.smCount;
    };
    CUdevResource res{};
    CUgreenCtx g = nullptr;
    // (the default streams have the current context)
    if (d.green && d.green_sms && st && st != cudaStreamLegacy && st != cudaStreamPerThread &&
        d.green(st, &g) == CUDA_SUCCESS && g) {
      least(d.green_sms(g, &res, CU_DEV_RESOURCE_TYPE_SM), res);
      return n;
    }
    CUcontext ctx = nullptr;
    if (d.current && d.sms && d.current(&ctx) == CUDA_SUCCESS && ctx)
      least(d.sms(ctx, &res, CU_DEV_RESOURCE_TYPE_SM), res);
    return n;
  }

  int
  swarm_gave_up()
  {
    set_error("PSO: the swarm's blocks waited for one another past their limit; "
              "the swarm is incomplete");
    return ZEUS_E_CUDA;
  }

  int
  sm_count()
  {
    static std::mutex mu;
    static std::map<int, int> cache;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess)
      return 148;
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(dev);
    if (it != cache.end())
      return it->second;
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) !=
          cudaSuccess ||
        v <= 0)
      v = 148;
    cache[dev] = v;
    return v;
  }

  // The census of a launch: one block, or a cluster of kCensusBlocks whose
  // counts and minima meet in the first one's shared memory (no workspace, one
  // launch).  A group of G lanes (the power of two at or above dim, at most a
  // warp) takes a run's coordinates, kCensusRuns runs in flight a group; its
  // sum of squares is the xor tree of a warp whose lanes past G add zeros,
  // for any G.  One block with a warp a run waited for one load after another:
  // 16384 runs of 10 coordinates 255 -> 24 us, 131072 of 4 2.0 ms -> 50 us,
  // 1 000 000 of 10 15.9 -> 1.2 ms (B200); up to 2048 runs a cluster's launch
  // costs what it saves.
  inline constexpr int kCensusBlocks = 8;
  inline constexpr int kCensusRuns = 4;
  inline constexpr int64_t kCensusOneBlock = 2048; // runs up to which one block does

  template <int G>
  __global__ void __launch_bounds__(1024)
    census_kernel(const double* __restrict__ fval, const int32_t* __restrict__ status,
                  const double* __restrict__ x, int64_t n, int dim,
                  const __grid_constant__ KnownMin km, Census* out)
  {
    __shared__ int cnt[4];
    __shared__ unsigned long long best_key;
    __shared__ int best_idx;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 4)
      cnt[threadIdx.x] = 0;
    __syncthreads();
    unsigned long long key = ~0ull;
    int idx = 0x7fffffff;
    int actual = 0, claimed = 0, stopped = 0, surr = 0;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t threads = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 4
    for (int64_t i = tid; i < n; i += threads) {
      const unsigned long long k = order_key(fval[i]);
      if (k < key || (k == key && (int)i < idx)) {
        key = k;
        idx = (int)i;
      }
      const int st = status[i];
      if (st == kConverged)
        ++claimed;
      else if (st == kStopped)
        ++stopped;
      else
        ++surr;
    }
    if (x) {
      // converged runs within 0.5 of the known minimum
      const int64_t groups = threads / G;
      const int m = threadIdx.x % G;
      for (int64_t i0 = tid / G; i0 - lane / G < n; i0 += groups * kCensusRuns) {
        double ss[kCensusRuns];
        bool conv[kCensusRuns];
#pragma unroll
        for (int r = 0; r < kCensusRuns; ++r) {
          const int64_t i = i0 + r * groups;
          conv[r] = i < n && status[i] == kConverged;
        }
#pragma unroll
        for (int r = 0; r < kCensusRuns; ++r) {
          const int64_t i = i0 + r * groups;
          ss[r] = 0.0;
          if (conv[r])
            for (int d = m; d < dim; d += G) {
              const double df = x[i * dim + d] - (km.has ? km.x[d] : 0.0);
              ss[r] = fma(df, df, ss[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < kCensusRuns; ++r) {
#pragma unroll
          for (int o = G / 2; o > 0; o >>= 1)
            ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], o);
          if (m == 0 && conv[r] && sqrt(ss[r]) < 0.5)
            ++actual;
        }
      }
    }
    const int sums[4] = {__reduce_add_sync(0xffffffffu, actual),
                         __reduce_add_sync(0xffffffffu, claimed),
                         __reduce_add_sync(0xffffffffu, surr),
                         __reduce_add_sync(0xffffffffu, stopped)};
    if (lane == 0)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (sums[q])
          atomicAdd(&cnt[q], sums[q]);
    block_argmin(key, idx);
    if (threadIdx.x == 0) {
      best_key = key;
      best_idx = idx;
    }
    __syncthreads();
    const cg::cluster_group cluster = cg::this_cluster();
    const int nb = (int)gridDim.x; // the grid is one cluster
    if (nb > 1)
      cluster.sync();
    if (cluster.block_rank() == 0 && threadIdx.x == 0) {
      int total[4] = {cnt[0], cnt[1], cnt[2], cnt[3]};
      for (int b = 1; b < nb; ++b) {
        const int* c = cluster.map_shared_rank(cnt, b);
        for (int q = 0; q < 4; ++q)
          total[q] += c[q];
        const unsigned long long k = *cluster.map_shared_rank(&best_key, b);
        const int ki = *cluster.map_shared_rank(&best_idx, b);
        if (k < key || (k == key && ki < idx)) {
          key = k;
          idx = ki;
        }
      }
      out->actual = total[0];
      out->claimed = total[1];
      out->surrendered = total[2];
      out->stopped = total[3];
      out->best_idx = (n > 0 && idx != 0x7fffffff) ? idx : -1;
      out->reserved = 0;
    }
    if (nb > 1)
      cluster.sync(); // the first block has read the others' shared memory
  }

  __global__ void
  nll_bins_kernel(const double* __restrict__ centres,
                  const int* __restrict__ counts, int nbins,
                  double* __restrict__ bins)
  {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nbins)
      return;
    const double x = centres[i];
    const double k = (double)counts[i];
    bins[4 * i + 0] = ::log(x);
    bins[4 * i + 1] = ::log(1.0 - x);
    bins[4 * i + 2] = k;
    bins[4 * i + 3] = ::lgamma(k + 1.0);
  }

  // Start points.  An item is a pair of neighbouring coordinates of one run
  // (Philox: one block of random words serves both) or one coordinate of
  // kSobolRuns consecutive runs (Sobol': their points differ in the low bits
  // of the run index alone, so the shift and the high bits' directions are
  // found once).  `items` a run or chunk of runs; a thread walks the items
  // with a fixed stride whose quotient and remainder by `items` are given, so
  // it divides once.  What bounds it is the ten Philox rounds and the 64-bit
  // conversions: 1 000 003 runs of 10 coordinates (80 MB) 58 -> 21 us against a
  // thread, a Philox block and a 64-bit division an element; 100 000 Sobol'
  // points of 150 coordinates 417 -> 69 us (B200).
  inline constexpr int kSobolRuns = 8;
  inline constexpr int kStartsBlock = 256;

  template <bool Sobol, bool Pairs>
  __global__ void __launch_bounds__(kStartsBlock)
    starts_kernel(uint64_t seed, int64_t n, int dim, double lower, double upper,
                  double* __restrict__ out, const uint32_t* __restrict__ sobol,
                  int64_t total, int items, int64_t step_q, int step_r)
  {
    const int64_t first = (int64_t)blockIdx.x * kStartsBlock + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * kStartsBlock;
    const double width = upper - lower;
    // no contraction: the same bits as lower + (upper - lower) * u in C
    const auto place = [&](double u) { return __dadd_rn(lower, __dmul_rn(width, u)); };
    int64_t i = first / items;
    int b = (int)(first - i * items);
    for (int64_t e = first; e < total; e += stride) {
      if constexpr (Sobol) {
        const int64_t run = i * kSobolRuns;
        const uint32_t* v = sobol + (size_t)b * kSobolBits;
        uint32_t x = sobol_shift(seed, (uint32_t)b);
        for (uint32_t m = (uint32_t)run; m; m &= m - 1u)
          x ^= v[ctz32(m)];
        const uint32_t v0 = v[0], v1 = v[1], v2 = v[2];
        const int cnt = (int)(n - run < kSobolRuns ? n - run : kSobolRuns);
        double* o = out + run * dim + b;
#pragma unroll
        for (int r = 0; r < kSobolRuns; ++r) {
          const uint32_t y =
            x ^ ((r & 1) ? v0 : 0u) ^ ((r & 2) ? v1 : 0u) ^ ((r & 4) ? v2 : 0u);
          if (r < cnt)
            o[(int64_t)r * dim] = place(((double)y + 0.5) * (1.0 / 4294967296.0));
        }
      } else {
        uint32_t w[4];
        philox4x32_10((uint32_t)i, (uint32_t)b, kTagStarts, (uint32_t)((uint64_t)i >> 32),
                      (uint32_t)seed, (uint32_t)(seed >> 32), w);
        const double u0 = place(uniform01_word(w[0], w[1]));
        const double u1 = place(uniform01_word(w[2], w[3]));
        double* o = out + i * dim + 2 * b;
        if constexpr (Pairs) {
          *reinterpret_cast<double2*>(o) = make_double2(u0, u1);
        } else {
          o[0] = u0;
          if (2 * b + 1 < dim)
            o[1] = u1;
        }
      }
      i += step_q;
      b += step_r;
      if (b >= items) {
        b -= items;
        ++i;
      }
    }
  }

  // The best run (the census's best_idx) beside the census, so that a host
  // call reads both with one copy: census (3 doubles) | gbest's value (0
  // without a swarm) | fval | ||g|| | status, iter | x[dim].
  inline constexpr int kBestHead = 3 + 4;

  __global__ void __launch_bounds__(128)
    best_run_kernel(const Census* __restrict__ cen, const double* __restrict__ fval,
                    const double* __restrict__ gnorm, const int32_t* __restrict__ status,
                    const int32_t* __restrict__ iter, const double* __restrict__ x, int dim,
                    const double* __restrict__ gbest, double* __restrict__ pack)
  {
    const int b = cen->best_idx;
    if (threadIdx.x == 0) {
      *reinterpret_cast<Census*>(pack) = *cen;
      pack[3] = gbest ? gbest[0] : 0.0;
    }
    if (b < 0)
      return;
    if (threadIdx.x == 0) {
      pack[4] = fval[b];
      pack[5] = gnorm[b];
      reinterpret_cast<int32_t*>(pack + 6)[0] = status[b];
      reinterpret_cast<int32_t*>(pack + 6)[1] = iter[b];
    }
    for (int d = threadIdx.x; d < dim; d += blockDim.x)
      pack[kBestHead + d] = x[(int64_t)b * dim + d];
  }

  __global__ void __launch_bounds__(256)
    fp64_probe_kernel(int64_t iters, double* __restrict__ sink)
  {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double a0 = 1.0 + t * 1e-9, a1 = a0 + 1e-3, a2 = a0 + 2e-3, a3 = a0 + 3e-3;
    double a4 = a0 + 4e-3, a5 = a0 + 5e-3, a6 = a0 + 6e-3, a7 = a0 + 7e-3;
    const double m = 0.999999999, c = 1e-9;
    for (int64_t i = 0; i < iters; ++i) {
      a0 = fma(a0, m, c);
      a1 = fma(a1, m, c);
      a2 = fma(a2, m, c);
      a3 = fma(a3, m, c);
      a4 = fma(a4, m, c);
      a5 = fma(a5, m, c);
      a6 = fma(a6, m, c);
      a7 = fma(a7, m, c);
    }
    sink[t] = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  }

  namespace {

    int
    check_problem(const zeus_problem* p)
    {
      if (!p) {
        set_error("problem is NULL");
        return ZEUS_E_INVALID;
      }
      if (!builtin_supported(p->kind, p->dim)) {
        set_error("objective kind %d with dim %d is not built", p->kind,
                  p->dim);
        return ZEUS_E_UNSUPPORTED;
      }
      if (p->kind == ZEUS_OBJ_GAUSSIAN && !p->data) {
        set_error("Gaussian objective needs its matrix (data)");
        return ZEUS_E_INVALID;
      }
      if (p->kind == ZEUS_OBJ_POISSON_NLL &&
          (!p->data || !p->idata || p->ndata <= 0)) {
        set_error("Poisson NLL needs centres, counts and ndata > 0");
        return ZEUS_E_INVALID;
      }
      return ZEUS_OK;
    }

    // The Sobol' direction table for generator `prng` on the current
    // device, or null for the Philox ones.
    int
    prng_table(int prng, int dim, const uint32_t** sobol)
    {
      *sobol = nullptr;
      if (prng == ZEUS_PRNG_XORWOW || prng == ZEUS_PRNG_PHILOX)
        return ZEUS_OK;
      if (prng != ZEUS_PRNG_SOBOL) {
        set_error("generator %d is not ZEUS_PRNG_XORWOW, _PHILOX or _SOBOL",
                  prng);
        return ZEUS_E_INVALID;
      }
      if (dim > kSobolMaxDim) {
        set_error("Sobol' starts are built for dim <= %d, got %d",
                  kSobolMaxDim, dim);
        return ZEUS_E_UNSUPPORTED;
      }
      return sobol_table_device(sobol);
    }

    Objective
    to_objective(const zeus_problem* p, const double* nll_bins)
    {
      Objective o;
      o.kind = p->kind;
      o.dim = p->dim;
      o.data = p->data;
      o.idata = p->idata;
      o.ndata = p->ndata;
      o.flags = p->flags;
      o.nll_bins = nll_bins;
      return o;
    }

    size_t
    nll_bytes(const zeus_problem* p)
    {
      return p->kind == ZEUS_OBJ_POISSON_NLL
               ? align_up(sizeof(double) * 4 * (size_t)p->ndata)
               : 0;
    }

    int
    check_config(const zeus_bfgs_config* c)
    {
      if (!c) {
        set_error("config is NULL");
        return ZEUS_E_INVALID;
      }
      if (c->max_iter < 0) {
        set_error("max_iter must be >= 0");
        return ZEUS_E_INVALID;
      }
      if (c->mode != ZEUS_MODE_EXACT && c->mode != ZEUS_MODE_FAST) {
        set_error("unknown mode %d", c->mode);
        return ZEUS_E_INVALID;
      }
      if (c->gradient != ZEUS_GRAD_DUAL && c->gradient != ZEUS_GRAD_ADJOINT) {
        set_error("unknown gradient %d", c->gradient);
        return ZEUS_E_INVALID;
      }
      if (c->mode == ZEUS_MODE_EXACT && c->gradient != ZEUS_GRAD_DUAL) {
        set_error("exact mode uses dual gradients only");
        return ZEUS_E_INVALID;
      }
      if (!(c->tolerance >= 0.0)) {
        set_error("tolerance must be >= 0");
        return ZEUS_E_INVALID;
      }
      return ZEUS_OK;
    }

    size_t
    kernel_ws(const zeus_problem* p, const zeus_bfgs_config* c, int64_t n)
    {
      Objective o = to_objective(p, nullptr);
      return c->mode == ZEUS_MODE_EXACT ? exact_workspace_bytes(o, n)
                                        : fast_workspace_bytes(o, *c, n);
    }

    // Autotuned layouts: (device, kind, dim, gradient) -> (layout, tile), for
    // batches and for launches whose thread layout has a thread a run (0), for
    // launches whose thread layout has a warp a run (1), and the one of them
    // that was reported (2).
    struct TuneTable {
      std::mutex mu;
      std::map<std::tuple<int, int, int, int>, std::pair<int, int>> m[3];
    };
    TuneTable&
    tune_table()
    {
      static TuneTable* t = new TuneTable;
      return *t;
    }

    // The library's own stream-ordered memory pool per device, for the
    // buffers a host-buffer call (zeus_optimize, the autotuner) allocates
    // and frees each time: its release threshold keeps the memory reserved
    // between calls, so a repeated call maps nothing new (the device's
    // default pool returns freed memory at every synchronisation, and the
    // next call's allocations then cost milliseconds).  The pool is never
    // destroyed; what it holds is at most the largest call's buffers.
    int
    pool_alloc(void** out, size_t bytes, cudaStream_t st)
    {
      static std::mutex mu;
      static std::map<int, cudaMemPool_t> pools;
      int dev = 0;
      cudaError_t e = cudaGetDevice(&dev);
      if (e != cudaSuccess)
        return cuda_fail(e, "current device");
      cudaMemPool_t pool = nullptr;
      {
        std::lock_guard<std::mutex> lk(mu);
        auto it = pools.find(dev);
        if (it == pools.end()) {
          cudaMemPoolProps props{};
          props.allocType = cudaMemAllocationTypePinned;
          props.handleTypes = cudaMemHandleTypeNone;
          props.location.type = cudaMemLocationTypeDevice;
          props.location.id = dev;
          if ((e = cudaMemPoolCreate(&pool, &props)) != cudaSuccess)
            return cuda_fail(e, "memory pool");
          uint64_t keep = ~0ull;
          cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
          pools[dev] = pool;
        } else {
          pool = it->second;
        }
      }
      return cuda_fail(cudaMallocFromPoolAsync(out, bytes ? bytes : 1, pool, st),
                       "allocation");
    }

    int
    tune_lookup(int form, int kind, int dim, int gradient, int32_t* layout, int32_t* tile)
    {
      int dev = 0;
      if (cudaGetDevice(&dev) != cudaSuccess)
        return 0;
      TuneTable& t = tune_table();
      std::lock_guard<std::mutex> lk(t.mu);
      auto it = t.m[form].find(std::make_tuple(dev, kind, dim, gradient));
      if (it == t.m[form].end())
        return 0;
      if (layout)
        *layout = it->second.first;
      if (tile)
        *tile = it->second.second;
      return 1;
    }

    int
    tune_record(int form, int kind, int dim, int gradient, int layout, int tile)
    {
      if (layout < ZEUS_LAYOUT_THREAD || layout > ZEUS_LAYOUT_ROWS) {
        set_error("zeus_autotune_record: layout must be THREAD, TILE, CTA or ROWS");
        return ZEUS_E_INVALID;
      }
      int dev = 0;
      cudaGetDevice(&dev);
      TuneTable& t = tune_table();
      std::lock_guard<std::mutex> lk(t.mu);
      t.m[form][std::make_tuple(dev, kind, dim, gradient)] = {layout, tile};
      return ZEUS_OK;
    }

    // Cached executable graphs for the PSO loop, keyed by the launch shape;
    // new pointer arguments go in through cudaGraphExecUpdate.
    struct GraphCache {
      std::mutex mu;
      std::map<std::tuple<int, int, int, int64_t, int>, cudaGraphExec_t> m;
    };
    GraphCache&
    graph_cache()
    {
      static GraphCache* c = new GraphCache; // never destroyed: exit-safe
      return *c;
    }

  } // namespace

  int
  autotune_lookup(bool warps, int kind, int dim, int gradient, int* layout, int* tile)
  {
    return tune_lookup(warps ? 1 : 0, kind, dim, gradient, layout, tile);
  }
} // namespace zb

using namespace zb;

extern "C" {

const char*
zeus_last_error(void)
{
  return g_err;
}

const char*
zeus_version(void)
{
  return "zeus_b200 0.1.0 (sm_100a)";
}

int
zeus_supported(int32_t kind, int32_t dim, int32_t mode, int32_t gradient)
{
  if (mode == ZEUS_MODE_EXACT)
    return gradient == ZEUS_GRAD_DUAL && exact_supported(kind, dim);
  if (mode == ZEUS_MODE_FAST)
    return fast_supported(kind, dim, gradient);
  return 0;
}

int
zeus_starts(uint64_t seed, int32_t prng, int64_t n, int32_t dim, double lower,
            double upper, double* d_out, void* stream)
{
  if (n < 0 || dim <= 0 || (n > 0 && !d_out)) {
    set_error("zeus_starts: bad arguments");
    return ZEUS_E_INVALID;
  }
  const uint32_t* sobol = nullptr;
  int rc = prng_table(prng, dim, &sobol);
  if (rc)
    return rc;
  if (n == 0)
    return ZEUS_OK;
  const int items = sobol ? dim : (dim + 1) / 2;
  const int64_t total = (sobol ? (n + kSobolRuns - 1) / kSobolRuns : n) * items;
  const int64_t most = (int64_t)sm_count() * 8;
  const int64_t need = (total + kStartsBlock - 1) / kStartsBlock;
  const unsigned grid = (unsigned)(need < most ? need : most);
  const int64_t stride = (int64_t)grid * kStartsBlock;
  // pairs are stored as one where every pair is 16-byte aligned
  const bool pairs = dim % 2 == 0 && (reinterpret_cast<uintptr_t>(d_out) & 15u) == 0;
  auto kern = sobol ? starts_kernel<true, false>
                    : pairs ? starts_kernel<false, true> : starts_kernel<false, false>;
  kern<<<grid, kStartsBlock, 0, (cudaStream_t)stream>>>(
    seed, n, dim, lower, upper, d_out, sobol, total, items, stride / items,
    (int)(stride % items));
  return cuda_fail(cudaGetLastError(), "starts launch");
}

int
zeus_starts_uniform(uint64_t seed, int64_t n, int32_t dim, double lower,
                    double upper, double* d_out, void* stream)
{
  return zeus_starts(seed, ZEUS_PRNG_PHILOX, n, dim, lower, upper, d_out,
                     stream);
}

size_t
zeus_pso_workspace_size(int64_t n, int32_t dim)
{
  if (n <= 0 || dim <= 0)
    return 0;
  return pso_workspace_bytes(n, dim);
}

int
zeus_pso_device(const zeus_problem* problem, uint64_t seed, int64_t n,
                double lower, double upper, int32_t iters, double w,
                double c1, double c2, double* d_pbest_x, double* d_pbest_f,
                double* d_gbest, void* d_workspace, size_t workspace_bytes,
                void* stream)
{
  return zeus_pso_device_prng(problem, seed, ZEUS_PRNG_PHILOX, n, lower, upper,
                              iters, w, c1, c2, d_pbest_x, d_pbest_f, d_gbest,
                              d_workspace, workspace_bytes, stream);
}

int
zeus_pso_device_prng(const zeus_problem* problem, uint64_t seed, int32_t prng,
                     int64_t n, double lower, double upper, int32_t iters,
                     double w, double c1, double c2, double* d_pbest_x,
                     double* d_pbest_f, double* d_gbest, void* d_workspace,
                     size_t workspace_bytes, void* stream)
{
  int rc = check_problem(problem);
  if (rc)
    return rc;
  if (n < 0 || iters < 0 || (n > 0 && (!d_pbest_x || !d_pbest_f || !d_gbest))) {
    set_error("zeus_pso_device: bad arguments");
    return ZEUS_E_INVALID;
  }
  const uint32_t* sobol = nullptr;
  if ((rc = prng_table(prng, problem->dim, &sobol)))
    return rc;
  if (n == 0)
    return ZEUS_OK;
  if (n > 0x7fffffffLL) {
    set_error("zeus_pso_device: n must fit in int32");
    return ZEUS_E_INVALID;
  }
  Objective o = to_objective(problem, nullptr);
  cudaStream_t st = (cudaStream_t)stream;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (st)
    cudaStreamIsCapturing(st, &cs);
  const bool direct = !st || cs != cudaStreamCaptureStatusNone;
  rc = launch_pso(o, seed, n, lower, upper, iters, w, c1, c2, d_pbest_x, d_pbest_f, d_gbest,
                  d_workspace, workspace_bytes, st, sobol,
                  direct ? PsoPath::any : PsoPath::one);
  if (direct || rc != kPsoNotOne)
    return rc;
  // A launch an iteration: capture them into one graph and launch it.
  rc = cuda_fail(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal),
                 "PSO capture begin");
  if (rc)
    return rc;
  const int lrc =
    launch_pso(o, seed, n, lower, upper, iters, w, c1, c2, d_pbest_x,
               d_pbest_f, d_gbest, d_workspace, workspace_bytes, st, sobol,
               PsoPath::steps);
  cudaGraph_t graph = nullptr;
  const cudaError_t ec = cudaStreamEndCapture(st, &graph);
  if (lrc) {
    if (graph)
      cudaGraphDestroy(graph);
    return lrc;
  }
  if ((rc = cuda_fail(ec, "PSO capture end")))
    return rc;
  int dev = 0;
  cudaGetDevice(&dev);
  auto key = std::make_tuple(dev, o.kind, o.dim, n, (int)iters);
  GraphCache& gc = graph_cache();
  std::lock_guard<std::mutex> lk(gc.mu);
  cudaGraphExec_t exec = nullptr;
  auto it = gc.m.find(key);
  if (it != gc.m.end()) {
    cudaGraphExecUpdateResultInfo info;
    if (cudaGraphExecUpdate(it->second, graph, &info) == cudaSuccess)
      exec = it->second;
    else {
      cudaGetLastError();
      cudaStreamSynchronize(st);
      cudaGraphExecDestroy(it->second);
      gc.m.erase(it);
    }
  }
  if (!exec) {
    rc = cuda_fail(cudaGraphInstantiate(&exec, graph, 0), "PSO graph");
    if (rc) {
      cudaGraphDestroy(graph);
      return rc;
    }
    gc.m[key] = exec;
  }
  cudaGraphDestroy(graph);
  return cuda_fail(cudaGraphLaunch(exec, st), "PSO graph launch");
}

size_t
zeus_bfgs_workspace_size(const zeus_problem* problem,
                         const zeus_bfgs_config* config, int64_t n)
{
  if (check_problem(problem) || check_config(config) || n <= 0)
    return 0;
  return nll_bytes(problem) + align_up(kernel_ws(problem, config, n));
}

int
zeus_bfgs_device(const zeus_problem* problem, const zeus_bfgs_config* config,
                 const double* d_starts, int64_t n,
                 const zeus_run_outputs* out, int32_t* d_control,
                 void* d_workspace, size_t workspace_bytes, void* stream)
{
  int rc = check_problem(problem);
  if (rc)
    return rc;
  if ((rc = check_config(config)))
    return rc;
  if (n < 0 || n > 0x7fffffffLL || !out || (n > 0 && (!d_starts || !d_control))) {
    set_error("zeus_bfgs_device: bad arguments");
    return ZEUS_E_INVALID;
  }
  if (n == 0)
    return ZEUS_OK;
  if (config->mode == ZEUS_MODE_FAST &&
      !fast_supported(problem->kind, problem->dim, config->gradient)) {
    set_error("fast mode: kind %d dim %d not built", problem->kind,
              problem->dim);
    return ZEUS_E_UNSUPPORTED;
  }
  const size_t need = zeus_bfgs_workspace_size(problem, config, n);
  if (need > 0 && (!d_workspace || workspace_bytes < need)) {
    set_error("zeus_bfgs_device: workspace of %zu bytes needed, got %zu",
              need, workspace_bytes);
    return ZEUS_E_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  char* ws = static_cast<char*>(d_workspace);
  const double* bins = nullptr;
  if (problem->kind == ZEUS_OBJ_POISSON_NLL) {
    double* b = reinterpret_cast<double*>(ws);
    nll_bins_kernel<<<(problem->ndata + 127) / 128, 128, 0, st>>>(
      problem->data, problem->idata, problem->ndata, b);
    if ((rc = cuda_fail(cudaGetLastError(), "NLL bins launch")))
      return rc;
    bins = b;
    ws += nll_bytes(problem);
  }
  const size_t kws = need - nll_bytes(problem);
  Objective o = to_objective(problem, bins);
  BfgsParams prm{n, config->max_iter, config->required_converged,
                 config->tolerance, config->flags};
  RunOut ro{out->fval,     out->status, out->iter,   out->gnorm,
            out->x,        out->counters, out->traj_x, out->traj_f,
            out->traj_g,   out->traj_status, out->cycles};
  Control* ctl = reinterpret_cast<Control*>(d_control);
  if (config->mode == ZEUS_MODE_EXACT)
    return launch_exact(o, prm, d_starts, ro, ctl, ws, kws, st);
  return launch_fast(o, *config, prm, d_starts, ro, ctl, ws, kws, st);
}

size_t
zeus_gradient_workspace_size(const zeus_problem* problem)
{
  if (check_problem(problem))
    return 0;
  return nll_bytes(problem);
}

uint32_t
zeus_tile_widths(int32_t kind, int32_t dim)
{
  return tile_widths(kind, dim);
}

int
zeus_gradient_device(const zeus_problem* problem, int32_t path,
                     int32_t gradient, int32_t width, const double* d_x,
                     const double* d_p, double alpha, int64_t n, double* d_f,
                     double* d_g, void* d_workspace, size_t workspace_bytes,
                     void* stream)
{
  int rc = check_problem(problem);
  if (rc)
    return rc;
  if (gradient != ZEUS_GRAD_DUAL && gradient != ZEUS_GRAD_ADJOINT) {
    set_error("unknown gradient %d", gradient);
    return ZEUS_E_INVALID;
  }
  if (n < 0 || n > 0x7fffffffLL || (n > 0 && (!d_x || !d_f || !d_g))) {
    set_error("zeus_gradient_device: bad arguments");
    return ZEUS_E_INVALID;
  }
  if (path == ZEUS_GRADPATH_CTA || path == ZEUS_GRADPATH_CTA_GRAD ||
      path == ZEUS_GRADPATH_QUADRATIC) {
    if (width < 32 || width > 512 || width % 32 != 0) {
      set_error("block gradient paths: width %d is not a multiple of 32 in "
                "[32, 512]",
                width);
      return ZEUS_E_INVALID;
    }
    if (path == ZEUS_GRADPATH_QUADRATIC && (width < problem->dim || !d_p)) {
      set_error("quadratic gradient path: needs width >= dim and directions");
      return ZEUS_E_INVALID;
    }
  }
  if (n == 0)
    return ZEUS_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const double* bins = nullptr;
  if (problem->kind == ZEUS_OBJ_POISSON_NLL) {
    if (!d_workspace || workspace_bytes < nll_bytes(problem)) {
      set_error("zeus_gradient_device: workspace of %zu bytes needed, got %zu",
                nll_bytes(problem), workspace_bytes);
      return ZEUS_E_WORKSPACE;
    }
    double* b = static_cast<double*>(d_workspace);
    nll_bins_kernel<<<(problem->ndata + 127) / 128, 128, 0, st>>>(
      problem->data, problem->idata, problem->ndata, b);
    if ((rc = cuda_fail(cudaGetLastError(), "NLL bins launch")))
      return rc;
    bins = b;
  }
  return launch_gradient(to_objective(problem, bins), path, gradient, width,
                         d_x, d_p, alpha, n, d_f, d_g, st);
}

int
zeus_census_device(const double* d_fval, const int32_t* d_status,
                   const double* d_x, int64_t n, int32_t dim,
                   const double* known_min, zeus_census* d_census,
                   void* stream)
{
  if (n < 0 || !d_census || (n > 0 && (!d_fval || !d_status)) || dim <= 0 ||
      (known_min && dim > kMaxKnownDim)) {
    set_error("zeus_census_device: bad arguments");
    return ZEUS_E_INVALID;
  }
  KnownMin km;
  km.has = known_min ? 1 : 0;
  for (int d = 0; d < kMaxKnownDim; ++d)
    km.x[d] = (known_min && d < dim) ? known_min[d] : 0.0;
  auto kern = dim <= 2    ? census_kernel<2>
              : dim <= 4  ? census_kernel<4>
              : dim <= 8  ? census_kernel<8>
              : dim <= 16 ? census_kernel<16>
                          : census_kernel<32>;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = n > kCensusOneBlock ? kCensusBlocks : 1;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(attr.val.clusterDim.x);
  lc.blockDim = dim3(1024);
  lc.stream = (cudaStream_t)stream;
  lc.attrs = &attr;
  lc.numAttrs = 1;
  return cuda_fail(cudaLaunchKernelEx(&lc, kern, d_fval, d_status, d_x, n, (int)dim, km,
                                      reinterpret_cast<Census*>(d_census)),
                   "census launch");
}

int
zeus_optimize(const zeus_problem* hp, double lower, double upper, int64_t n,
              int32_t max_iter, int32_t pso_iter, int32_t required_converged,
              double tolerance, uint64_t seed, const zeus_bfgs_config* config,
              zeus_result* best, double* best_x, zeus_census* census,
              double* per_run_fval, int32_t* per_run_status, void* stream)
{
  if (!best) {
    set_error("zeus_optimize: best is NULL");
    return ZEUS_E_INVALID;
  }
  *best = zeus_result{-1, -1, 37.0, 0.0, 0, 0}; // util.hpp:36-54 defaults
  if (census)
    *census = zeus_census{0, 0, 0, 0, -1, 0};
  int rc = check_problem(hp);
  if (rc)
    return rc;
  zeus_bfgs_config cfg;
  if (config)
    cfg = *config;
  else {
    cfg = zeus_bfgs_config{};
    cfg.mode = ZEUS_MODE_FAST;
    cfg.gradient = ZEUS_GRAD_ADJOINT;
  }
  cfg.max_iter = max_iter;
  cfg.required_converged = required_converged;
  cfg.tolerance = tolerance;
  if ((rc = check_config(&cfg)))
    return rc;
  if (n < 0) {
    set_error("zeus_optimize: n < 0");
    return ZEUS_E_INVALID;
  }
  if (n == 0) // zeus.cuh:58-60: N == 0 returns the default Result
    return ZEUS_OK;
  const int dim = hp->dim;
  cudaStream_t st = (cudaStream_t)stream;

  // One device allocation holds everything the call needs, each part aligned:
  // allocating, freeing and copying back a part at a time was a third of a
  // small call (200 Gaussian-8 runs: 189 -> 130 us, the rest unchanged).
  zeus_problem dp = *hp;
  if (hp->kind == ZEUS_OBJ_GAUSSIAN) {
    bool symmetric = true;
    for (int i = 0; i < dim && symmetric; ++i)
      for (int j = i + 1; j < dim; ++j)
        if (hp->data[(size_t)i * dim + j] != hp->data[(size_t)j * dim + i]) {
          symmetric = false;
          break;
        }
    dp.flags = symmetric ? ZEUS_PROBLEM_SYMMETRIC : 0;
  }
  const size_t nd = (size_t)n * dim;
  size_t total = 0;
  const auto part = [&](size_t bytes) {
    const size_t at = total;
    total += align_up(bytes);
    return at;
  };
  size_t data_bytes = 0, idata_bytes = 0;
  if (hp->kind == ZEUS_OBJ_GAUSSIAN)
    data_bytes = sizeof(double) * (size_t)dim * dim;
  if (hp->kind == ZEUS_OBJ_POISSON_NLL) {
    data_bytes = sizeof(double) * hp->ndata;
    idata_bytes = sizeof(int32_t) * hp->ndata;
  }
  const bool swarm = pso_iter >= 0;
  const size_t pws = swarm ? zeus_pso_workspace_size(n, dim) : 0;
  const size_t bw = zeus_bfgs_workspace_size(hp, &cfg, n);
  const size_t pack_bytes = sizeof(double) * (kBestHead + (size_t)dim);
  const size_t o_data = part(data_bytes), o_idata = part(idata_bytes);
  const size_t o_starts = part(sizeof(double) * nd), o_fval = part(sizeof(double) * n);
  const size_t o_status = part(sizeof(int32_t) * n), o_iter = part(sizeof(int32_t) * n);
  const size_t o_gnorm = part(sizeof(double) * n), o_x = part(sizeof(double) * nd);
  const size_t o_ctl = part(sizeof(int32_t) * 2), o_cen = part(sizeof(zeus_census));
  const size_t o_pack = part(pack_bytes);
  const size_t o_pbf = part(swarm ? sizeof(double) * n : 0);
  const size_t o_gbest = part(swarm ? sizeof(double) * (dim + 1) : 0);
  const size_t o_pws = part(pws), o_bws = part(bw);
  void* slab = nullptr;
  auto fail = [&](int code) {
    if (slab)
      cudaFreeAsync(slab, st);
    cudaStreamSynchronize(st);
    best->status = (code == ZEUS_E_NOMEM) ? ZEUS_STATUS_NOMEM
                                          : ZEUS_STATUS_KERNEL;
    return code;
  };
  if ((rc = pool_alloc(&slab, total, st)))
    return fail(rc);
  char* base = static_cast<char*>(slab);
  const auto dbl = [&](size_t at) { return reinterpret_cast<double*>(base + at); };
  const auto i32 = [&](size_t at) { return reinterpret_cast<int32_t*>(base + at); };
  if (data_bytes) {
    if ((rc = cuda_fail(cudaMemcpyAsync(base + o_data, hp->data, data_bytes,
                                        cudaMemcpyHostToDevice, st),
                        "H2D problem data")))
      return fail(rc);
    dp.data = dbl(o_data);
  }
  if (idata_bytes) {
    if ((rc = cuda_fail(cudaMemcpyAsync(base + o_idata, hp->idata, idata_bytes,
                                        cudaMemcpyHostToDevice, st),
                        "H2D counts")))
      return fail(rc);
    dp.idata = i32(o_idata);
  }
  if (swarm) {
    if ((rc = zeus_pso_device_prng(&dp, seed, cfg.prng, n, lower, upper, pso_iter, 0.5, 1.2,
                                   1.5, dbl(o_starts), dbl(o_pbf), dbl(o_gbest),
                                   base + o_pws, pws, st)))
      return fail(rc);
  } else if ((rc = zeus_starts(seed, cfg.prng, n, dim, lower, upper, dbl(o_starts), st))) {
    return fail(rc);
  }
  if ((rc = cuda_fail(cudaMemsetAsync(base + o_ctl, 0, sizeof(int32_t) * 2, st),
                      "control reset")))
    return fail(rc);
  zeus_run_outputs ro{};
  ro.fval = dbl(o_fval);
  ro.status = i32(o_status);
  ro.iter = i32(o_iter);
  ro.gnorm = dbl(o_gnorm);
  ro.x = dbl(o_x);
  if ((rc = zeus_bfgs_device(&dp, &cfg, dbl(o_starts), n, &ro, i32(o_ctl), base + o_bws, bw,
                             st)))
    return fail(rc);
  std::vector<double> km;
  if (hp->kind == ZEUS_OBJ_ROSENBROCK)
    km.assign(dim, 1.0);
  auto* cen = reinterpret_cast<zeus_census*>(base + o_cen);
  if ((rc = zeus_census_device(ro.fval, ro.status, ro.x, n, dim,
                               km.empty() ? nullptr : km.data(), cen, st)))
    return fail(rc);
  best_run_kernel<<<1, 128, 0, st>>>(reinterpret_cast<const Census*>(cen), ro.fval, ro.gnorm,
                                     ro.status, ro.iter, ro.x, dim,
                                     swarm ? dbl(o_gbest) : nullptr, dbl(o_pack));
  std::vector<double> pack(kBestHead + (size_t)dim);
  if ((rc = cuda_fail(cudaGetLastError(), "best run launch")) ||
      (rc = cuda_fail(cudaMemcpyAsync(pack.data(), dbl(o_pack), pack_bytes,
                                      cudaMemcpyDeviceToHost, st),
                      "D2H census and best run")) ||
      (rc = cuda_fail(cudaStreamSynchronize(st), "BFGS run")))
    return fail(rc);
  if (std::isnan(pack[3]))
    return fail(swarm_gave_up());
  zeus_census hc;
  std::memcpy(&hc, pack.data(), sizeof hc);
  if (census)
    *census = hc;
  if (hc.best_idx >= 0) {
    if (per_run_fval &&
        (rc = cuda_fail(cudaMemcpyAsync(per_run_fval, ro.fval, sizeof(double) * n,
                                        cudaMemcpyDeviceToHost, st),
                        "D2H fvals")))
      return fail(rc);
    if (per_run_status &&
        (rc = cuda_fail(cudaMemcpyAsync(per_run_status, ro.status, sizeof(int32_t) * n,
                                        cudaMemcpyDeviceToHost, st),
                        "D2H statuses")))
      return fail(rc);
    best->idx = hc.best_idx;
    best->fval = pack[4];
    best->gradient_norm = pack[5];
    int32_t si[2];
    std::memcpy(si, &pack[6], sizeof si);
    best->status = si[0];
    best->iter = si[1];
    if (best_x)
      std::memcpy(best_x, pack.data() + kBestHead, sizeof(double) * dim);
  }
  cudaFreeAsync(slab, st);
  return cuda_fail(cudaStreamSynchronize(st), "free");
}

int
zeus_autotune_lookup(int32_t kind, int32_t dim, int32_t gradient,
                     int32_t* layout, int32_t* tile)
{
  return tune_lookup(2, kind, dim, gradient, layout, tile);
}

int
zeus_autotune_record(int32_t kind, int32_t dim, int32_t gradient,
                     int32_t layout, int32_t tile)
{
  for (int form = 0; form < 3; ++form)
    if (int rc = tune_record(form, kind, dim, gradient, layout, tile))
      return rc;
  return ZEUS_OK;
}

// iterations of the autotuner's single-run latency measurement
static constexpr int kTuneLatencyIters = 200;

int
zeus_autotune(const zeus_problem* problem, const zeus_bfgs_config* config,
              int64_t n_sample, uint64_t seed, double lower, double upper,
              int32_t* best_layout, int32_t* best_tile, float* best_ms,
              void* stream)
{
  int rc = check_problem(problem);
  if (rc)
    return rc;
  if ((rc = check_config(config)))
    return rc;
  if (config->mode != ZEUS_MODE_FAST || n_sample <= 0) {
    set_error("zeus_autotune: fast mode and n_sample > 0 required");
    return ZEUS_E_INVALID;
  }
  const int kind = problem->kind, dim = problem->dim;
  // layout, tile, block: the thread layout in either form it may have
  struct Candidate {
    int layout, tile, block;
  };
  std::vector<Candidate> cand;
  if (thread_layout_supported(kind, dim)) {
    cand.push_back({ZEUS_LAYOUT_THREAD, 0, config->block > 0 ? config->block : 128});
    if (thread_layout_warps(kind, dim, config->gradient, config->max_iter, 1))
      cand.push_back({ZEUS_LAYOUT_THREAD, 0, kBlockWarps});
  }
  const unsigned w = tile_widths(kind, dim);
  for (int k = 1; k <= 5; ++k)
    if ((w >> k) & 1u)
      cand.push_back({ZEUS_LAYOUT_TILE, 1 << k, config->block});
  if (cta_layout_supported(kind, dim))
    cand.push_back({ZEUS_LAYOUT_CTA, 0, config->block});
  if (rows_layout_supported(kind, dim))
    cand.push_back({ZEUS_LAYOUT_ROWS, 0, config->block});
  if (cand.empty()) {
    set_error("zeus_autotune: no layout built for kind %d dim %d", kind, dim);
    return ZEUS_E_UNSUPPORTED;
  }
  cudaStream_t st = (cudaStream_t)stream;
  std::vector<void*> allocs;
  auto cleanup = [&]() {
    for (void* p : allocs)
      cudaFreeAsync(p, st);
    cudaStreamSynchronize(st);
  };
  auto alloc = [&](size_t bytes, void** out) -> int {
    const int r = pool_alloc(out, bytes, st);
    if (r == ZEUS_OK)
      allocs.push_back(*out);
    return r;
  };
  void *starts, *fval, *status, *iters, *gnorm, *xo, *ctl, *ws;
  const size_t nd = (size_t)n_sample * dim;
  zeus_bfgs_config c0 = *config;
  c0.layout = ZEUS_LAYOUT_TILE; // any; the workspace does not depend on it
  const size_t wsz = zeus_bfgs_workspace_size(problem, &c0, n_sample);
  // (CTA and row layouts: the same run queue)
  if ((rc = alloc(sizeof(double) * nd, &starts)) ||
      (rc = alloc(sizeof(double) * n_sample, &fval)) ||
      (rc = alloc(sizeof(int32_t) * n_sample, &status)) ||
      (rc = alloc(sizeof(int32_t) * n_sample, &iters)) ||
      (rc = alloc(sizeof(double) * n_sample, &gnorm)) ||
      (rc = alloc(sizeof(double) * nd, &xo)) ||
      (rc = alloc(sizeof(int32_t) * 2, &ctl)) || (rc = alloc(wsz, &ws))) {
    cleanup();
    return rc;
  }
  if ((rc = zeus_starts_uniform(seed, n_sample, dim, lower, upper,
                                static_cast<double*>(starts), st))) {
    cleanup();
    return rc;
  }
  zeus_run_outputs ro{};
  ro.fval = static_cast<double*>(fval);
  ro.status = static_cast<int32_t*>(status);
  ro.iter = static_cast<int32_t*>(iters);
  ro.gnorm = static_cast<double*>(gnorm);
  ro.x = static_cast<double*>(xo);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  // the records' bests: with a thread a run in the thread layout (launches of
  // many runs, and batches) and with a warp a run
  float best[2] = {3.4e38f, 3.4e38f};
  int bl[2] = {-1, -1}, bt[2] = {0, 0};
  for (const Candidate& cd : cand) {
    zeus_bfgs_config c = *config;
    c.layout = cd.layout;
    c.tile = cd.tile;
    c.block = cd.block;
    float ms_min = 3.4e38f;
    for (int rep = 0; rep < 2 && rc == ZEUS_OK; ++rep) { // warm-up + timed
      cudaMemsetAsync(ctl, 0, sizeof(int32_t) * 2, st);
      cudaEventRecord(e0, st);
      rc = zeus_bfgs_device(problem, &c, static_cast<double*>(starts), n_sample,
                            &ro, static_cast<int32_t*>(ctl), ws, wsz, st);
      cudaEventRecord(e1, st);
      if (rc == ZEUS_OK)
        rc = cuda_fail(cudaEventSynchronize(e1), "autotune run");
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (rep > 0)
        ms_min = ms;
    }
    if (rc != ZEUS_OK)
      break;
    // the latency of one iteration of one run alone: a run that iterates to
    // max_iter (one that neither converges nor reaches a fixed point) takes
    // max_iter of them, and a batch lasts as long as its slowest run
    float lat_ms = 0.f;
    if (config->max_iter > 0) {
      zeus_bfgs_config cl = c;
      cl.max_iter = kTuneLatencyIters;
      cl.tolerance = 0.0;                      // never converges
      cl.flags |= ZEUS_FLAG_NO_FIXED_POINT;    // never stops early
      cl.required_converged = 0x7fffffff;
      for (int rep = 0; rep < 2 && rc == ZEUS_OK; ++rep) {
        cudaMemsetAsync(ctl, 0, sizeof(int32_t) * 2, st);
        cudaEventRecord(e0, st);
        rc = zeus_bfgs_device(problem, &cl, static_cast<double*>(starts), 1, &ro,
                              static_cast<int32_t*>(ctl), ws, wsz, st);
        cudaEventRecord(e1, st);
        if (rc == ZEUS_OK)
          rc = cuda_fail(cudaEventSynchronize(e1), "autotune latency run");
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (rep > 0)
          lat_ms = ms / kTuneLatencyIters;
      }
      if (rc != ZEUS_OK)
        break;
    }
    // the class alone would take about the longer of its bulk (the sample)
    // and one run iterating to max_iter
    const float est = std::max(ms_min, lat_ms * (float)config->max_iter);
    const bool thread = cd.layout == ZEUS_LAYOUT_THREAD, warps = cd.block == kBlockWarps;
    for (int form = 0; form < 2; ++form)
      if ((!thread || warps == (form == 1)) && est < best[form]) {
        best[form] = est;
        bl[form] = cd.layout;
        bt[form] = cd.tile;
      }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cleanup();
  if (rc != ZEUS_OK)
    return rc;
  for (int form = 0; form < 2; ++form)
    if (bl[form] > 0)
      tune_record(form, kind, dim, config->gradient, bl[form], bt[form]);
  // reported: the choice for a launch like the sample
  const int rep = config->block <= 0 && thread_layout_warps(kind, dim, config->gradient,
                                                            config->max_iter, n_sample)
                    ? 1
                    : 0;
  tune_record(2, kind, dim, config->gradient, bl[rep], bt[rep]);
  if (best_layout)
    *best_layout = bl[rep];
  if (best_tile)
    *best_tile = bt[rep];
  if (best_ms)
    *best_ms = best[rep];
  return ZEUS_OK;
}

void
zeus_probe_fp64_shape(int32_t* grid, int32_t* block)
{
  if (grid)
    *grid = sm_count() * 8;
  if (block)
    *block = 256;
}

int
zeus_probe_fp64(int64_t iters, double* d_sink, void* stream)
{
  if (iters < 0 || !d_sink) {
    set_error("zeus_probe_fp64: bad arguments");
    return ZEUS_E_INVALID;
  }
  fp64_probe_kernel<<<sm_count() * 8, 256, 0, (cudaStream_t)stream>>>(iters,
                                                                       d_sink);
  return cuda_fail(cudaGetLastError(), "FP64 probe launch");
}

} // extern "C"
