// A whole PSO -- initial swarm and every iteration -- in one launch.
//
// The per-iteration kernels (zb_pso.cuh) spend their time on launches, on
// positions, velocities and bests that go out to memory and back, and on a
// last block that reduces while the others wait: 14 us an iteration for 16384
// particles at D = 10 and for 1024 at D = 150, where the arithmetic is 1-2 us.
// One launch: 16384 Rastrigin-10 particles, 20 iterations, 291 -> 94 us; 1024
// Gaussian-150 particles, 10 iterations, 159 -> 71 us (of a 77 us build's
// iteration 5500 cycles were the tensor-core product, 2960 of them its issue,
// and 3000 the meeting); 20000 Rosenbrock-32 particles, 10 iterations, 487 -> 104
// us (B200).
// Here a block keeps its particles' state in shared memory for the whole
// call.  Its threads take (particle, coordinate) elements, so the random
// numbers and moves of one particle are spread over D threads; where the
// objective is a sum of terms over coordinates the terms are formed the same
// way and one thread per particle adds them in the reference's order.  The
// arithmetic and its order are the per-iteration kernels': the same bits.
//
// Blocks meet once an iteration: each publishes its best (key, index and,
// where it beats gbest, position) in a slot tagged with the iteration, two
// slots in turn, reads the others' until all have arrived and finds the swarm's
// best by itself.
// The launch is cooperative (every block resident), so the wait is as long as
// the slowest block's evaluation.  It has a limit all the same: a block that has
// read the slots SwarmArgs::wait times gives up, fills its rows of pbx and pbf
// with NaN and publishes nothing more.  So block 0, which waits for all in every
// iteration, gives up as well, and gbest's value is NaN (which no swarm's best
// is) whenever a row is not the swarm's.
#pragma once

#include "zb_objectives.cuh"
#include "zb_pso.cuh"
#include "zb_pso_dmma.cuh"

namespace zb {

  // Reads of the slots before a block gives up: about two seconds.
  inline constexpr int kSwarmWait = 1 << 22;
  inline constexpr int kSwarmMaxBlocks = 160; // slots read by one block
  inline constexpr int kSwarmAhead = 4; // elements a thread moves ahead of gbest

  struct SwarmArgs {
    int64_t n;
    int per_block; // particles of a block
    int iters;
    double lower, upper, w, c1, c2;
    uint64_t seed;
    const uint32_t* sobol;
    double* pbx;
    double* pbf;
    double* gbest;
    // slots [2][gridDim.x][4], zeroed before the launch: the key's high and
    // low words and the index, each below the iteration's tag
    unsigned long long* slots;
    double* slot_x; // [2][gridDim.x][D]
    int wait;       // reads of the slots before a block gives up
  };

  // f as a sum of per-coordinate terms added in index order: term(x, i) for
  // i < count(), fold(t) over a particle's terms.
  template <class F>
  struct SwarmTerms {
    static constexpr bool value = false;
  };
  template <std::size_t D>
  struct SwarmTerms<zeus::Rosenbrock<D>> {
    static constexpr bool value = true;
    static constexpr int count = (int)D - 1;
    __device__ static __forceinline__ double
    term(const double* x, int i)
    {
      const double t1 = 1.0 - x[i];
      const double t2 = x[i + 1] - x[i] * x[i];
      return t1 * t1 + 100.0 * t2 * t2;
    }
    __device__ static __forceinline__ double
    fold(const double* t, const double*)
    {
      double sum = 0.0;
#pragma unroll 8
      for (int i = 0; i < count; ++i)
        sum += t[i];
      return sum;
    }
  };
  template <std::size_t D>
  struct SwarmTerms<zeus::Rastrigin<D>> {
    static constexpr bool value = true;
    static constexpr int count = (int)D;
    __device__ static __forceinline__ double
    term(const double* x, int i)
    {
      return x[i] * x[i] - 10.0 * ::cos(zeus::kTwoPi * x[i]);
    }
    __device__ static __forceinline__ double
    fold(const double* t, const double*)
    {
      double sum = 10.0 * D;
#pragma unroll 8
      for (int i = 0; i < count; ++i)
        sum += t[i];
      return sum;
    }
  };
  template <std::size_t D>
  struct SwarmTerms<zeus::Ackley<D>> {
    static constexpr bool value = true;
    static constexpr int count = (int)D;
    __device__ static __forceinline__ double
    term(const double* x, int i)
    {
      return ::cos(zeus::kTwoPi * x[i]);
    }
    __device__ static __forceinline__ double
    fold(const double* t, const double* x)
    {
      double sum_sq = 0.0, sum_cos = 0.0;
#pragma unroll 8
      for (int i = 0; i < count; ++i) {
        sum_sq += x[i] * x[i];
        sum_cos += t[i];
      }
      const double term1 = -20.0 * ::exp(-0.2 * ::sqrt(sum_sq / D));
      const double term2 = -::exp(sum_cos / D);
      return term1 + term2 + 20.0 + ::exp(1.0);
    }
  };

  // How a block evaluates f: terms shared out over its threads, one particle
  // to a thread, a warp (D >= kPsoCoopMinDim), or eight to the FP64 tensor
  // cores (the Gaussian there).
  template <class F, int D>
  constexpr bool
  swarm_dmma()
  {
    return D >= kPsoCoopMinDim && D <= kPsoDmmaMaxDim && F::kind == 3;
  }
  template <class F, int D>
  constexpr bool
  swarm_terms()
  {
    return D < kPsoCoopMinDim && SwarmTerms<F>::value;
  }
  // (a warp for each 8-column tile of the tensor-core product, whose sums stay
  // split over eight warps' worth)
  template <class F, int D>
  constexpr int
  swarm_threads()
  {
    return !swarm_dmma<F, D>() ? 512 : D <= 192 ? 768 : 1024;
  }

  // Row stride of a block's positions (and of C): odd below kPsoCoopMinDim,
  // where a thread walks its own particle's row; for the tensor-core
  // fragments, four consecutive entries of eight rows, 4 or 12 modulo the 16
  // banks of doubles, so that a half warp's four rows do not share any (at
  // D = 150 a stride of 150 took twice the wavefronts: 7300 cycles an
  // evaluation).
  template <class F, int D>
  constexpr int
  swarm_stride()
  {
    if (D < kPsoCoopMinDim)
      return D | 1;
    int s = D;
    if (swarm_dmma<F, D>())
      while (s % 16 != 4 && s % 16 != 12)
        ++s;
    return s;
  }

  // Doubles of shared memory of a block of `per` particles: positions,
  // velocities, bests, terms, values and best values, gbest's position, warp
  // scratch, flags; and the Gaussian's C.
  template <class F, int D>
  constexpr size_t
  swarm_doubles(int64_t per)
  {
    const size_t sd = swarm_stride<F, D>();
    return (size_t)per * (sd + 2 * D + (swarm_terms<F, D>() ? sd : 0) + 2) + D +
           swarm_threads<F, D>() + (size_t)(per + 1) / 2 + 2 +
           (F::kind == 3 ? D * (swarm_dmma<F, D>() ? sd : (size_t)D) : 0);
  }

  // What a block's static arrays leave of an SM's shared memory.
  inline constexpr size_t kSwarmSmem = 227 * 1024 - 1280;

  // Whether any swarm of the objective fits a block: a particle, or the eight
  // of the tensor-core product (D = 150; the kernel's tiles and hand-over
  // array are laid out for the dimensions that fit, and no others are built).
  template <class F, int D>
  constexpr bool
  swarm_built()
  {
    return sizeof(double) * swarm_doubles<F, D>(swarm_dmma<F, D>() ? kPsoDmmaParticles : 1) <=
           kSwarmSmem;
  }

  // f of eight particles (rows of Xs) with C in shared memory, the bits of
  // gauss_f8_dmma on eight warps: its warp v sums the tiles v, v + 8, ... of
  // Y = X C^T against X in turn.  Here each tile is a warp's; the warps past
  // the eighth hand theirs over through `ex` (64 doubles a tile past 8).  Thread
  // t < 8 returns particle t's value; ends with `part` read.
  template <int D, int SD, int NT>
  __device__ __forceinline__ double
  swarm_f8_dmma(const double* Cs, const double* Xs, double* ex, double* part)
  {
    constexpr int JT = (D + 7) / 8, KT = (D + 3) / 4;
    static_assert(JT <= NT / 32, "a warp a tile");
    static_assert((JT - 8) * 64 <= NT, "ex holds the tiles past the eighth");
    const int lane = threadIdx.x & 31, jt = threadIdx.x >> 5;
    const int r = lane >> 2, c4 = lane & 3;
    const double* xr = Xs + r * SD;
    double d0 = 0.0, d1 = 0.0;
    if (jt < JT) {
      double e0 = 0.0, e1 = 0.0, o0 = 0.0, o1 = 0.0;
      const int jb = jt * 8 + r; // the B column (a row of C) this lane loads
      const bool bv = jb < D;
      const double* cb = Cs + (bv ? jb : 0) * SD;
#pragma unroll 10
      for (int kk = 0; kk < KT; kk += 2) {
        const int k = kk * 4 + c4, k2 = k + 4;
        const double a = k < D ? xr[k] : 0.0, b = bv && k < D ? cb[k] : 0.0;
        const double a2 = k2 < D ? xr[k2] : 0.0, b2 = bv && k2 < D ? cb[k2] : 0.0;
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
            "{%0, %1}, {%2}, {%3}, {%0, %1};"
            : "+d"(e0), "+d"(e1)
            : "d"(a), "d"(b));
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
            "{%0, %1}, {%2}, {%3}, {%0, %1};"
            : "+d"(o0), "+d"(o1)
            : "d"(a2), "d"(b2));
      }
      d0 = e0 + o0;
      d1 = e1 + o1;
      if (jt >= 8) {
        ex[(jt - 8) * 64 + lane] = d0;
        ex[(jt - 8) * 64 + 32 + lane] = d1;
      }
    }
    __syncthreads();
    if (jt < 8) {
      double acc = 0.0;
      for (int q = jt; q < JT; q += 8) {
        if (q >= 8) {
          d0 = ex[(q - 8) * 64 + lane];
          d1 = ex[(q - 8) * 64 + 32 + lane];
        }
        const int j0 = q * 8 + c4 * 2;
        if (j0 < D)
          acc = fma(xr[j0], d0, acc);
        if (j0 + 1 < D)
          acc = fma(xr[j0 + 1], d1, acc);
      }
      // the four lanes of a row hold its partial sums
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      if (c4 == 0)
        part[jt * 8 + r] = acc;
    }
    __syncthreads();
    double f = 0.0;
    if (threadIdx.x < kPsoDmmaParticles)
      for (int w = 0; w < 8; ++w)
        f += part[w * 8 + threadIdx.x];
    return 0.5 * f;
  }

  __device__ __forceinline__ unsigned long long
  load_relaxed(const unsigned long long* p)
  {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
  }
  __device__ __forceinline__ void
  store_relaxed(unsigned long long* p, unsigned long long v)
  {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
  }
  // the value an order_key came from
  __device__ __forceinline__ double
  order_value(unsigned long long key)
  {
    const unsigned long long b =
      (key & 0x8000000000000000ull) ? (key & 0x7fffffffffffffffull) : ~key;
    return __longlong_as_double((long long)b);
  }

  // The lowest (key, index) of a warp, in every lane.
  __device__ __forceinline__ void
  warp_argmin(unsigned long long& key, int& idx)
  {
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned mh = __reduce_min_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? lo : 0xffffffffu);
    idx = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? idx : 0x7fffffff);
    key = ((unsigned long long)mh << 32) | ml;
  }

  template <class F, int D>
  __global__ void __launch_bounds__(swarm_threads<F, D>(), 1)
    pso_swarm_kernel(F f, const __grid_constant__ SwarmArgs a)
  {
    constexpr int NT = swarm_threads<F, D>(), SD = swarm_stride<F, D>();
    extern __shared__ __align__(16) double sm[];
    const int per = a.per_block;
    constexpr bool kMatrix = F::kind == 3;
    double* Cs = sm; // C where kMatrix
    constexpr int CS = swarm_dmma<F, D>() ? SD : D; // row stride of C
    double* X = Cs + (kMatrix ? D * CS : 0);
    double* V = X + (size_t)per * SD;
    double* P = V + (size_t)per * D;
    double* T = P + (size_t)per * D;
    double* FV = T + (swarm_terms<F, D>() ? (size_t)per * SD : 0);
    double* PF = FV + per;
    double* gb = PF + per;
    double* scr = gb + D;
    int* better = reinterpret_cast<int*>(scr + NT);
    __shared__ double part[(kPsoBlock / 32) * 8];
    __shared__ unsigned long long sh_key[NT / 32];
    __shared__ int sh_idx[NT / 32];
    __shared__ int sh_win, sh_late;
    __shared__ double sh_f;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nb = (int)gridDim.x;
    const int64_t i0 = (int64_t)blockIdx.x * per;
    const int cnt = (int)(a.n - i0 < per ? a.n - i0 : per);
    const int elems = cnt * D;
    constexpr int kMeetWarp = NT / 32 - 1; // reads the other blocks' slots
    const int kwarps = (cnt + 31) / 32; // warps that hold a particle's key
    double gbf = __longlong_as_double(0x7ff0000000000000ll);

    if constexpr (kMatrix)
#pragma unroll 10
      for (int e = t; e < D * D; e += NT)
        Cs[e / D * CS + e % D] = f.C[e];
    if (t < D)
      gb[t] = 0.0;
    for (int d = t + NT; d < D; d += NT)
      gb[d] = 0.0;
    for (int p = t; p < per; p += NT)
      better[p] = 0;
    if (t == 0)
      sh_late = 0;
    if constexpr (swarm_dmma<F, D>())
      for (int e = cnt * SD + t; e < per * SD; e += NT) // rows past the swarm
        X[e] = 0.0;
    {
      const double vr = (a.upper - a.lower) * 0.1;
      for (int e = t; e < elems; e += NT) {
        const int p = e / D, d = e % D;
        const uint64_t i = (uint64_t)(i0 + p);
        const double ux = position01(a.sobol, a.seed, kTagPsoX, i, (uint32_t)d);
        const double uv = uniform01(a.seed, kTagPsoV, i, (uint32_t)d);
        const double rx = a.lower + (a.upper - a.lower) * ux;
        const double rv = -vr + (vr - -vr) * uv;
        X[p * SD + d] = rx;
        V[e] = rv;
        P[e] = rx;
      }
    }

    for (int it = 0;; ++it) {
      __syncthreads(); // positions are in place
      // ---- f of every particle into FV
      if constexpr (swarm_dmma<F, D>()) {
        const double fv = swarm_f8_dmma<D, SD, NT>(Cs, X, scr, part);
        if (t < cnt) // (eight particles to a block)
          FV[t] = fv;
      } else if constexpr (D >= kPsoCoopMinDim) {
        const TileGroup<32> grp(cg::tiled_partition<32>(cg::this_thread_block()),
                                scr + (t & ~31));
        for (int p = warp; p < cnt; p += NT / 32) {
          const double fv = coop_value<F, D>(f, grp, X + p * SD);
          if (lane == 0)
            FV[p] = fv;
        }
        __syncthreads();
      } else if constexpr (swarm_terms<F, D>()) {
        using ST = SwarmTerms<F>;
        for (int e = t; e < cnt * ST::count; e += NT) {
          const int p = e / ST::count, i = e % ST::count;
          T[p * SD + i] = ST::term(X + p * SD, i);
        }
        __syncthreads();
        if (t < cnt)
          FV[t] = ST::fold(T + t * SD, X + t * SD);
      } else if constexpr (F::kind == 3) {
        // the quadratic form's D^2 terms in order: products and loads run
        // ahead of the chain of additions
        if (t < cnt) {
          const double* x = X + t * SD;
          double q = 0.0;
          for (int i = 0; i < D; ++i) {
            const double xi = x[i];
#pragma unroll(D < 16 ? D : 16)
            for (int j = 0; j < D; ++j)
              q += xi * Cs[i * D + j] * x[j];
          }
          FV[t] = 0.5 * q;
        }
      } else {
        if (t < cnt) {
          std::array<double, D> xa;
#pragma unroll 1
          for (int d = 0; d < D; ++d)
            xa[d] = X[t * SD + d];
          FV[t] = f(xa);
        }
      }
      // ---- bests
      unsigned long long key = ~0ull;
      int kidx = 0x7fffffff;
      if (t < cnt) { // (thread t wrote FV[t], or a barrier has passed)
        const double fv = FV[t];
        const bool b = it == 0 || fv < PF[t];
        better[t] = b;
        if (b)
          PF[t] = fv;
        key = order_key(fv);
        kidx = (int)(i0 + t);
      }
      if (warp < kwarps) {
        warp_argmin(key, kidx);
        if (lane == 0) {
          sh_key[warp] = key;
          sh_idx[warp] = kidx;
        }
      }
      __syncthreads(); // also publishes `better`
      // (every warp finds the block's best for itself)
      key = lane < kwarps ? sh_key[lane] : ~0ull;
      kidx = lane < kwarps ? sh_idx[lane] : 0x7fffffff;
      warp_argmin(key, kidx);
      const int par = it & 1;
      if (nb > 1) {
        // ---- publish the block's best where it beats gbest (another cannot
        // become it; its position then need not be written)
        const bool beats = key != ~0ull && order_value(key) < gbf;
        if (beats) {
          double* sx = a.slot_x + ((size_t)par * nb + blockIdx.x) * D;
          for (int d = t; d < D; d += NT)
            sx[d] = X[(int)(kidx - i0) * SD + d];
        } else {
          key = ~0ull;
          kidx = 0x7fffffff;
        }
        if constexpr (D > 32) {
          if (beats)
            __syncthreads(); // written by several warps
        } else
          __syncwarp();
        if (t == 0) {
          // three words, each with the iteration's tag: a reader that sees
          // the tag has the word; the position is ordered before them
          unsigned long long* slot = a.slots + 4 * ((size_t)par * nb + blockIdx.x);
          const unsigned long long tag = (unsigned long long)(it + 1) << 32;
          if (beats)
            __threadfence();
          store_relaxed(slot + 0, tag | (key >> 32));
          store_relaxed(slot + 1, tag | (key & 0xffffffffull));
          store_relaxed(slot + 2, tag | (unsigned)kidx);
        }
      }
      if (it > 0)
        for (int e = t; e < elems; e += NT) {
          const int p = e / D;
          if (better[p])
            P[e] = X[p * SD + e % D];
        }
      if (nb > 1 && it == a.iters && blockIdx.x != 0)
        break; // block 0 reports gbest
      // ---- the next move up to gbest's part, while the blocks meet: of
      // w v + c1 r1 (pb - x) + c2 r2 (gb - x) the first sum and c2 r2
      double base[kSwarmAhead], c2r[kSwarmAhead];
      const auto ahead = [&](int e, double& bs, double& cr) {
        const int p = e / D, d = e % D;
        uint32_t o[4];
        const uint64_t i = (uint64_t)(i0 + p);
        // r1 and r2 (indices 2d and 2d + 1) share one Philox block
        philox4x32_10((uint32_t)i, (uint32_t)d, kTagPsoIter + (uint32_t)(it + 1),
                      (uint32_t)(i >> 32), (uint32_t)a.seed, (uint32_t)(a.seed >> 32), o);
        const double r1 = uniform01_word(o[0], o[1]), r2 = uniform01_word(o[2], o[3]);
        bs = a.w * V[e] + a.c1 * r1 * (P[e] - X[p * SD + d]);
        cr = a.c2 * r2;
      };
      if (it < a.iters)
#pragma unroll
        for (int k = 0; k < kSwarmAhead; ++k)
          if (t + k * NT < elems)
            ahead(t + k * NT, base[k], c2r[k]);
      // ---- the swarm's best
      if (warp == kMeetWarp) {
        if (nb > 1) {
          key = ~0ull;
          kidx = 0x7fffffff;
          // every slot's words at once, until all are this iteration's
          constexpr int SL = kSwarmMaxBlocks / 32;
          unsigned long long w[SL][3] = {};
          bool late = true;
          for (int reads = 0; reads < a.wait; ++reads) {
            bool all = true;
#pragma unroll
            for (int k = 0; k < SL; ++k)
              if (lane + 32 * k < nb) {
                const unsigned long long* sl =
                  a.slots + 4 * ((size_t)par * nb + lane + 32 * k);
#pragma unroll
                for (int q = 0; q < 3; ++q)
                  w[k][q] = load_relaxed(sl + q);
              }
#pragma unroll
            for (int k = 0; k < SL; ++k)
              if (lane + 32 * k < nb)
#pragma unroll
                for (int q = 0; q < 3; ++q)
                  all &= (unsigned)(w[k][q] >> 32) == (unsigned)(it + 1);
            if (all) {
              late = false;
              break;
            }
          }
          __threadfence(); // before any position is read
#pragma unroll
          for (int k = 0; k < SL; ++k)
            if (lane + 32 * k < nb) {
              const unsigned long long kk = (w[k][0] << 32) | (unsigned)w[k][1];
              const int ki = (int)(unsigned)w[k][2];
              if (kk < key || (kk == key && ki < kidx)) {
                key = kk;
                kidx = ki;
              }
            }
          late = __any_sync(0xffffffffu, late);
          if (late && lane == 0)
            sh_late = 1;
          warp_argmin(key, kidx);
        }
        if (lane == 0) {
          sh_win = key != ~0ull ? kidx : -1;
          sh_f = order_value(key);
        }
      }
      __syncthreads();
      if (sh_late)
        break;
      if (sh_win >= 0 && sh_f < gbf) {
        gbf = sh_f;
        const int win = sh_win;
        if (nb > 1) {
          const double* sx = a.slot_x + ((size_t)par * nb + win / per) * D;
          for (int d = t; d < D; d += NT)
            gb[d] = *reinterpret_cast<const volatile double*>(sx + d);
        } else {
          for (int d = t; d < D; d += NT)
            gb[d] = X[win * SD + d];
        }
      }
      if (it == a.iters)
        break;
      __syncthreads(); // gb is in place
      // ---- move
      const auto move = [&](int e, double bs, double cr) {
        const int p = e / D, d = e % D;
        const double xi = X[p * SD + d];
        const double nv = bs + cr * (gb[d] - xi);
        V[e] = nv;
        X[p * SD + d] = xi + nv;
      };
#pragma unroll
      for (int k = 0; k < kSwarmAhead; ++k)
        if (t + k * NT < elems)
          move(t + k * NT, base[k], c2r[k]);
      for (int e = t + kSwarmAhead * NT; e < elems; e += NT) {
        double bs, cr;
        ahead(e, bs, cr);
        move(e, bs, cr);
      }
    }
    __syncthreads();
    const bool late = sh_late != 0;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    for (int e = t; e < elems; e += NT)
      a.pbx[i0 * D + e] = late ? nan : P[e];
    for (int p = t; p < cnt; p += NT)
      a.pbf[i0 + p] = late ? nan : PF[p];
    if (blockIdx.x == 0) {
      if (t == 0)
        a.gbest[0] = late ? nan : gbf;
      for (int d = t; d < D; d += NT)
        a.gbest[1 + d] = gb[d];
    }
  }

} // namespace zb
