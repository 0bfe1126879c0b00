// Fast BFGS for a symmetric quadratic form, one run per block, with the
// matrix C in shared memory and the inverse Hessian H in registers.
//
// The algorithm is the CTA layout's for symmetric C (cta_run): one pass over C
// an iteration forms C x and C p, the line search is decided on the exact
// quadratic model, one sweep over H applies the previous iteration's deferred
// update and forms H y and H g, and an end of a run is confirmed on f and g
// formed exactly at x.  Every sum keeps that kernel's split and order for its
// 512-thread block, so results are the same bits: Q segments of rows for the
// pass (two chains each) and the sweep, Q1 for the exact evaluation, the
// reductions' xor trees.
//
// What bounds it: the CTA layout keeps H in shared memory (D = 150: 180 KB),
// which leaves C to be read from L2 by every block in every iteration (7000 of
// an iteration's 16 000 cycles at D = 150) and moves H through shared memory
// twice (5900).  A thread here owns the same H elements throughout -- a
// column pair's rows q, q + Q, ... -- so H lives in its registers but for
// KS rows, and C takes H's place in shared memory, copied once per block for
// all the runs it takes.  An iteration at D = 150 is then 7500 cycles: 2400 the
// pass over C (2100 shared-memory wavefronts), 1600 the sweep (six FP64
// operations an element), 3500 the partial sums, two reductions and the O(D)
// work, a chain of latencies.  1024 runs 1106 -> 673 us on a B200, 64 runs
// 723 -> 439, 8192 runs 5280 -> 3167.  A run on a cluster of two blocks, each
// with half the columns, was shorter alone (64 runs: 377 us) but two blocks'
// barriers and exchanges outweighed the halved passes (1024 runs 807 us, 8192
// runs 4960); clusters of four more so.
#pragma once

#include "zb_bfgs_coop.cuh"

namespace zb {

  // The CTA layout's block, whose split of every sum this kernel keeps.
  inline constexpr int kQuadSplitBlock = 512;

  template <int D>
  struct QuadShape {
    static constexpr int NP = D / 2;                          // column pairs
    static constexpr int Q = cta_sweep_q(D, kQuadSplitBlock); // segments of rows
    static constexpr int Q1 = kQuadSplitBlock / D;            // ... exact evaluation
    static constexpr int T = NP * Q;                          // working threads
    static constexpr int RW = (D + 31) / 32;                  // warps of owners
    static constexpr int NT = ((T > 32 * RW ? T : 32 * RW) + 31) / 32 * 32;
    static constexpr int RQ = (D + Q - 1) / Q;                // rows a thread
    // rows a thread keeps in shared memory: what the register limit leaves no
    // room for beside the sweep's operands
    static constexpr int KS = 4;
    // C | {x, p} | {s, w} | {y, g_x} | partial sums | rows of H | reductions |
    // run index, stop flag
    static constexpr size_t doubles = (size_t)D * D + 6 * (size_t)D + 2 * (size_t)Q * D +
                                      2 * (size_t)KS * T + 2 * 64 + 2;
    static constexpr bool fits = D % 2 == 0 && Q >= 1 && Q1 >= 2 && Q1 * D <= T && RW <= 8 &&
                                 NT <= 512 && RQ > KS && 2 * (RQ - KS) <= 48 &&
                                 doubles * sizeof(double) <= 227 * 1024;
  };

  // Sums of K values over the block's first RW warps (the other warps hold
  // none), the bits of CtaGroup::sum: xor trees within the warps, then over
  // the warps.  One barrier; `buf` (8 K doubles) is free again after the
  // caller's next barrier.
  template <int K, int RW>
  __device__ __forceinline__ void
  quad_sum(double (&v)[K], double* buf)
  {
    using RS = ReduceScatter<K>;
    const auto shx = [](double x, int m) { return __shfl_xor_sync(0xffffffffu, x, m); };
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int idx = RS::template index<32>(lane);
    if (warp < RW) {
      const double mine = RS::template run<32>(v, lane, shx);
      if ((lane & (32 / RS::P - 1)) == 0 && idx < K)
        buf[idx * 8 + warp] = mine;
    }
    __syncthreads();
    double a[8];
#pragma unroll
    for (int w = 0; w < 8; ++w)
      a[w] = w < RW && idx < K ? buf[idx * 8 + w] : 0.0;
#pragma unroll
    for (int m = 4; m > 0; m >>= 1)
#pragma unroll
      for (int i = 0; i < m; ++i)
        if (i + m < RW)
          a[i] += a[i + m];
#pragma unroll
    for (int k = 0; k < K; ++k)
      v[k] = __shfl_sync(0xffffffffu, a[0], RS::template owner<32>(k));
  }

  template <class F, int D>
  __global__ void __launch_bounds__(QuadShape<D>::NT, 1)
    bfgs_quad_kernel(F f, BfgsParams prm, const double* __restrict__ starts, RunOut out,
                     Control* ctl, unsigned long long* queue)
  {
    using S = QuadShape<D>;
    constexpr int NP = S::NP, Q = S::Q, Q1 = S::Q1, T = S::T, NT = S::NT, RQ = S::RQ;
    constexpr int KS = S::KS, KR = RQ - KS, RW = S::RW;
    extern __shared__ __align__(16) double sm[];
    double* Cs = sm;                                          // C, row-major
    double2* XP = reinterpret_cast<double2*>(Cs + D * D);     // {x, p}
    double2* SW = XP + D;                                     // {s, w}, deferred update
    double2* YG = SW + D;                                     // {y, g_x}
    double* pa = reinterpret_cast<double*>(YG + D);           // partial sums, Q x D
    double* pb = pa + Q * D;                                  // ...
    double2* HS = reinterpret_cast<double2*>(pb + Q * D);     // KS x T pairs of H
    double* red3 = reinterpret_cast<double*>(HS + KS * T);
    double* red7 = red3 + 64;
    long long* slot = reinterpret_cast<long long*>(red7 + 64); // run index
    int* stop_slot = reinterpret_cast<int*>(slot + 1);
    const int t = threadIdx.x, lane = t & 31;
    const bool own = t < D;           // thread t keeps coordinate t
    const bool works = t < T;
    const int c = t % NP, q = t / NP; // column pair and segment
    const double tol_sq4 = 4.0 * prm.tol * prm.tol;

    for (int e = t; e < D * NP; e += NT)
      reinterpret_cast<double2*>(Cs)[e] = reinterpret_cast<const double2*>(f.C)[e];

    // C^T x at the x of XP, into thread t < D (the CTA layout's ctx_coop)
    const auto ctx = [&]() {
      const int i = t % D, q1 = t / D;
      if (q1 < Q1) {
        double a = 0.0, a1 = 0.0;
        int j = q1;
#pragma unroll 5
        for (; j + Q1 < D; j += 2 * Q1) {
          a = fma(Cs[j * D + i], XP[j].x, a);
          a1 = fma(Cs[(j + Q1) * D + i], XP[j + Q1].x, a1);
        }
        if (j < D)
          a = fma(Cs[j * D + i], XP[j].x, a);
        pa[q1 * D + i] = a + a1;
      }
      __syncthreads();
      double b = 0.0;
      if (own)
        for (int k = 0; k < Q1; ++k)
          b += pa[k * D + t];
      __syncthreads();
      return b;
    };

    int64_t run = blockIdx.x;
    while (run < prm.n) {
      double x = own ? starts[run * D + t] : 0.0, p = 0.0;
      double H[KR][2];
#pragma unroll
      for (int r = 0; r < KR; ++r) {
        H[r][0] = q + Q * r == 2 * c ? 1.0 : 0.0;
        H[r][1] = q + Q * r == 2 * c + 1 ? 1.0 : 0.0;
      }
      if (works)
#pragma unroll
        for (int k = 0; k < KS; ++k)
          HS[k * T + t] = make_double2(q + Q * (KR + k) == 2 * c ? 1.0 : 0.0,
                                       q + Q * (KR + k) == 2 * c + 1 ? 1.0 : 0.0);
      if (own)
        XP[t] = make_double2(x, 0.0);
      if (t == 0)
        *stop_slot = load_stop(ctl);
      __syncthreads(); // C and x are in place
      {
        const double g0 = ctx();
        if (own) {
          p = -g0;
          XP[t].y = p;
        }
      }
      bool stop = *stop_slot != 0;
      long long n_eval = 1, n_grad = 1;
      int status = kUnset, iter, executed = -1;
      double fout = 0.0, gout = 0.0;
      bool pend = false; // SW holds an update not yet applied to H
      // f and ||g|| formed exactly at x
      const auto exact_at_x = [&](double& fd, double& gd) {
        __syncthreads(); // XP no longer read
        if (own)
          XP[t].x = x;
        __syncthreads();
        const double g = ctx();
        double vf[1] = {own ? fma(x, g, 0.0) : 0.0};
        quad_sum<1, RW>(vf, red3);
        fd = 0.5 * vf[0];
        double vg[1] = {own ? g * g : 0.0};
        quad_sum<1, RW>(vg, red7);
        gd = sqrt(vg[0]);
        ++n_eval;
        __syncthreads(); // red3 and red7 are free
      };

      for (iter = 0; iter < prm.max_iter; ++iter) {
        if (stop) {
          status = kStopped;
          break;
        }
        __syncthreads(); // {x, p} and {s, w} are in place
        int stop_now = 0;
        if (t == 0 && iter % kStopEvery == 0)
          stop_now = load_stop(ctl);
        // ---- C x and C p, two chains of rows a segment
        if (works) {
          double ax0 = 0.0, ax1 = 0.0, ap0 = 0.0, ap1 = 0.0;
          double bx0 = 0.0, bx1 = 0.0, bp0 = 0.0, bp1 = 0.0;
          const double2* C2 = reinterpret_cast<const double2*>(Cs) + c;
#pragma unroll
          for (int r = 0; r < (D + 2 * Q - 1) / (2 * Q); ++r) {
            const int j = q + 2 * Q * r;
            if (D % (2 * Q) == 0 || j < D) {
              const double2 e = C2[j * NP], v = XP[j];
              ax0 = fma(e.x, v.x, ax0);
              ax1 = fma(e.y, v.x, ax1);
              ap0 = fma(e.x, v.y, ap0);
              ap1 = fma(e.y, v.y, ap1);
            }
            if (D % (2 * Q) == 0 || j + Q < D) {
              const double2 e = C2[(j + Q) * NP], v = XP[j + Q];
              bx0 = fma(e.x, v.x, bx0);
              bx1 = fma(e.y, v.x, bx1);
              bp0 = fma(e.x, v.y, bp0);
              bp1 = fma(e.y, v.y, bp1);
            }
          }
          *reinterpret_cast<double2*>(pa + q * D + 2 * c) = make_double2(ax0 + bx0, ax1 + bx1);
          *reinterpret_cast<double2*>(pb + q * D + 2 * c) = make_double2(ap0 + bp0, ap1 + bp1);
        }
        __syncthreads();
        double g = 0.0, gn = 0.0; // the gradients at x and at the accepted point
        double v3[3] = {0.0, 0.0, 0.0};
        if (own) {
#pragma unroll
          for (int k = 0; k < Q; ++k) {
            g += pa[k * D + t];
            gn += pb[k * D + t];
          }
          v3[0] = x * g;
          v3[1] = p * gn;
          v3[2] = g * p;
        }
        quad_sum<3, RW>(v3, red3);
        const double best = 0.5 * v3[0];
        const double fp = 0.5 * v3[1], ddir = v3[2];
        n_eval += 2;
        const double alpha = pow2neg(model_trial(best, ddir, fp, lane));
        const double fnew = best + alpha * fma(alpha, fp, ddir);
        const bool take = fnew < best;
        const double xn = fma(alpha, p, x);
        double s = 0.0, y = 0.0, gx = 0.0;
        if (own) {
          gn = fma(alpha, gn, g);
          s = xn - x;
          y = gn - g;
          gx = take ? gn : g;
          YG[t] = make_double2(y, gx);
        }
        ++n_grad;
        __syncthreads();

        // ---- sweep: deferred update, column sums of H y and H g_x
        if (works) {
          double au0 = 0.0, au1 = 0.0, ah0 = 0.0, ah1 = 0.0;
          const auto sums = [&](double h0, double h1, double2 yg) {
            ah0 = fma(h0, yg.y, ah0);
            au0 = fma(h0, yg.x, au0);
            ah1 = fma(h1, yg.y, ah1);
            au1 = fma(h1, yg.x, au1);
          };
          if (pend) {
            const double2 sw0 = SW[2 * c], sw1 = SW[2 * c + 1];
            const auto update = [&](double& h0, double& h1, double2 sw) {
              h0 += __dadd_rn(__dmul_rn(sw.x, sw0.y), __dmul_rn(sw.y, sw0.x));
              h1 += __dadd_rn(__dmul_rn(sw.x, sw1.y), __dmul_rn(sw.y, sw1.x));
            };
#pragma unroll
            for (int r = 0; r < KR; ++r) {
              update(H[r][0], H[r][1], SW[q + Q * r]);
              sums(H[r][0], H[r][1], YG[q + Q * r]);
            }
#pragma unroll
            for (int k = 0; k < KS; ++k) {
              const int m = q + Q * (KR + k);
              if (D % Q == 0 || m < D) {
                double2 h = HS[k * T + t];
                update(h.x, h.y, SW[m]);
                HS[k * T + t] = h;
                sums(h.x, h.y, YG[m]);
              }
            }
          } else {
#pragma unroll
            for (int r = 0; r < KR; ++r)
              sums(H[r][0], H[r][1], YG[q + Q * r]);
#pragma unroll
            for (int k = 0; k < KS; ++k) {
              const int m = q + Q * (KR + k);
              if (D % Q == 0 || m < D) {
                const double2 h = HS[k * T + t];
                sums(h.x, h.y, YG[m]);
              }
            }
          }
          *reinterpret_cast<double2*>(pa + q * D + 2 * c) = make_double2(au0, au1);
          *reinterpret_cast<double2*>(pb + q * D + 2 * c) = make_double2(ah0, ah1);
        }
        if (t == 0)
          *stop_slot = stop_now;
        __syncthreads();
        double u = 0.0, h = 0.0;
        double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (own) {
#pragma unroll
          for (int k = 0; k < Q; ++k) {
            u += pa[k * D + t];
            h += pb[k * D + t];
          }
          v[0] = s * y;
          v[1] = y * u;
          v[2] = u * gx;
          v[3] = s * gx;
          v[4] = gx * h;
          v[5] = gx * gx;
        }
        quad_sum<6, RW>(v, red7);
        stop = *stop_slot != 0;
        const bool skipped = fabs(v[0]) < kMinCurvature;
        const double sg = v[3];
        double rho = 0.0, hb = 0.0, wg = 0.0;
        if (!skipped) {
          rho = 1.0 / v[0];
          hb = 0.5 * rho * fma(rho, v[1], 1.0);
          wg = hb * sg - rho * v[2];
        }
        if (take)
          x = xn;
        if (own) {
          if (!skipped) {
            const double w = fma(hb, s, -rho * u);
            p = -(h + s * wg + w * sg);
            SW[t] = make_double2(s, w);
          } else {
            p = -h;
          }
          XP[t] = make_double2(x, p);
        }
        pend = !skipped;
        // ||g|| = sqrt(g.g): taken only where it decides something (far
        // above tol^2, g.g cannot pass the test)
        if (!isfinite(v[5]) || !isfinite(fnew)) {
          status = kNonFinite;
          fout = fnew;
          gout = sqrt(v[5]);
          break;
        }
        if (v[5] <= tol_sq4 && sqrt(v[5]) < prm.tol) {
          // converged on the carried gradient: confirm on the exact one
          double fd, gd;
          exact_at_x(fd, gd);
          if (!(gd < prm.tol))
            continue;
          if (t == 0)
            note_converged(ctl, prm.required);
          status = kConverged;
          fout = fd;
          gout = gd;
          break;
        }
        if (!take && skipped && !(prm.flags & kFlagNoFixedPoint)) {
          executed = iter + 1;
          iter = prm.max_iter;
          break;
        }
      }
      if (status == kUnset || status == kStopped) {
        if (status == kUnset)
          status = kSurrender;
        exact_at_x(fout, gout);
      }
      if (own && out.x)
        out.x[run * D + t] = x;
      if (t == 0) {
        if (out.fval)
          out.fval[run] = fout;
        if (out.status)
          out.status[run] = status;
        if (out.iter)
          out.iter[run] = iter;
        if (out.gnorm)
          out.gnorm[run] = gout;
        if (out.counters) {
          out.counters[3 * run + 0] = executed >= 0 ? executed : iter;
          out.counters[3 * run + 1] = n_eval;
          out.counters[3 * run + 2] = n_grad;
        }
        *slot = (long long)gridDim.x + (long long)atomicAdd(queue, 1ull);
      }
      __syncthreads();
      run = *slot;
      __syncthreads();
    }
  }

} // namespace zb
