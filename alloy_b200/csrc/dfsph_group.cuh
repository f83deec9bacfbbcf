// SPDX-License-Identifier: Apache-2.0
// A whole pressure solve as ONE cooperative launch (the solve of pressure.py:196-480 with the iteration loops of
// solve_driver.py:121-186 and krylov.py:254-297): the start, every iteration with its stop tests, and the velocity
// update, in phases separated by grid-wide barriers. The per-particle arithmetic is that of the one-kernel-per-phase
// path (solve_init_one, pressure_accel, accel_divergence, jacobi_update, apply_one), the error sums follow the same
// chunks and trees, so the results are the same bits.
//
// What bounded the one-kernel-per-phase path: a Jacobi iteration was four graph nodes (acceleration, update, stop test,
// loop condition) and a CG iteration ten, each some microseconds of launch, ramp and tail around 1 to 5 us of gathers
// on a world of a few ten thousand particles; the CG launches covered every particle until the slowest world had
// converged.
//
// Work of the iterations: runs of 32 particles (a warp each) of the worlds still iterating: with one world its liquid
// range; with more, a list that every stop test writes anew for the next iteration, in any order (no result depends on
// it). With one world every block folds the chunk partials of the stop test itself, so its result needs no further
// barrier; with more, one warp per world does, and a barrier publishes it.
//
// Every barrier wait is bounded: a wait that gives up sets the status word and its block leaves; every block leaves at
// its next barrier once the status is set, and the host reports the solve as failed instead of results.
#pragma once

#include "dfsph_kernels.cuh"

namespace adf {

// Threads of a block and blocks per SM: one block of up to 1,024 threads of 64 registers, or two of up to 640 of 48 (a
// quarter more threads, each a sixth dearer by the spills and the narrower share of the L1: taken where it saves rounds
// over the liquid; 32 worlds of 5,120: 5.59 ms deep, 5.28 wide; 403,200 particles: 6.24 deep, 6.82 wide).
constexpr int GRID_BLOCK = 1024, WIDE_BLOCK = 640;
constexpr int RUN = 32;                             // particles of a list entry

// Counters of one solve (zeroed before it): barrier arrivals on a line of their own, then the two lists' lengths, each
// one 64-bit word (worlds << 44 | items << 22 | chunks) that a world joins with one atomic.
constexpr int CT_ARRIVE = 0, CT_LISTS = 32, CT_CLAMPED = 36, CT_SIZE = 64;
constexpr int LIST_BITS = 22, LIST_MASK = (1 << LIST_BITS) - 1;
constexpr long long LIST_MAX_WORLDS = (1 << (64 - 2 * LIST_BITS)) - 1, LIST_MAX_ITEMS = LIST_MASK;
static_assert(LIST_MAX_WORLDS >> (64 - 2 * LIST_BITS) == 0 && LIST_MAX_ITEMS >> LIST_BITS == 0,
              "the largest counts fit their fields of the word");

struct SolveArgs {
  int init;              // 1: the start (source, bounds, warm start) is part of this launch; 0: it ran before
  int* ctr;              // [CT_SIZE]
  int2* items[2];        // lists of the running and the next iteration: (first particle, world << 6 | particles)
  int* chunks[2];        // chunks of the listed worlds
  int* worlds[2];
  unsigned extra;        // extra arrivals a barrier waits for (only the wait-expiry test sets it)
  long long wait_limit;  // polls of one wait before it gives up
  int* status;           // set to 1 when a wait gave up; [2], 8 bytes: the host word that is set with it
  int* iters_out;        // [W] the solve's statistics
  float* mean_out;
  float* max_out;        // null: not kept (divergence)
};

// The grid's barrier: false when the kernel must stop. Thread 0's release arrival follows the block's barrier, so it
// covers the block's writes; its acquire makes the other blocks' writes visible to the block after the second one.
struct GridSync {
  unsigned epoch, expect;
  int* arrive;
  int* status;
  long long wait_limit;
  __device__ __forceinline__ bool operator()() {
    __shared__ int stop;
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(arrive), "r"(1u) : "memory");
      const unsigned target = ++epoch * expect;
      int bad = 0;
      for (long long it = 0;; ++it) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrive) : "memory");
        if (v >= target) break;
        if ((it & 63) == 63 && *(volatile int*)status != 0) {
          bad = 1;
          break;
        }
        if (it >= wait_limit) {
          atomicExch(status, 1);
          *reinterpret_cast<int* volatile*>(status + 2)[0] = 1;  // the host's next call sees it without a read-back
          bad = 1;
          break;
        }
      }
      stop = bad;
    }
    __syncthreads();
    return stop == 0;
  }
};

// fold256's tree over the 256 values of a block's first 8 warps (one a thread), with the maximum of m; the results in
// every thread of the block. All threads of the block call it together.
__device__ __forceinline__ void block_fold2(double& x, double& y, float& m) {
  __shared__ double sx[8], sy[8];
  __shared__ float sm[8];
  const int wid = threadIdx.x >> 5;
  if (wid < 8) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      x = x + __shfl_down_sync(0xffffffffu, x, o);
      y = y + __shfl_down_sync(0xffffffffu, y, o);
      m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    }
    if ((threadIdx.x & 31) == 0) {
      sx[wid] = x;
      sy[wid] = y;
      sm[wid] = m;
    }
  }
  __syncthreads();
  double u[8], v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    u[k] = sx[k];
    v[k] = sy[k];
    m = k == 0 ? sm[0] : fmaxf(m, sm[k]);
  }
#pragma unroll
  for (int o = 4; o >= 1; o >>= 1)
#pragma unroll
    for (int l = 0; l < o; ++l) {
      u[l] = u[l] + u[l + o];
      v[l] = v[l] + v[l + o];
    }
  x = u[0];
  y = v[0];
}

// The sums of a world's chunk partials [c0, c1), in every thread of the block (k_world_check's order: value L of the 256
// is the sum of partials L, L + 256, ...).
__device__ __forceinline__ void fold_world(const DevP& P, int c0, int c1, double& x, double& y, float& mx) {
  x = y = 0.0;
  mx = -3.4e38f;
  if (threadIdx.x < 256)
    for (int k = c0 + threadIdx.x; k < c1; k += 256) {
      const double2 pk = __ldcg(&P.part2[k]);
      x = x + pk.x;
      y = y + pk.y;
      mx = fmaxf(mx, __ldcg(&P.part_max[k]));
    }
  block_fold2(x, y, mx);
}

// Chunk c = [b, e) of the caller's order, by a warp: the sums of x and y = value(i, x, y) and the maximum of y.
template <class F>
__device__ __forceinline__ void fold_chunk(const DevP& P, int c, int b, int e, F value) {
  float m = -3.4e38f;
  double x2, y2;
  fold256_warp2([&](int L, double& x, double& y) {
    float vx = 0.0f, vy = 0.0f;
    if (b + L < e) {
      value(b + L, vx, vy);
      m = fmaxf(m, vy);
    }
    x = (double)vx;
    y = (double)vy;
  }, x2, y2);
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) {
    P.part2[c] = make_double2(x2, y2);
    P.part_max[c] = m;
  }
}

// World w's partials folded by a warp: f(x, y, mx) with the sums (in lane 0) and the maximum.
__device__ __forceinline__ void fold_world_warp(const DevP& P, int w, double& x, double& y, float& mx) {
  const int b = P.world_chunk_start[w], e = P.world_chunk_start[w + 1];
  float m = -3.4e38f;
  fold256_warp2([&](int L, double& vx, double& vy) {
    vx = 0.0;
    vy = 0.0;
    for (int c = b + L; c < e; c += 256) {
      const double2 pk = __ldcg(&P.part2[c]);
      vx = vx + pk.x;
      vy = vy + pk.y;
      m = fmaxf(m, __ldcg(&P.part_max[c]));
    }
  }, x, y);
  mx = warp_max(m);
}

// A world's statistics after its stop test (one thread); true while it goes on.
__device__ __forceinline__ bool record_test(const DevP& P, int w, int it, int n, double sum, float mx, bool count_work) {
  const float mean = (float)(sum / (double)n);
  const bool done = stop_test(P, w, it, mean, mx);
  P.iters[w] = it;
  P.err_mean[w] = mean;
  P.emax[w] = mx;
  if (done) P.converged[w] = 1;
  if (P.iter_work && count_work) atomicAdd(P.iter_work, (unsigned long long)n);
  return !done;
}

template <bool MS, bool CG, bool ONE>
struct GridSolve {
  // gathers in flight of the neighbour loops (and as many row entries loaded ahead)
  static constexpr int NBX = 4 | (MS ? MS_FLAG : 0);
  const DevP& P;
  const SolveArgs& A;
  GridSync sync;
  int cur;           // the lists of the running iteration, and their lengths
  int n_worlds, n_items, n_chunks;
  int run0;          // this warp's first list entry
  int2 first;        // (its value)
  // ONE: the world's liquid range, caller range and chunks
  int lb, le, ib, ie, c0, c1;

  __device__ __forceinline__ int tid() const { return blockIdx.x * blockDim.x + threadIdx.x; }
  __device__ __forceinline__ int threads() const { return gridDim.x * blockDim.x; }
  // This warp's turn at a list of folds: one for each block before a second, since the warps of an SM share its shuffles.
  __device__ __forceinline__ int turn() const { return (threadIdx.x >> 5) * gridDim.x + blockIdx.x; }

  // f(p, w) for the particles of every listed run. Warps take runs in turn, so that an SM's warps work on neighbouring
  // bricks of cells (runs handed out by a counter evened the SMs out, but the phases of a million particles, bound by
  // the L1's gathers on every SM, ended no sooner).
  template <class F>
  __device__ __forceinline__ void for_particles(F f) {
    if constexpr (ONE) {
      for (int p = lb + tid(); p < le; p += threads()) f(p, 0);
    } else {
      const int lane = threadIdx.x & 31, step = threads() / RUN;
      int2 r = first;
      for (int i = run0; i < n_items; i += step) {
        int2 next = r;
        if (i + step < n_items) next = __ldcg(&A.items[cur][i + step]);
        if (lane < (r.y & 63)) f(r.x + lane, r.y >> 6);
        r = next;
      }
    }
  }

  // The lengths of the lists in `cur`, and this warp's first run.
  __device__ __forceinline__ void open_lists() {
    if constexpr (ONE) {
      n_worlds = 1;
      n_chunks = c1 - c0;
    } else {
      const unsigned long long v = __ldcg(lists() + cur);
      n_worlds = (int)(v >> (2 * LIST_BITS));
      n_items = (int)(v >> LIST_BITS) & LIST_MASK;
      n_chunks = (int)v & LIST_MASK;
      // Its place among them is the warp's own, so that an SM's warps take neighbouring runs; where there are fewer runs
      // than warps (few worlds still iterate), the blocks take even shares and no SM idles while others work through 32
      // warps' gathers.
      run0 = tid() / RUN;
      if (n_items < threads() / RUN) {
        const int share = (n_items + (int)gridDim.x - 1) / (int)gridDim.x, wid = threadIdx.x / RUN;
        run0 = wid < share ? (int)blockIdx.x * share + wid : n_items;
      }
      if (run0 < n_items) first = __ldcg(&A.items[cur][run0]);
    }
  }
  __device__ __forceinline__ unsigned long long* lists() const {
    return reinterpret_cast<unsigned long long*>(A.ctr + CT_LISTS);
  }

  // acc = pressure acceleration of the field (kap, kr = kap / rho0); `skip(w)`: the world is left out
  template <class S>
  __device__ __forceinline__ void accel(float* kap, float* kr, S skip) {
    DevP Q = P;
    Q.kappa = kap;
    Q.kr = kr;
    for_particles([&](int p, int w) {
      if (skip(w)) return;
      float ax, ay, az;
      pressure_accel<NBX>(Q, p, P.pos[p], ax, ay, az);
      P.acc[p] = make_float4(ax, ay, az, 0.0f);
    });
  }

  // f(p, w, rho0, Ar), Ar the divergence of the accelerations
  template <class S, class F>
  __device__ __forceinline__ void divergence(S skip, F f) {
    for_particles([&](int p, int w) {
      if (skip(w)) return;
      const float r0 = P.vel[p].w;
      f(p, w, r0, accel_divergence<NBX>(P, p, 1.0f / r0));
    });
  }

  // The listed worlds' chunk partials: sums of x and y = value(i, x, y) and the maximum of y, per chunk 256 threads.
  template <class F>
  __device__ __forceinline__ void fold_chunks(F value) {
    for (int k = turn(); k < n_chunks; k += threads() >> 5) {  // a warp each
      const int c = ONE ? c0 + k : __ldcg(&A.chunks[cur][k]);
      const int b = ONE ? ib + 256 * k : P.chunk_begin[c];
      fold_chunk(P, c, b, ONE ? min(b + 256, ie) : P.chunk_end[c], value);
    }
  }

  // ONE: the world's sums from its chunk partials, in every thread of the block.
  __device__ __forceinline__ void fold_one(double& x, double& y, float& mx) { fold_world(P, c0, c1, x, y, mx); }

  // Several worlds: f(w, x, y, mx) in lane 0 of the warp that folds world w.
  template <class F>
  __device__ __forceinline__ void fold_worlds(F f) {
    for (int k = turn(); k < n_worlds; k += threads() >> 5) {
      const int w = __ldcg(&A.worlds[cur][k]);
      double x, y;
      float m;
      fold_world_warp(P, w, x, y, m);
      const int keep = f(w, x, y, m);
      if (__shfl_sync(0xffffffffu, keep, 0)) list_world(w, cur ^ 1);
    }
  }

  // World w's items and chunks into list `to` (a whole warp; the liquid range is not empty).
  __device__ __forceinline__ void list_world(int w, int to) {
    const int lane = threadIdx.x & 31;
    const int2 r = P.wrange[w];
    const int b = P.world_chunk_start[w], e = P.world_chunk_start[w + 1];
    const int segs = (r.y - r.x + RUN - 1) / RUN;
    unsigned long long at = 0;
    if (lane == 0) {
      at = atomicAdd(lists() + to, (1ull << (2 * LIST_BITS)) | ((unsigned long long)segs << LIST_BITS) |
                                       (unsigned long long)(e - b));
      A.worlds[to][at >> (2 * LIST_BITS)] = w;
    }
    at = __shfl_sync(0xffffffffu, at, 0);
    const int at_i = (int)(at >> LIST_BITS) & LIST_MASK, at_c = (int)at & LIST_MASK;
    for (int k = lane; k < segs; k += 32) {
      const int p = r.x + k * RUN;
      A.items[to][at_i + k] = make_int2(p, (w << 6) | min(RUN, r.y - p));
    }
    for (int k = lane; k < e - b; k += 32) A.chunks[to][at_c + k] = b + k;
  }

  // The next lists' lengths back to zero: in a phase between the last reading of these lists (the previous iteration's)
  // and the stop tests that write them.
  __device__ __forceinline__ void clear_next() {
    if (!ONE && tid() == 0) lists()[cur ^ 1] = 0ull;
  }

  __device__ __forceinline__ bool test_world(int w, int it, int n, double sum, float mx) {
    return record_test(P, w, it, n, sum, mx, !CG);
  }

  __device__ __forceinline__ bool jacobi(int it) {
    const auto all = [](int) { return false; };
    for (int loop = 0; loop < P.max_it + 2; ++loop) {
      clear_next();
      accel(P.kappa, P.kr, all);
      if (!sync()) return false;
      divergence(all, [&](int p, int, float r0, float ar) { jacobi_update(P, p, r0, ar); });
      if (!sync()) return false;
      fold_chunks([&](int i, float& x, float& y) { x = y = P.err_orig[i]; });
      if (!sync()) return false;
      if constexpr (ONE) {
        double x, sum;
        float mx;
        fold_one(x, sum, mx);
        mx = maxr(mx, 0.0f);
        ++it;
        if (tid() == 0) test_world(0, it, le - lb, sum, mx);
        if (stop_test(P, 0, it, (float)(sum / (double)(le - lb)), mx)) return true;
      } else {
        fold_worlds([&](int w, double, double sum, float mx) -> int {
          if ((threadIdx.x & 31) != 0) return 0;
          const int2 r = P.wrange[w];
          return test_world(w, P.iters[w] + 1, r.y - r.x, sum, maxr(mx, 0.0f)) ? 1 : 0;
        });
        if (!sync()) return false;
        cur ^= 1;
        open_lists();
        if (n_worlds == 0) return true;
      }
    }
    return true;
  }

  // z = M^-1 r on the active set, the error of the bound-constrained residual, and (r.z, error) of one particle after
  // its w update; `act0` its activity before, the returned value its activity after (k_cg_apply_finish's finish).
  __device__ __forceinline__ int finish(int p, float wv, int act0, float kap, float scale, bool div) {
    const int act = (act0 || wv < 0.0f) ? 1 : 0;
    const float zi = act ? ((-wv) * P.alpha[p]) / scale : 0.0f;
    P.cg_z[p] = zi;
    float e = maxr(-wv, 0.0f);
    if (kap > P.lower[p]) e = fabsf(wv);
    if (div) {
      if (P.neff[p] < P.min_nb) e = 0.0f;
      e = e * P.dt;
    }
    const int i = P.id_of[p];
    P.err_orig[i] = e;
    P.cg_pair[i] = make_float2(-wv * zi, e);
    return act;
  }

  // The projected CG (krylov.py:254-297). The finish of an iteration (activation, z, error) runs with the step as if
  // nothing was clamped; only in worlds whose step did clamp a variable does the correction product follow, and the
  // finish is done again there from the activity before it (bit 0 of cg_act; bit 1 holds the activity after it). The
  // correction's two phases are skipped when no world clamped anything. cg_restart and cg_act_new count on from
  // iteration to iteration: a change since the last one is what matters.
  __device__ __forceinline__ bool cg(int it) {
    const float dt = P.dt;
    const bool div = P.mode == 0;
    const float scale = div ? dt : dt * dt;
    const auto all = [](int) { return false; };
    const auto pairs = [&](int i, float& x, float& y) {
      const float2 v = P.cg_pair[i];
      x = v.x;
      y = v.y;
    };
    accel(P.kappa, P.kr, all);
    if (!sync()) return false;
    divergence(all, [&](int p, int, float r0, float ar) {
      const float t = ADF_FMA(-P.reg[p], P.kappa[p], ar);
      const float wv = -(scale * t) - (div ? P.src[p] : P.src[p] - 1.0f);
      P.cg_w[p] = wv;
      const int act = (P.kappa[p] > P.lower[p] || wv < 0.0f) ? 1 : 0;
      const float zi = act ? ((-wv) * P.alpha[p]) / scale : 0.0f;
      P.cg_act[p] = 3 * act;
      P.cg_z[p] = zi;
      P.cg_pd[p] = zi;
      P.cg_pdr[p] = zi / r0;
      P.cg_pair[P.id_of[p]] = make_float2(-wv * zi, 0.0f);
    });
    if (!sync()) return false;
    fold_chunks(pairs);
    if (!sync()) return false;
    double rz = 0.0;  // ONE
    if constexpr (ONE) {
      double y;
      float mx;
      fold_one(rz, y, mx);
    } else {
      fold_worlds([&](int w, double x, double, float) -> int {
        if ((threadIdx.x & 31) == 0) P.cg_rz[w] = x;
        return 0;
      });
      // read first in the stop test's fold, barriers later
    }
    int acts = 0;
    if constexpr (ONE) acts = __ldcg(&P.cg_act_new[0]);
    for (int loop = 0; loop < P.max_it + 2; ++loop) {
      clear_next();
      accel(P.cg_pd, P.cg_pdr, all);
      if (!sync()) return false;
      divergence(all, [&](int p, int, float, float ar) {
        const float v = -(scale * ADF_FMA(-P.reg[p], P.cg_pd[p], ar));
        P.cg_pair[P.id_of[p]] = make_float2(P.cg_pd[p] * v, 0.0f);
        P.cg_ap[p] = v;
      });
      if (!sync()) return false;
      fold_chunks(pairs);
      if (!sync()) return false;
      float a1 = 0.0f;
      if constexpr (ONE) {
        double pap, y;
        float mx;
        fold_one(pap, y, mx);
        a1 = (float)(pap > 1.0e-30 ? rz / pap : 0.0);
      } else {
        fold_worlds([&](int w, double pap, double, float) -> int {
          if ((threadIdx.x & 31) == 0) {
            P.cg_sums[w] = make_double2(pap > 1.0e-30 ? P.cg_rz[w] / pap : 0.0, 0.0);  // the step length
            P.cg_restart[w] = 0;
            P.cg_act_new[w] = 0;
          }
          return 0;
        });
        if (!sync()) return false;
      }
      for_particles([&](int p, int w) {
        const float a = ONE ? a1 : (float)P.cg_sums[w].x;
        const float r0 = P.vel[p].w;
        float c = 0.0f, kap = P.kappa[p];
        int act = P.cg_act[p] >> 1;
        if (act) {
          float k = ADF_FMA(a, P.cg_pd[p], kap);
          const float lb = P.lower[p];
          if (k < lb) {
            c = lb - k;
            k = lb;
            act = 0;
            P.cg_restart[w] = loop + 1;
            A.ctr[CT_CLAMPED] = loop + 1;
          }
          P.kappa[p] = k;
          P.kr[p] = k / r0;
          kap = k;
        }
        P.cg_corr[p] = c;
        P.cg_corrr[p] = c / r0;
        const float wv = ADF_FMA(a, P.cg_ap[p], P.cg_w[p]);
        P.cg_w[p] = wv;
        const int now = finish(p, wv, act, kap, scale, div);
        if (now && !act) P.cg_act_new[w] = ONE ? acts + 1 : 1;
        P.cg_act[p] = act | (now << 1);
      });
      if (!sync()) return false;
      const bool clamped = __ldcg(&A.ctr[CT_CLAMPED]) == loop + 1;
      if (clamped) {  // w += A corr, and the finish again
        const auto kept = [&](int w) { return !ONE && __ldcg(&P.cg_restart[w]) == 0; };
        accel(P.cg_corr, P.cg_corrr, kept);
        if (!sync()) return false;
        divergence(kept, [&](int p, int, float, float ar) {
          const float t = ADF_FMA(-P.reg[p], P.cg_corr[p], ar);
          const float wv = -(scale * t) + P.cg_w[p];
          P.cg_w[p] = wv;
          const int act = P.cg_act[p] & 1;
          P.cg_act[p] = act | (finish(p, wv, act, P.kappa[p], scale, div) << 1);
        });
        if (!sync()) return false;
      }
      fold_chunks(pairs);
      if (!sync()) return false;
      float beta1 = 0.0f;
      if constexpr (ONE) {
        double rz_new, sum;
        float mx;
        fold_one(rz_new, sum, mx);
        mx = maxr(mx, 0.0f);
        ++it;
        const int now = __ldcg(&P.cg_act_new[0]);
        beta1 = (float)((!clamped && now == acts && rz > 1.0e-30) ? rz_new / rz : 0.0);
        acts = now;
        rz = rz_new;
        if (tid() == 0) test_world(0, it, le - lb, sum, mx);
        if (stop_test(P, 0, it, (float)(sum / (double)(le - lb)), mx)) return true;
      } else {
        fold_worlds([&](int w, double rz_new, double sum, float mx) -> int {
          if ((threadIdx.x & 31) != 0) return 0;
          const int2 r = P.wrange[w];
          const bool same = P.cg_restart[w] == 0 && P.cg_act_new[w] == 0;
          P.cg_step[w] = (same && P.cg_rz[w] > 1.0e-30) ? rz_new / P.cg_rz[w] : 0.0;
          P.cg_rz[w] = rz_new;
          return test_world(w, P.iters[w] + 1, r.y - r.x, sum, maxr(mx, 0.0f)) ? 1 : 0;
        });
        if (!sync()) return false;
        cur ^= 1;
        open_lists();
        if (n_worlds == 0) return true;
      }
      for_particles([&](int p, int w) {
        const float beta = ONE ? beta1 : (float)P.cg_step[w];
        const float pd = (P.cg_act[p] >> 1) ? ADF_FMA(beta, P.cg_pd[p], P.cg_z[p]) : 0.0f;
        P.cg_pd[p] = pd;
        P.cg_pdr[p] = pd / P.vel[p].w;
      });
      if (!sync()) return false;
    }
    return true;
  }

  __device__ __forceinline__ void run() {
    const int nf = P.nfw[0];
    cur = 0;
    int it = 0;
    if constexpr (ONE) {
      const int2 r = P.wrange[0];
      lb = r.x;
      le = r.y;
      ib = P.skin_ws[0];
      ie = P.skin_ws[1];
      c0 = P.world_chunk_start[0];
      c1 = P.world_chunk_start[1];
      if (!A.init) it = P.iters[0];
    }
    if (CG)
      for (int i = tid(); i < P.n; i += threads()) P.cg_pair[i] = make_float2(0.0f, 0.0f);
    if (A.init) {
      for (int i = tid(); i < P.n; i += threads()) P.err_orig[i] = 0.0f;
      for (int p = tid(); p < nf; p += threads()) solve_init_one<NBX>(P, p);
    }
    // k_begin_solve for every world, and the first lists
    bool open = false;
    if constexpr (ONE) {
      open = le > lb && (A.init || P.converged[0] == 0);
      if (A.init && tid() == 0) {
        P.iters[0] = 0;
        P.err_mean[0] = 0.0f;
        P.emax[0] = 0.0f;
      }
      if (P.iter_work && CG && open && tid() == 0) atomicAdd(P.iter_work, (unsigned long long)(le - lb));
    } else {
      for (int w = tid() >> 5; w < P.W; w += threads() >> 5) {
        const int2 r = P.wrange[w];
        const bool on = r.y > r.x && (A.init || P.converged[w] == 0);
        __syncwarp();
        if ((threadIdx.x & 31) == 0) {
          if (A.init) {
            P.iters[w] = 0;
            P.err_mean[w] = 0.0f;
            P.emax[w] = 0.0f;
            P.converged[w] = on ? 0 : 1;
          }
          if (CG && on && P.iter_work) atomicAdd(P.iter_work, (unsigned long long)(r.y - r.x));
        }
        if (on) list_world(w, 0);
      }
    }
    if (!sync()) return;
    open_lists();
    if constexpr (!ONE) open = n_worlds > 0;
    if (open) {
      if constexpr (CG) {
        if (!cg(it)) return;
      } else {
        if (!jacobi(it)) return;
      }
    }
    for (int p = tid(); p < nf; p += threads()) apply_one<NBX>(P, p);
    // the statistics: written by the last stop test of each world, barriers ago (with one world, by this thread)
    for (int w = tid(); w < P.W; w += threads()) {
      A.iters_out[w] = P.iters[w];
      A.mean_out[w] = P.err_mean[w];
      if (A.max_out) A.max_out[w] = P.emax[w];
    }
  }
};

template <bool MS, bool CG, bool ONE, bool WIDE>
__global__ void __launch_bounds__(WIDE ? WIDE_BLOCK : GRID_BLOCK, WIDE ? 2 : 1)
k_grid_solve(const __grid_constant__ DevP P, const __grid_constant__ SolveArgs A) {
  GridSolve<MS, CG, ONE> g{P, A, GridSync{0u, gridDim.x + A.extra, A.ctr + CT_ARRIVE, A.status, A.wait_limit}};
  g.run();
}

}  // namespace adf
