// SPDX-License-Identifier: Apache-2.0
// The cooperative pressure solve (dfsph_group.cuh) of a model small enough for a thread per particle: at most
// SMALL_BLOCK liquid particles per SM. A particle's row stays on its SM for the whole solve, in shared memory: the
// pair's offset r_ij, gradient factor F, neighbour and neighbour's mass, 24 bytes an entry, ROW_RES entries a particle
// (the few rows with more read the rest from memory as the other paths do). Its own state (kappa, the CG vectors, source,
// bounds, wall gradients) stays in the thread's registers. A phase then gathers one thing per neighbour, the value that
// changes (kappa / rho0 or the direction, 4 bytes, for the acceleration; the acceleration, 16 bytes, for its
// divergence), all gathers of a row in flight at once, instead of rows, positions and that value.
//
// A step of such a model is one launch after its rows and walls (k_small_step): density, both solves, XSPH and the finish
// read the rows once. Against a launch for each: four steps of 2,016 particles 673 -> 615 us, of 8,000 with reports 1,074
// -> 1,010, of the 30k column 2,563 -> 2,514, of the 30k tank 1,971 -> 1,914.
//
// What bounded these phases before: on 30,720 particles an acceleration or divergence phase took 7 to 9 us, 21 MB
// through the L2 after every barrier's L1 invalidation, in eight dependent trips a thread.
//
// The arithmetic and its order are the other paths': the offsets, products and sums are formed by the same operations
// from the same values, so the results are the same bits.
#pragma once

#include "dfsph_group.cuh"

namespace adf {

constexpr int SMALL_BLOCK = 256;  // threads of a block, one block per SM
constexpr int ROW_RES = 36;       // row entries kept in shared memory
constexpr size_t SMALL_SMEM = (size_t)ROW_RES * SMALL_BLOCK * (sizeof(float4) + sizeof(int2));

template <bool MS, bool CG, bool ONE>
struct SmallSolve {
  static constexpr int NS = MS ? 4 : 1;  // wall slots
  static constexpr int NB = 12;          // gathers in flight (a divisor of ROW_RES)
  const DevP& P;
  const SolveArgs& A;
  GridSync sync;
  float4* geo;  // [ROW_RES][SMALL_BLOCK] r_ij, F
  int2* jm;     // [ROW_RES][SMALL_BLOCK] j, bits of m_j
  int p, w, c, id;
  bool on;      // this thread has a particle, of a world that still iterates
  bool mine;    // this thread has a particle
  bool few;     // too few neighbours for the divergence solve
  int ns;
  float gx[NS], gy[NS], gz[NS];  // wall gradients
  float r0, reg, alpha, lower, src, kap;
  float ax, ay, az;  // the particle's acceleration of the running product
  float dt, scale;
  bool div;
  int c0, c1, ib, ie, n_one;  // ONE: chunks, caller range and liquid

  __device__ __forceinline__ int tid() const { return blockIdx.x * SMALL_BLOCK + threadIdx.x; }
  __device__ __forceinline__ int threads() const { return gridDim.x * SMALL_BLOCK; }
  // this warp's turn at a list of folds: one for each block before a second (GridSolve::turn)
  __device__ __forceinline__ int warp() const { return (threadIdx.x >> 5) * gridDim.x + blockIdx.x; }
  __device__ __forceinline__ int warps() const { return threads() >> 5; }
  __device__ __forceinline__ int at(int k) const { return k * SMALL_BLOCK + threadIdx.x; }

  // The row into shared memory, as the density pass left it.
  __device__ __forceinline__ void load(const float4& xi) {
    const int m = min(c, ROW_RES);
    for (int k = 0; k < m; k += NB) {
      int j[NB];
      float f[NB];
      load_row_batch_f(P, p, m, k, j, f);
      float4 x[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) x[u] = P.pos[j[u]];
#pragma unroll
      for (int u = 0; u < NB; ++u)
        if (k + u < m) {
          geo[at(k + u)] = make_float4(xi.x - x[u].x, xi.y - x[u].y, xi.z - x[u].z, f[u]);
          jm[at(k + u)] = make_int2(j[u], __float_as_int(x[u].w));
        }
    }
    walls();
  }

  // The density pass (density_one) with the row kept; only entries past the resident ones are written out.
  __device__ __forceinline__ void load_density(const float4& xi) {
    const float inv_r0 = 1.0f / r0;
    const float bi = xi.w * inv_r0;
    float rho = xi.w * P.kc.sigma, Gx = 0.0f, Gy = 0.0f, Gz = 0.0f, sq = 0.0f;
    for (int k = 0; k < c; k += NB) {
      int j[NB];
      load_row_batch(P, p, c, k, j);
      float4 x[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) x[u] = P.pos[j[u]];
#pragma unroll
      for (int u = 0; u < NB; ++u)
        if (k + u < c) {
          const float rx = xi.x - x[u].x, ry = xi.y - x[u].y, rz = xi.z - x[u].z;
          const float r2 = dot_plain(rx, ry, rz, rx, ry, rz);
          float W, F;
          wf(P.kc, r2, W, F);
          if (k + u < ROW_RES) {
            geo[at(k + u)] = make_float4(rx, ry, rz, F);
            jm[at(k + u)] = make_int2(j[u], __float_as_int(x[u].w));
          } else {
            P.nbrjf[(size_t)(k + u) * P.n + p] = make_int2(j[u], __float_as_int(F));
          }
          rho = ADF_FMA(x[u].w, W, rho);
          const float a = x[u].w * inv_r0;
          const float aF = a * F;
          Gx = ADF_FMA(aF, rx, Gx);
          Gy = ADF_FMA(aF, ry, Gy);
          Gz = ADF_FMA(aF, rz, Gz);
          sq = ADF_FMA(bi * a, (F * F) * r2, sq);
        }
    }
    density_finish<MS>(P, p, c, inv_r0, rho, Gx, Gy, Gz, sq);
    walls();
  }

  // The walls' gradients into registers.
  __device__ __forceinline__ void walls() {
    if constexpr (MS) {
      ns = P.slot_cnt[p];
#pragma unroll
      for (int b = 0; b < NS; ++b) {
        const float4 g = b < ns ? P.slot_g[slot_at(P, b, p)] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        gx[b] = g.x;
        gy[b] = g.y;
        gz[b] = g.z;
      }
    } else {
      const float4 g = P.slot_g[p];
      ns = g.w >= 0.0f ? 1 : 0;
      gx[0] = g.x;
      gy[0] = g.y;
      gz[0] = g.z;
    }
  }

  // f(value, r_ij and F, m_j) for the row's entries in order, value = gather(j)
  template <class V, class G, class F>
  __device__ __forceinline__ void for_row(G gather, F f) {
    const int m = min(c, ROW_RES);
#pragma unroll 1
    for (int k = 0; k < m; k += NB) {
      V v[NB];
      float mj[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u)
        if (k + u < m) {
          const int2 e = jm[at(k + u)];
          v[u] = gather(e.x);
          mj[u] = __int_as_float(e.y);
        }
#pragma unroll
      for (int u = 0; u < NB; ++u)
        if (k + u < m) f(v[u], geo[at(k + u)], mj[u]);
    }
    for (int k = m; k < c; ++k) {  // past the resident entries
      const int2 e = row_entry(P, p, k);
      const float4 xi = P.pos[p], xj = P.pos[e.x];
      f(gather(e.x), make_float4(xi.x - xj.x, xi.y - xj.y, xi.z - xj.z, __int_as_float(e.y)), xj.w);
    }
  }

  // pressure_accel of the field with own values kk and ki = kk / rho0 and neighbours' kr
  __device__ __forceinline__ void accel_of(const float* kr, float kk, float ki, float& x, float& y, float& z) {
    x = y = z = 0.0f;
    for_row<float>([&](int j) { return kr[j]; },
                   [&](float kj, const float4& g, float mj) {
                     const float cF = (mj * (ki + kj)) * g.w;
                     x = ADF_FMA(-cF, g.x, x);
                     y = ADF_FMA(-cF, g.y, y);
                     z = ADF_FMA(-cF, g.z, z);
                   });
#pragma unroll
    for (int b = 0; b < NS; ++b)
      if (b < ns) {
        x = ADF_FMA(-kk, gx[b], x);
        y = ADF_FMA(-kk, gy[b], y);
        z = ADF_FMA(-kk, gz[b], z);
      }
  }
  __device__ __forceinline__ void accel(const float* kr, float kk, float ki) {
    accel_of(kr, kk, ki, ax, ay, az);
    P.acc[p] = make_float4(ax, ay, az, 0.0f);
  }

  // accel_divergence
  __device__ __forceinline__ float divergence() {
    const float inv_r0 = 1.0f / r0;
    float ar = 0.0f;
    for_row<float4>([&](int j) { return P.acc[j]; },
                    [&](const float4& aj, const float4& g, float mj) {
                      const float aF = (mj * inv_r0) * g.w;
                      ar = ADF_FMA(aF, dotf(ax - aj.x, ay - aj.y, az - aj.z, g.x, g.y, g.z), ar);
                    });
#pragma unroll
    for (int b = 0; b < NS; ++b)
      if (b < ns) ar = ar + dotf(ax, ay, az, gx[b], gy[b], gz[b]);
    return ar;
  }

  // Partials of the chunks of the worlds still iterating.
  template <class F>
  __device__ __forceinline__ void fold_chunks(F value) {
    if constexpr (ONE) {
      for (int c = c0 + warp(); c < c1; c += warps()) {
        const int b = ib + 256 * (c - c0);
        fold_chunk(P, c, b, min(b + 256, ie), value);
      }
    } else {
      for (int c = warp(); c < P.n_chunks; c += warps())
        if (!__ldcg(&P.converged[P.chunk_world[c]])) fold_chunk(P, c, P.chunk_begin[c], P.chunk_end[c], value);
    }
  }

  // Several worlds: f(w, x, y, mx) in lane 0 of the warp of each world still iterating.
  template <class F>
  __device__ __forceinline__ void fold_worlds(F f) {
    for (int v = warp(); v < P.W; v += warps()) {
      if (__ldcg(&P.converged[v])) continue;
      double x, y;
      float m;
      fold_world_warp(P, v, x, y, m);
      if ((threadIdx.x & 31) == 0) f(v, x, y, m);
    }
  }

  // Several worlds: counts the worlds that go on after a stop test (CT_LISTS + parity of the iteration), cleared two
  // phases before.
  __device__ __forceinline__ int* open_count(int loop) { return A.ctr + CT_LISTS + (loop & 1); }

  __device__ __forceinline__ void update(float ar) {  // jacobi_update
    ar = ADF_FMA(-reg, kap, ar);
    ar = ar * (div ? dt : dt * dt);
    const float inv = div ? 1.0f / dt : 1.0f / (dt * dt);
    const float s = div ? -src : 1.0f - src;
    const float r = s - ar;
    const float knew = maxr(kap - ((P.omega * r) * alpha) * inv, lower);
    kap = knew;
    P.kr[p] = knew / r0;
    float e = maxr(-r, 0.0f);
    if (knew > lower) e = fabsf(r);
    if (div) {
      if (few) e = 0.0f;
      e = e * dt;
    }
    P.err_orig[id] = e;
  }

  __device__ __forceinline__ bool jacobi(int it) {
    for (int loop = 0; loop < P.max_it + 2; ++loop) {
      if (!ONE && tid() == 0) *open_count(loop) = 0;
      if (on) accel(P.kr, kap, kap / r0);
      if (!sync()) return false;
      if (on) update(divergence());
      if (!sync()) return false;
      fold_chunks([&](int i, float& x, float& y) { x = y = P.err_orig[i]; });
      if (!sync()) return false;
      if constexpr (ONE) {
        double x, sum;
        float mx;
        fold_world(P, c0, c1, x, sum, mx);
        mx = maxr(mx, 0.0f);
        ++it;
        if (tid() == 0) record_test(P, 0, it, n_one, sum, mx, true);
        if (stop_test(P, 0, it, (float)(sum / (double)n_one), mx)) return true;
      } else {
        fold_worlds([&](int v, double, double sum, float mx) {
          const int2 r = P.wrange[v];
          if (record_test(P, v, P.iters[v] + 1, r.y - r.x, sum, maxr(mx, 0.0f), true)) atomicAdd(open_count(loop), 1);
        });
        if (!sync()) return false;
        if (__ldcg(open_count(loop)) == 0) return true;
        if (on) on = __ldcg(&P.converged[w]) == 0;
      }
    }
    return true;
  }

  // z = M^-1 r on the active set, the error, and (r.z, error) of the particle after its w update; its activity after.
  __device__ __forceinline__ int finish(float wv, int act0, float& z) {
    const int act = (act0 || wv < 0.0f) ? 1 : 0;
    z = act ? ((-wv) * alpha) / scale : 0.0f;
    float e = maxr(-wv, 0.0f);
    if (kap > lower) e = fabsf(wv);
    if (div) {
      if (few) e = 0.0f;
      e = e * dt;
    }
    P.err_orig[id] = e;
    P.cg_pair[id] = make_float2(-wv * z, e);
    return act;
  }

  // The projected CG as GridSolve::cg runs it, the particle's vectors in registers.
  __device__ __forceinline__ bool cg(int it) {
    const auto pairs = [&](int i, float& x, float& y) {
      const float2 v = P.cg_pair[i];
      x = v.x;
      y = v.y;
    };
    float wv = 0.0f, z = 0.0f, pd = 0.0f, pdr = 0.0f, ap = 0.0f;
    int act = 0;
    if (on) accel(P.kr, kap, kap / r0);
    if (!sync()) return false;
    if (on) {
      const float t = ADF_FMA(-reg, kap, divergence());
      wv = -(scale * t) - (div ? src : src - 1.0f);
      act = (kap > lower || wv < 0.0f) ? 1 : 0;
      z = act ? ((-wv) * alpha) / scale : 0.0f;
      pd = z;
      pdr = z / r0;
      P.cg_pdr[p] = pdr;
      P.cg_pair[id] = make_float2(-wv * z, 0.0f);
    }
    if (!sync()) return false;
    fold_chunks(pairs);
    if (!sync()) return false;
    double rz = 0.0;  // ONE
    int acts = 0;
    if constexpr (ONE) {
      double y;
      float mx;
      fold_world(P, c0, c1, rz, y, mx);
      acts = __ldcg(&P.cg_act_new[0]);
    } else {
      fold_worlds([&](int v, double x, double, float) { P.cg_rz[v] = x; });
    }
    for (int loop = 0; loop < P.max_it + 2; ++loop) {
      if (!ONE && tid() == 0) *open_count(loop) = 0;
      if (on) accel(P.cg_pdr, pd, pdr);
      if (!sync()) return false;
      if (on) {
        ap = -(scale * ADF_FMA(-reg, pd, divergence()));
        P.cg_pair[id] = make_float2(pd * ap, 0.0f);
      }
      if (!sync()) return false;
      fold_chunks(pairs);
      if (!sync()) return false;
      float a = 0.0f;
      if constexpr (ONE) {
        double pap, y;
        float mx;
        fold_world(P, c0, c1, pap, y, mx);
        a = (float)(pap > 1.0e-30 ? rz / pap : 0.0);
      } else {
        fold_worlds([&](int v, double pap, double, float) {
          P.cg_sums[v] = make_double2(pap > 1.0e-30 ? P.cg_rz[v] / pap : 0.0, 0.0);  // the step length
          P.cg_restart[v] = 0;
          P.cg_act_new[v] = 0;
        });
        if (!sync()) return false;
        if (on) a = (float)__ldcg(&P.cg_sums[w].x);
      }
      float corr = 0.0f;
      int now = 0;
      if (on) {
        if (act) {
          float k = ADF_FMA(a, pd, kap);
          if (k < lower) {
            corr = lower - k;
            k = lower;
            act = 0;
            P.cg_restart[w] = loop + 1;
            A.ctr[CT_CLAMPED] = loop + 1;
          }
          kap = k;
        }
        P.cg_corrr[p] = corr / r0;
        wv = ADF_FMA(a, ap, wv);
        now = finish(wv, act, z);
        if (now && !act) P.cg_act_new[w] = ONE ? acts + 1 : 1;
      }
      if (!sync()) return false;
      const bool clamped = __ldcg(&A.ctr[CT_CLAMPED]) == loop + 1;
      if (clamped) {
        const bool redo = on && (ONE || __ldcg(&P.cg_restart[w]) != 0);
        if (redo) accel(P.cg_corrr, corr, corr / r0);
        if (!sync()) return false;
        if (redo) {
          const float t = ADF_FMA(-reg, corr, divergence());
          wv = -(scale * t) + wv;
          now = finish(wv, act, z);
        }
        if (!sync()) return false;
      }
      act = now;
      fold_chunks(pairs);
      if (!sync()) return false;
      float beta = 0.0f;
      if constexpr (ONE) {
        double rz_new, sum;
        float mx;
        fold_world(P, c0, c1, rz_new, sum, mx);
        mx = maxr(mx, 0.0f);
        ++it;
        const int seen = __ldcg(&P.cg_act_new[0]);
        beta = (float)((!clamped && seen == acts && rz > 1.0e-30) ? rz_new / rz : 0.0);
        acts = seen;
        rz = rz_new;
        if (tid() == 0) record_test(P, 0, it, n_one, sum, mx, false);
        if (stop_test(P, 0, it, (float)(sum / (double)n_one), mx)) return true;
      } else {
        fold_worlds([&](int v, double rz_new, double sum, float mx) {
          const int2 r = P.wrange[v];
          const bool same = P.cg_restart[v] == 0 && P.cg_act_new[v] == 0;
          const double old = P.cg_rz[v];
          P.cg_step[v] = (same && old > 1.0e-30) ? rz_new / old : 0.0;
          P.cg_rz[v] = rz_new;
          if (record_test(P, v, P.iters[v] + 1, r.y - r.x, sum, maxr(mx, 0.0f), false)) atomicAdd(open_count(loop), 1);
        });
        if (!sync()) return false;
        if (__ldcg(open_count(loop)) == 0) return true;
        if (on) {
          on = __ldcg(&P.converged[w]) == 0;
          beta = (float)__ldcg(&P.cg_step[w]);
        }
      }
      if (on) {
        pd = act ? ADF_FMA(beta, pd, z) : 0.0f;
        pdr = pd / r0;
        P.cg_pdr[p] = pdr;
      }
      if (!sync()) return false;
    }
    return true;
  }

  // This thread's particle: blocks take even shares of the liquid in whole warps.
  __device__ __forceinline__ void place() {
    const int nf = P.nfw[0];
    const int share = ((nf + (int)gridDim.x - 1) / (int)gridDim.x + 31) & ~31;
    p = blockIdx.x * share + threadIdx.x;
    mine = (int)threadIdx.x < share && p < nf;
    if constexpr (ONE) {
      const int2 r = P.wrange[0];
      n_one = r.y - r.x;
      ib = P.skin_ws[0];
      ie = P.skin_ws[1];
      c0 = P.world_chunk_start[0];
      c1 = P.world_chunk_start[1];
    }
    if (mine) {
      w = ONE ? 0 : P.world_s[p];
      c = P.cnt[p];
      id = P.id_of[p];
      r0 = P.vel[p].w;
    }
  }

  // The world's part of a solve's start (k_begin_solve) and the cleared residuals; `it` the iterations done before.
  __device__ __forceinline__ void begin(int& it, bool& open) {
    div = P.mode == 0;
    dt = P.dt;
    scale = div ? dt : dt * dt;
    it = 0;
    if constexpr (ONE) {
      open = n_one > 0 && (A.init || P.converged[0] == 0);
      if (!A.init) it = P.iters[0];
      else if (tid() == 0) {
        P.iters[0] = 0;
        P.err_mean[0] = 0.0f;
        P.emax[0] = 0.0f;
      }
      if (P.iter_work && CG && open && tid() == 0) atomicAdd(P.iter_work, (unsigned long long)n_one);
    } else {
      for (int v = tid(); v < P.W; v += threads()) {
        const int2 r = P.wrange[v];
        bool go = r.y > r.x;
        if (A.init) {
          P.iters[v] = 0;
          P.err_mean[v] = 0.0f;
          P.emax[v] = 0.0f;
          P.converged[v] = go ? 0 : 1;
        } else {
          go = go && P.converged[v] == 0;
        }
        if (go) atomicAdd(open_count(1), 1);
        if (CG && go && P.iter_work) atomicAdd(P.iter_work, (unsigned long long)(r.y - r.x));
      }
    }
    if (CG)
      for (int i = tid(); i < P.n; i += threads()) P.cg_pair[i] = make_float2(0.0f, 0.0f);
    if (A.init)
      for (int i = tid(); i < P.n; i += threads()) P.err_orig[i] = 0.0f;
  }

  // The particle's part (solve_init_one), its row resident.
  __device__ __forceinline__ void start() {
    reg = P.reg[p];
    alpha = P.alpha[p];
    few = P.neff[p] < P.min_nb;
    if (A.init) {
      const float4 vi = P.vel[p];
      const float inv_r0 = 1.0f / r0;
      float rate = 0.0f;
      for_row<float4>([&](int j) { return P.vel[j]; },
                      [&](const float4& vj, const float4& g, float mj) {
                        const float aF = (mj * inv_r0) * g.w;
                        rate = ADF_FMA(aF, dotf(vi.x - vj.x, vi.y - vj.y, vi.z - vj.z, g.x, g.y, g.z), rate);
                      });
#pragma unroll
      for (int b = 0; b < NS; ++b)
        if (b < ns) {
          const float4 vb = P.slot_vb[slot_at(P, b, p)];
          rate = rate + dotf(vi.x - vb.x, vi.y - vb.y, vi.z - vb.z, gx[b], gy[b], gz[b]);
        }
      solve_start(P, p, vi, rate, kap, lower, src);
    } else {
      kap = P.kappa[p];
      lower = P.lower[p];
      src = P.src[p];
    }
  }

  // From the start on: the iterations, the velocity update and the statistics. False when a wait gave up.
  __device__ __forceinline__ bool solve(int it, bool open) {
    if (!sync()) return false;
    if constexpr (ONE) {
      on = mine && open;
    } else {
      open = __ldcg(open_count(1)) != 0;
      on = mine && __ldcg(&P.converged[w]) == 0;
    }
    if (open) {
      if constexpr (CG) {
        if (!cg(it)) return false;
      } else {
        if (!jacobi(it)) return false;
      }
    }
    if (CG && open) {  // the solved kappa / rho0 for the neighbours' acceleration
      if (mine) P.kr[p] = kap / r0;
      if (!sync()) return false;
    }
    if (mine) {
      P.kappa[p] = kap;
      apply_with<MS>(P, p, [&](float& x, float& y, float& z) { accel_of(P.kr, P.kappa[p], P.kr[p], x, y, z); });
    }
    for (int v = tid(); v < P.W; v += threads()) {
      A.iters_out[v] = P.iters[v];
      A.mean_out[v] = P.err_mean[v];
      if (A.max_out) A.max_out[v] = P.emax[v];
    }
    return true;
  }

  __device__ __forceinline__ void run() {
    int it;
    bool open;
    place();
    begin(it, open);
    if (mine) {
      load(P.pos[p]);
      start();
    }
    solve(it, open);
  }

  // The step from its rows and walls on: density, divergence solve, XSPH (velocities into D.vel, the density solve's),
  // density solve (parameters D and B), finish.
  __device__ __forceinline__ void run_step(const DevP& D, const SolveArgs& B) {
    int it;
    bool open;
    place();
    begin(it, open);
    if (mine) {
      load_density(P.pos[p]);
      start();
    }
    if (!solve(it, open)) return;
    if (!sync()) return;
    struct Other {
      float4 v;
      float ratio;
    };
    if (mine)
      xsph_with(P, p, [&](const float4& vi, float rho_i, float& cx, float& cy, float& cz) {
        for_row<Other>([&](int j) { return Other{P.vel[j], P.ratio[j]}; },
                       [&](const Other& o, const float4& g, float mj) {
                         xsph_term(vi, rho_i, o.v, o.ratio, mj, kernel_w(P.kc, dot_plain(g.x, g.y, g.z, g.x, g.y, g.z)), cx,
                                   cy, cz);
                       });
      });
    const int nf = P.nfw[0], all = nf + P.nfw[1];
    for (int q = nf + tid(); q < all; q += threads()) P.vel2[q] = P.vel[q];
    if (!sync()) return;
    SmallSolve d{D, B, sync, geo, jm};
    d.p = p;
    d.w = w;
    d.c = c;
    d.id = id;
    d.mine = mine;
    d.r0 = r0;
    d.ns = ns;
#pragma unroll
    for (int b = 0; b < NS; ++b) {
      d.gx[b] = gx[b];
      d.gy[b] = gy[b];
      d.gz[b] = gz[b];
    }
    d.c0 = c0;
    d.c1 = c1;
    d.ib = ib;
    d.ie = ie;
    d.n_one = n_one;
    d.begin(it, open);
    if (mine) d.start();
    if (!d.solve(it, open)) return;
    if (mine) finish_one<MS>(D, p, nf);
    for (int q = nf + tid(); q < all; q += threads()) finish_one<MS>(D, q, nf);
  }
};

// The solve when the liquid outgrew the blocks: particles that were no liquid at creation became liquid since. Out of
// line, so that the kernels below carry neither its code nor its registers.
template <bool MS, bool CG, bool ONE>
__device__ __noinline__ void outgrown_solve(const DevP& P, const SolveArgs& A) {
  GridSolve<MS, CG, ONE> g{P, A, GridSync{0u, gridDim.x + A.extra, A.ctr + CT_ARRIVE, A.status, A.wait_limit}};
  g.run();
}

template <bool MS, bool CG, bool ONE>
__global__ void __launch_bounds__(SMALL_BLOCK, 1)
k_small_solve(const __grid_constant__ DevP P, const __grid_constant__ SolveArgs A) {
  extern __shared__ float4 small_rows[];
  if (P.nfw[0] > (int)gridDim.x * SMALL_BLOCK) {
    outgrown_solve<MS, CG, ONE>(P, A);
    return;
  }
  SmallSolve<MS, CG, ONE> g{P, A, GridSync{0u, gridDim.x + A.extra, A.ctr + CT_ARRIVE, A.status, A.wait_limit}, small_rows,
                            reinterpret_cast<int2*>(small_rows + ROW_RES * SMALL_BLOCK)};
  g.run();
}

// Everything of a step after its neighbour rows and wall slots in one launch: the rows are read once for the density pass,
// both solves and XSPH, and the launches between them go. P and A are the divergence solve's, D and B the density solve's
// (D.vel is P.vel2); `between` are the counters of the barriers between the phases when the liquid outgrew the blocks.
template <bool MS, bool CG, bool ONE>
__global__ void __launch_bounds__(SMALL_BLOCK, 1)
k_small_step(const __grid_constant__ DevP P, const __grid_constant__ DevP D, const __grid_constant__ SolveArgs A,
             const __grid_constant__ SolveArgs B, int* between) {
  extern __shared__ float4 small_rows[];
  if (P.nfw[0] > (int)gridDim.x * SMALL_BLOCK) {
    constexpr int NBX = 4 | (MS ? MS_FLAG : 0);
    const int nf = P.nfw[0], all = nf + P.nfw[1], first = blockIdx.x * SMALL_BLOCK + threadIdx.x,
              step = gridDim.x * SMALL_BLOCK;
    GridSync sync{0u, gridDim.x + A.extra, between + CT_ARRIVE, A.status, A.wait_limit};
    for (int p = first; p < nf; p += step) density_one<NBX>(P, p);
    if (!sync()) return;
    outgrown_solve<MS, CG, ONE>(P, A);
    if (!sync()) return;
    for (int p = first; p < all; p += step) {
      if (p < nf) xsph_one<NBX>(P, p);
      else P.vel2[p] = P.vel[p];
    }
    if (!sync()) return;
    outgrown_solve<MS, CG, ONE>(D, B);
    if (!sync()) return;
    for (int p = first; p < all; p += step) finish_one<MS>(D, p, nf);
    return;
  }
  SmallSolve<MS, CG, ONE> g{P, A, GridSync{0u, gridDim.x + A.extra, A.ctr + CT_ARRIVE, A.status, A.wait_limit}, small_rows,
                            reinterpret_cast<int2*>(small_rows + ROW_RES * SMALL_BLOCK)};
  g.run_step(D, B);
}

}  // namespace adf
