// onecta.cu -- the per-trajectory propagation kernel for tables that fit the shared memory
// of one SM (H2): fixed-step RK4 in FP64, standard and AT-MQCT, with or without the
// coupled-states approximation (DOTRAJECT, MQCT_SOURCE_CODES/propagator.f:2283-4645, with
// DERIVS_BK and DERIVS_BK_adia, MQCT_SOURCE_CODES/mqct_eqtns.f:112-499, 720-879, and RK4,
// MQCT_SOURCE_CODES/suppl_routines.f:1076-1113).
//
// What bounds it: the chain of dependent steps of one right-hand side.  propagate_kernel
// (propagate.cu) takes 7.4 us for one of 165 states (1 749 matrix elements): its serial
// scalars, table reads from L2, interpolation, products and sums follow one another between
// eight block barriers, while the arithmetic is below half a microsecond.  Here
//   * the two knot rows of the trajectory's spline interval stay in shared memory (full
//     squares of the m-blocks: lo, hi - lo, lo'', hi'' per element), loaded again only when R
//     leaves the interval, every fifty right-hand sides or so;
//   * the products are formed with the four knot values, Z_q = K_q bt, before the spline
//     factors are known: y = Z_0 + bb Z_1 + c1 Z_2 + c2 Z_3 and M' bt = Z_1 / h + d1 Z_2 + d2 Z_3
//     per row (the difference hi - lo keeps the force free of cancellation);
//   * R and phi of a point depend on the momenta of the point before it, not on its force, so a
//     warp of its own sums the force of a right-hand side, completes the next point and
//     prepares the one after it (interval, factors) while the row warps work, and another
//     forms the phases of the next time; two barriers per right-hand side are left, of the
//     row warps after the stage input, of all after the products;
//   * AT mode needs neither force nor classical step: its path points are evaluated 32 at a
//     time, one per lane, from the path's splines.
// tpr threads of a warp share a row, with the rows of a warp adjacent: reads of K are
// conflict-free and the reads of bt broadcast.  Every sum has a fixed order.
// Measured on a B200 (tables of 165 states, 1 749 elements): 400 steps of 48 trajectories 8.0 ->
// 2.5 ms (1.6 us a right-hand side, of which the classical warp's chain and the rows' work, side by
// side, are 1.4), of 600 30.5 -> 12.4 ms; standard batches of 48 at 800 cm^-1 to the end 107 to 131
// -> 39 to 43 ms (the longest trajectory decides); AT 80 -> 20 ms with its set-up.
#include <algorithm>
#include <vector>

#include "propagate.cuh"

namespace mqct {

constexpr int OC_MAX_WARPS = 24;      // of a CTA: row warps, the classical and the phase warp
constexpr int OC_RING = 32;           // AT path points evaluated at a time

// Places in a CTA's dynamic shared memory (bytes).
struct OcSmem {
  int k01, k23, ain, bt, parts, ph, rg, ih, c5, ev, ring, total;
};

struct OcDev {
  OcSmem L;
  const mqct_traj_init_t* init;
  int n_traj, tpr, n_sq;
  const int* sq0;          // per block: first element of its square
  const int* sq_slot;      // per square element: slot of the knot rows
  int* queue;
  double* amp;
  double* cls;
  double* diag;
};

// The point of a right-hand side, published by the classical warp.
struct OcPoint {
  double bb, c1, c2, hinv, d1, d2, dphidt;
  double dt, h6;
  int key;                 // spline interval, or nR - 1 above the grid (the matrix is zero)
  int stage;               // 0..3 RK4 stages, 4 closing evaluation, 5 done
};

// The classical warp's state, alike in its lanes.  theta and P_theta do not change in
// DOTRAJECT's motion (their derivatives are zero), so their terms are constants of a
// trajectory.
struct OcCls {
  double R, PR, phi, Pphi;            // the state at the step's start
  double tR, tPR, tphi, tPphi;        // the point of the right-hand side being evaluated
  double kR, kphi, kPR, kPphi;        // first-stage derivatives
  double mR, mphi, mPR, mPphi;        // sums of the second and third stages
  double nR, nphi;                    // R and phi of the next point (or the step's end)
  double w, pre, ir;                  // dphi/dt per P_phi; dP_R/dt without the force; 1/R
  double th, Pth, sin_t, is2, h6;
  double tcur, eki, eqi, tmpR1, tmpR2;
  double ring_t, at_dt;               // AT: time at the ring's first step, the step's length
  int counter, status, vib, period, hint;
  int stage;                          // of the last point prepared
  int ring_w, at_step, path_hint, at_last;
};

static OcSmem oc_layout(int64_t n_sq, int N, int n_e, int nR) {
  OcSmem s{};
  int64_t o = 0;
  auto take = [&](int64_t bytes) {
    const int at = (int)o;
    o += (bytes + 15) & ~int64_t(15);
    return at;
  };
  s.k01 = take(n_sq * 16);
  s.k23 = take(n_sq * 16);
  s.ain = take((int64_t)N * 16);
  s.bt = take((int64_t)N * 16);
  s.parts = take((int64_t)N * 48);
  s.ph = take((int64_t)n_e * 32);
  s.rg = take((int64_t)nR * 8);
  s.ih = take((int64_t)nR * 8);
  s.c5 = take((int64_t)nR * 8);
  s.ev = take((int64_t)n_e * 8);
  s.ring = take((int64_t)sizeof(OcPoint) * OC_RING);
  s.total = (int)o;
  return s;
}

// The radial grid in shared memory, with 1/h and h^2/6 of each interval: the divisions would
// sit on the classical chain.
struct OcGrid {
  const double *R, *ih, *c5;
  int n;
};

// Spline interval and factors at x (as spline_at).  *hint: the interval found last (0-based).
__device__ inline void oc_point(OcPoint& p, const OcGrid& g, double x, int* hint) {
  int k = *hint;
  if (!(k >= 0 && k + 1 < g.n && g.R[k] <= x && x < g.R[k + 1])) {
    int lo = 0, hi = g.n - 1;
    while (hi - lo > 1) {
      const int m = (hi + lo) >> 1;
      if (g.R[m] > x) hi = m;
      else lo = m;
    }
    k = lo;
    *hint = k;
  }
  const double ih = g.ih[k], c5 = g.c5[k], c6 = c5 * ih;
  const double aa = (g.R[k + 1] - x) * ih, bb = (x - g.R[k]) * ih;
  p.bb = bb;
  p.c1 = (aa * aa * aa - aa) * c5;
  p.c2 = (bb * bb * bb - bb) * c5;
  p.hinv = ih;
  p.d1 = -(3 * aa * aa - 1.0) * c6;
  p.d2 = (3 * bb * bb - 1.0) * c6;
  p.key = x > g.R[g.n - 1] ? g.n - 1 : k;
}

// Value at time t of column col (splined: y2 column yc) of an AT path whose interval
// [klo, klo + 1] (0-based) holds t (splint, MQCT_SOURCE_CODES/suppl_routines.f:968-1002).
__device__ inline double oc_path(const double* rec, const double* y2, int klo, int col, int yc,
                                 double t) {
  const double xlo = rec[8 * klo], xhi = rec[8 * (klo + 1)];
  const double h = xhi - xlo, a = (xhi - t) / h, b = (t - xlo) / h;
  return a * rec[8 * klo + col] + b * rec[8 * (klo + 1) + col] +
         ((a * a * a - a) * y2[kAtCols * klo + yc] + (b * b * b - b) * y2[kAtCols * (klo + 1) + yc]) *
             (h * h) / 6.0;
}

// AT: point idx (two per step) of the path -> S, from the ring of points that the warp fills
// a window at a time, each lane stepping the time to its own point as the run does.
__device__ __forceinline__ void oc_publish_at(OcCls& c, OcPoint& S, OcPoint* ring,
                                              const PropDev& d, const OcGrid& grid,
                                              const double* rec, const double* y2p, int n_rec,
                                              double t_end, double dt0, int idx) {
  const int lane = threadIdx.x & 31;
  if (idx / OC_RING != c.ring_w) {
    double t = c.ring_t;
    const int w = c.ring_w + 1, w0 = w * OC_RING, mine = w0 + lane;
    if (w > 0)
      for (int q = 0; q < OC_RING / 2; ++q) t += t + dt0 >= t_end ? t_end - t : dt0;
    c.ring_t = t;
    c.ring_w = w;
    double tm = t;
    for (int q = w0 / 2;; ++q) {
      double dt = dt0;
      const bool last = t + dt >= t_end;
      if (last) dt = t_end - t;
      if (mine < 2 * q + 2) {
        tm = t + (mine & 1 ? dt * 0.5 : 0.0);
        break;
      }
      t += dt;
      tm = t;
      if (last) break;
    }
    int klo = c.path_hint, khi = n_rec - 1;            // rec[klo] <= tm from the last window on
    while (khi - klo > 1) {
      const int k = (khi + klo) >> 1;
      if (rec[8 * k] > tm) khi = k;
      else klo = k;
    }
    const double R = oc_path(rec, y2p, klo, 1, 0, tm), th = oc_path(rec, y2p, klo, 3, 1, tm),
                 Pphi = oc_path(rec, y2p, klo, 6, 3, tm);
    const double sn = sin(th), ir = 1.0 / R;
    OcPoint q;
    int h = -1;
    oc_point(q, grid, R, &h);
    q.dphidt = Pphi * ir * ir * d.inv_mass * (1.0 / (sn * sn));
    __syncwarp();
    ring[lane] = q;
    __syncwarp();
    c.path_hint = __shfl_sync(0xffffffffu, klo, 0);
  }
  if (lane == 0) {
    OcPoint q = ring[idx % OC_RING];
    q.dt = c.at_dt;
    q.h6 = c.at_dt / 6.0;
    q.stage = c.stage;
    S = q;
  }
}

// From a complete point (its P_R, P_phi and dphi/dt; not its force): R and phi of the next one,
// at the end of a step the stop rules (MQCT_SOURCE_CODES/propagator.f:4011-4050), and the next
// point's factors but dphi/dt -> S.
__device__ __forceinline__ void oc_before(OcCls& c, OcPoint& S, double dphidt, const PropDev& d,
                                 const mqct_traj_init_t& ti, const OcGrid& grid) {
  const double dt = ti.dt, hh = dt * 0.5, im = d.inv_mass;
  const bool lead = (threadIdx.x & 31) == 0;
  if (c.stage >= 4) {
    c.stage = 5;
    if (lead) S.stage = 5;
    return;
  }
  const double dR = c.tPR * im, ir3m = c.ir * c.ir * c.ir * im;
  c.pre = c.Pth * c.Pth * ir3m + c.tPphi * c.tPphi * ir3m * c.is2;
  const int s = c.stage;
  double R, phi;
  if (s == 0) {
    c.kR = dR;
    c.kphi = dphidt;
    R = c.R + hh * dR;
    phi = c.phi + hh * dphidt;
    c.stage = 1;
  } else if (s == 1) {
    c.mR = dR;
    c.mphi = dphidt;
    R = c.R + hh * dR;
    phi = c.phi + hh * dphidt;
    c.stage = 2;
  } else if (s == 2) {
    c.mR += dR;
    c.mphi += dphidt;
    R = c.R + dt * dR;
    phi = c.phi + dt * dphidt;
    c.stage = 3;
  } else {
    R = c.R + c.h6 * (c.kR + dR + 2.0 * c.mR);
    phi = c.phi + c.h6 * (c.kphi + dphidt + 2.0 * c.mphi);
    c.R = R;
    c.phi = phi;
    c.tcur += dt;
    bool run = true;
    if (c.tcur - dt > dt && c.counter > 2) {
      if ((c.tmpR2 - c.tmpR1) < 0.0 && (c.tmpR1 - R) > 0.0) c.vib += 1;
    }
    c.tmpR2 = c.tmpR1;
    c.tmpR1 = R;
    c.period = fabs(phi) < 6.28 ? 0 : (int)(fabs(phi) / 2.0 / kPi);
    if (ti.numb_orb_prds <= c.period) run = false;
    if (c.vib >= ti.numb_oscl_prds) run = false;
    if (ti.time_lim > 0 && c.tcur >= ti.time_lim) run = false;
    if (R > ti.r_fin) run = false;
    if (!(R == R)) {
      run = false;
      c.status = 3;
    }
    if (run && ti.max_steps > 0 && c.counter >= ti.max_steps) {
      run = false;
      c.status = 1;
    }
    if (run) c.counter += 1;
    c.stage = run ? 0 : 4;
  }
  c.tR = R;
  c.tphi = phi;
  const double ir = 1.0 / R;
  c.ir = ir;
  c.w = ir * ir * im * c.is2;
  OcPoint q;
  oc_point(q, grid, R, &c.hint);
  q.dt = dt;
  q.h6 = c.h6;
  q.stage = c.stage;
  q.dphidt = 0.0;
  if (lead) S = q;
}

// With the sums of a right-hand side of stage s: P_R and P_phi of the point that oc_before has
// prepared; returns its dphi/dt.
__device__ __forceinline__ double oc_after(OcCls& c, int s, double dt, double F, double g) {
  const double dPR = -F + c.pre, dPphi = c.sin_t * g, hh = dt * 0.5;
  if (s == 0) {
    c.kPR = dPR;
    c.kPphi = dPphi;
    c.tPR = c.PR + hh * dPR;
    c.tPphi = c.Pphi + hh * dPphi;
  } else if (s == 1) {
    c.mPR = dPR;
    c.mPphi = dPphi;
    c.tPR = c.PR + hh * dPR;
    c.tPphi = c.Pphi + hh * dPphi;
  } else if (s == 2) {
    c.mPR += dPR;
    c.mPphi += dPphi;
    c.tPR = c.PR + dt * dPR;
    c.tPphi = c.Pphi + dt * dPphi;
  } else {
    c.PR += c.h6 * (c.kPR + dPR + 2.0 * c.mPR);
    c.Pphi += c.h6 * (c.kPphi + dPphi + 2.0 * c.mPphi);
    c.tPR = c.PR;
    c.tPphi = c.Pphi;
  }
  return c.tPphi * c.w;
}

// AT: the step's stage and time advance.
__device__ __forceinline__ void oc_advance_at(OcCls& c, int64_t max_steps, double dt0,
                                              double t_end) {
  if (c.stage == 3) {
    c.tcur += c.at_dt;
    c.at_step += 1;
    bool run = !c.at_last;
    if (run && max_steps > 0 && c.counter >= max_steps) {
      run = false;
      c.status = 1;
    }
    c.stage = run ? 0 : 5;
    if (run) {
      c.counter += 1;
      c.at_last = c.tcur + dt0 >= t_end;
      c.at_dt = c.at_last ? t_end - c.tcur : dt0;
    }
  } else {
    c.stage += 1;
  }
}

// Barrier `id` of n threads (the roles meet at it from different places in the code).
__device__ __forceinline__ void oc_bar(int id, int n) {
  asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// What the roles of a CTA share.  S: the points of this right-hand side and the next two.
struct OcShared {
  OcPoint S[3];
  mqct_traj_init_t ti;
  double t0, t_end;        // AT: the path's first and last times
  int tr, skip;
};
// The trajectory's states: all, or the initial m-block's (coupled states).
struct OcRows {
  int s_int, lo, n, sq_lo;
};

// The row warps of one trajectory: tpr threads per row, rows of a warp adjacent.
template <bool at>
__device__ __forceinline__ void oc_rows(const PropDev& d, const OcDev& D, unsigned char* sm,
                                        OcShared& sh, const OcRows& rw, int n_threads, int& key) {
  double2* ain = reinterpret_cast<double2*>(sm + D.L.ain);
  double2* bt = reinterpret_cast<double2*>(sm + D.L.bt);
  double* parts = reinterpret_cast<double*>(sm + D.L.parts);   // F, g, pot: N each
  const double2* ph = reinterpret_cast<const double2*>(sm + D.L.ph);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, N = d.N, nR = d.nR;
  const int rpw = 32 / D.tpr, sub = lane / rpw;
  const int ri = warp * rpw + (lane - sub * rpw);
  const bool live = ri < rw.n;                    // the lane works on a row
  const bool own = live && sub == 0;              // and keeps its state
  const int row = live ? rw.lo + ri : rw.lo;
  int n = 0, b0 = 0, sq = 0, ec = 0, nbp = -1, nbm = -1;
  double cp = 0.0, cm = 0.0;
  if (live) {
    const int b = d.st_blk[row];
    n = d.blk_n[b];
    b0 = d.blk_s0[b];
    sq = D.sq0[b] + (row - b0);
    ec = d.st_e[row];
    if (own && !d.cs) {
      nbp = d.nb_plus[row];
      nbm = d.nb_minus[row];
      cp = d.cplus[row];
      cm = d.cminus[row];
    }
  }
  double2 y = make_double2(row == rw.s_int && own ? 1.0 : 0.0, 0.0), k1{0.0, 0.0}, k23{0.0, 0.0};
  double2 p = make_double2(1.0, 0.0);             // e^{-iEt} of the row's class
  oc_bar(1, n_threads);                           // the start: points and phases
  if (sh.skip) return;
  if (own) {
    p = ph[ec];
    ain[row] = y;
    bt[row] = make_double2(p.x * y.x - p.y * y.y, p.x * y.y + p.y * y.x);
  }
  const int n_row_threads = n_threads - 64;
  int cur = 0, buf = 0;                           // this right-hand side's point and parts
  oc_bar(2, n_row_threads);                       // (A) of the first right-hand side
  for (;;) {
    if (sh.S[cur].stage == 5) break;
    if (sh.S[cur].key != key) {
      key = sh.S[cur].key;
      if (key < nR - 1) {  // another interval: its knot rows
        const double2* lo = reinterpret_cast<const double2*>(d.knots) + (int64_t)key * d.S;
        const double2* hi = lo + d.S;
        double2* K01 = reinterpret_cast<double2*>(sm + D.L.k01);
        double2* K23 = reinterpret_cast<double2*>(sm + D.L.k23);
        const int sq_n = d.cs ? rw.n * rw.n : D.n_sq;
        for (int e = threadIdx.x; e < sq_n; e += n_row_threads) {
          const int k = D.sq_slot[rw.sq_lo + e];
          const double2 a = __ldg(lo + k), b = __ldg(hi + k);
          K01[e] = make_double2(a.x, b.x - a.x);
          K23[e] = make_double2(a.y, b.y);
        }
        oc_bar(2, n_row_threads);
      }
    }
    double z[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) z[q] = 0.0;
    double2 u = make_double2(0.0, 0.0);
    if (key < nR - 1) {
      const double2* zb = bt + b0;
      auto add = [&](const double2& a, const double2& b, const double2& v) {
        z[0] = fma(a.x, v.x, z[0]);
        z[1] = fma(a.x, v.y, z[1]);
        z[2] = fma(a.y, v.x, z[2]);
        z[3] = fma(a.y, v.y, z[3]);
        z[4] = fma(b.x, v.x, z[4]);
        z[5] = fma(b.x, v.y, z[5]);
        z[6] = fma(b.y, v.x, z[6]);
        z[7] = fma(b.y, v.y, z[7]);
      };
      const double2* k23 = reinterpret_cast<const double2*>(sm + D.L.k23) + sq - rw.sq_lo;
      const double2* k01 = reinterpret_cast<const double2*>(sm + D.L.k01) + sq - rw.sq_lo;
#pragma unroll 4
      for (int j = sub; j < n; j += D.tpr) add(k01[j * n], k23[j * n], zb[j]);
      for (int o = rpw; o < 32; o <<= 1)
#pragma unroll
        for (int q = 0; q < 8; ++q) z[q] += __shfl_xor_sync(0xffffffffu, z[q], o);
    }
    // u = (J_+ + J_-) a (MQCT_SOURCE_CODES/mqct_eqtns.f:447-464)
    if (nbp >= 0) {
      const double2 a = ain[nbp];
      u.x += cp * a.x;
      u.y += cp * a.y;
    }
    if (nbm >= 0) {
      const double2 a = ain[nbm];
      u.x += cm * a.x;
      u.y += cm * a.y;
    }
    // y and M' bt with the point's factors (known since the last barrier), the row's parts of
    // F, g and pot
    const OcPoint& q = sh.S[cur];
    const int stage = q.stage;
    double yr = 0.0, yi = 0.0;
    if (own) {
      const double2 b2 = bt[row];
      double* pt = parts + 3 * N * buf;
      if (key < nR - 1) {
        yr = z[0] + q.bb * z[2] + q.c1 * z[4] + q.c2 * z[6];
        yi = z[1] + q.bb * z[3] + q.c1 * z[5] + q.c2 * z[7];
      }
      if (stage == 4) {
        const double w2 = y.x * y.x + y.y * y.y;
        pt[ri] = w2 * reinterpret_cast<const double*>(sm + D.L.ev)[ec];
        pt[N + ri] = w2;
        pt[2 * N + ri] = b2.x * yr + b2.y * yi;
      } else if (!at) {
        double dr = 0.0, di = 0.0;
        if (key < nR - 1) {
          dr = q.hinv * z[2] + q.d1 * z[4] + q.d2 * z[6];
          di = q.hinv * z[3] + q.d1 * z[5] + q.d2 * z[7];
        }
        const double utr = p.x * u.x - p.y * u.y, uti = p.x * u.y + p.y * u.x;
        pt[ri] = b2.x * dr + b2.y * di;           // Re(bt^+ M' bt)
        pt[N + ri] = utr * yi - uti * yr;         // Im((D^* u)^+ y)
        pt[2 * N + ri] = b2.x * yr + b2.y * yi;   // Re(bt^+ y)
      }
    }
    oc_bar(1, n_threads);                         // (B) parts, dphi/dt and phases are ready
    if (own && stage != 4) {
      // da = -i e^{iEt} y - i (dphi/2) u, and the RK4 stage of the row
      const double hd = 0.5 * q.dphidt, dt = q.dt;
      const double cr = p.x * yr + p.y * yi + hd * u.x;
      const double ci = p.x * yi - p.y * yr + hd * u.y;
      const double2 k = make_double2(ci, -cr);
      double2 a;
      if (stage == 0) {
        k1 = k;
        a = make_double2(y.x + dt * 0.5 * k.x, y.y + dt * 0.5 * k.y);
        p = ph[d.n_e + ec];                       // t + dt/2: buffer 1
      } else if (stage == 1) {
        k23 = k;
        a = make_double2(y.x + dt * 0.5 * k.x, y.y + dt * 0.5 * k.y);
      } else if (stage == 2) {
        k23 = make_double2(k23.x + k.x, k23.y + k.y);
        a = make_double2(y.x + dt * k.x, y.y + dt * k.y);
        p = ph[ec];                               // t + dt: buffer 0
      } else {
        const double h6 = q.h6;
        y = make_double2(y.x + h6 * (k1.x + k.x + 2.0 * k23.x), y.y + h6 * (k1.y + k.y + 2.0 * k23.y));
        a = y;
      }
      ain[row] = a;
      bt[row] = make_double2(p.x * a.x - p.y * a.y, p.x * a.y + p.y * a.x);
    }
    cur = cur == 2 ? 0 : cur + 1;
    buf ^= 1;
    oc_bar(2, n_row_threads);                     // (A) the stage input of every row is ready
  }
  if (own) {
    double* amp = D.amp + (size_t)sh.tr * 2 * N;
    const int o = d.perm[row];
    amp[o] = y.x;
    amp[N + o] = y.y;
    if (at) parts[ri] = y.x * y.x + y.y * y.y;
  }
  if (at) oc_bar(1, n_threads);                   // the norm's parts
}

// Sum of the rows' parts by the classical warp (fixed order), in every lane.
__device__ __forceinline__ double oc_sum(const double* v, int n) {
  const int lane = threadIdx.x & 31;
  double x = 0.0;
  for (int i = lane; i < n; i += 32) x += v[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
// F and g together: half a warp sums each, four chains a lane.
__device__ __forceinline__ void oc_sum2(const double* v, int N, int n, double& F, double& g) {
  const int lane = threadIdx.x & 31;
  const double* w = v + (lane >> 4) * N;
  double x[4] = {0.0, 0.0, 0.0, 0.0};
  int i = lane & 15;
  for (; i + 48 < n; i += 64) {
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] += w[i + 16 * q];
  }
#pragma unroll
  for (int q = 0; q < 3; ++q)
    if (i + 16 * q < n) x[q] += w[i + 16 * q];
  double s = (x[0] + x[1]) + (x[2] + x[3]);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  F = __shfl_sync(0xffffffffu, s, 0);
  g = __shfl_sync(0xffffffffu, s, 16);
}

// The classical warp of one trajectory.  From barrier (B) of a right-hand side to the next it
// sums that right-hand side's parts, completes the next point (P_R, P_phi, dphi/dt) and
// prepares the one after it (R, interval, factors), so that its whole chain runs beside the
// rows' work.  AT: the path point after the next.
template <bool at>
__device__ __forceinline__ void oc_classical(const PropDev& d, const OcDev& D, unsigned char* sm,
                                             OcShared& sh, const OcRows& rw, int n_threads,
                                             const OcGrid& grid) {
  const double* parts = reinterpret_cast<const double*>(sm + D.L.parts);
  const double* ev = reinterpret_cast<const double*>(sm + D.L.ev);
  OcPoint* ring = reinterpret_cast<OcPoint*>(sm + D.L.ring);
  const int lane = threadIdx.x & 31, tr = sh.tr, N = d.N;
  const double* rec = at ? d.at_rec + 8 * d.at_off[tr] : nullptr;
  const double* y2p = at ? d.at_y2 + kAtCols * d.at_off[tr] : nullptr;
  const int n_rec = at ? d.at_n[tr] : 0;
  const double t_end = sh.t_end, dt = sh.ti.dt;
  // the start: the first two points
  OcCls c{};
  c.tcur = c.ring_t = sh.t0;
  c.ring_w = c.hint = -1;
  c.counter = 1;
  c.h6 = dt / 6.0;
  bool skip = false;
  if (at) {
    c.at_last = sh.t0 + dt >= t_end;
    c.at_dt = c.at_last ? t_end - sh.t0 : dt;
    oc_publish_at(c, sh.S[0], ring, d, grid, rec, y2p, n_rec, t_end, dt, 0);
    c.stage = 1;
    oc_publish_at(c, sh.S[1], ring, d, grid, rec, y2p, n_rec, t_end, dt, 1);
  } else {
    const double k_vec = sqrt(d.mass * 2.0 * sh.ti.e_coll);
    const double l_orb = sqrt(sh.ti.l_real * (sh.ti.l_real + 1.0));
    c.R = sh.ti.r_start;
    skip = l_orb / k_vec > sh.ti.r_start;  // impact parameter beyond the start
    if (!skip) {  // initial conditions, MQCT_SOURCE_CODES/propagator.f:2531-2566
      c.PR = -sqrt(k_vec * k_vec - l_orb * l_orb / (sh.ti.r_start * sh.ti.r_start));
      c.th = acos(0.0);
      c.Pth = l_orb * sin(0.0);
      c.Pphi = l_orb * cos(0.0);
      c.sin_t = sin(c.th);
      c.is2 = 1.0 / (c.sin_t * c.sin_t);
      c.tR = c.R;
      c.tPR = c.PR;
      c.tPphi = c.Pphi;
      c.eki = kinetic(Cls{c.R, c.PR, c.th, c.Pth, 0.0, c.Pphi}, d.mass);
      c.ir = 1.0 / c.R;
      c.w = c.ir * c.ir * d.inv_mass * c.is2;
      OcPoint q;
      oc_point(q, grid, c.R, &c.hint);
      q.dphidt = c.Pphi * c.w;
      q.dt = dt;
      q.h6 = c.h6;
      q.stage = 0;
      if (lane == 0) sh.S[0] = q;
      oc_before(c, sh.S[1], q.dphidt, d, sh.ti, grid);
    }
  }
  if (lane == 0) sh.skip = skip ? 1 : 0;
  __syncwarp();
  oc_bar(1, n_threads);               // the start
  if (skip) return;
  int nx = 1, buf = 0;                // the next point's place, this right-hand side's parts
  int stage = 0, next = c.stage;      // stages of this right-hand side and the next
  bool init = true;
  double eq = 0.0, nrm = 0.0, pot = 0.0;
  while (stage != 5) {
    oc_bar(1, n_threads);             // (B)
    const int nn = nx == 2 ? 0 : nx + 1;
    if (at) {
      if (next != 5) {
        oc_advance_at(c, sh.ti.max_steps, dt, t_end);
        if (c.stage == 5) {
          if (lane == 0) sh.S[nn].stage = 5;
        } else {
          oc_publish_at(c, sh.S[nn], ring, d, grid, rec, y2p, n_rec, t_end, dt,
                        2 * c.at_step + (c.stage == 0 ? 0 : c.stage == 3 ? 2 : 1));
        }
      }
    } else if (stage == 4) {
      // the closing evaluation's parts: quantum energy, norm, coupling energy
      const double* pt = parts + 3 * N * buf;
      eq = oc_sum(pt, rw.n);
      nrm = oc_sum(pt + N, rw.n);
      pot = oc_sum(pt + 2 * N, rw.n);
    } else {
      const double* pt = parts + 3 * N * buf;
      double F, g;
      oc_sum2(pt, N, rw.n, F, g);
      if (init) c.eqi = ev[d.st_e[rw.s_int]] + oc_sum(pt + 2 * N, rw.n);  // propagator.f:2695-2810
      init = false;
      const double dphidt = oc_after(c, stage, dt, F, g);
      if (lane == 0) sh.S[nx].dphidt = dphidt;
      oc_before(c, sh.S[nn], dphidt, d, sh.ti, grid);
    }
    __syncwarp();
    stage = next;
    next = c.stage;
    nx = nn;
    buf ^= 1;
  }
  if (at) {
    oc_bar(1, n_threads);             // the norm's parts
    nrm = oc_sum(parts, rw.n);
  }
  if (lane == 0) {                    // MQCT_SOURCE_CODES/propagator.f:4182-4343
    double* cl = D.cls + (size_t)tr * 6;
    cl[0] = at ? 0.0 : c.R;
    cl[1] = c.PR;
    cl[2] = c.th;
    cl[3] = c.Pth;
    cl[4] = c.phi;
    cl[5] = c.Pphi;
    double* dg = D.diag + (size_t)tr * 8;
    dg[0] = c.tcur;
    dg[1] = (double)c.counter;
    dg[2] = fabs(1.0 - nrm);
    dg[3] = at ? 0.0
               : fabs(eq + kinetic(Cls{c.R, c.PR, c.th, c.Pth, c.phi, c.Pphi}, d.mass) + pot -
                      c.eki - c.eqi);
    dg[4] = c.status;
    dg[5] = c.period;
    dg[6] = c.vib;
    dg[7] = pot;
  }
}

// The phase warp of one trajectory: the phases of the next new time, t + dt/2 in stage 0 (into
// buffer 1), t + dt in stage 2 (into buffer 0), before barrier (B).
template <bool at>
__device__ __forceinline__ void oc_phases(const PropDev& d, const OcDev& D, unsigned char* sm,
                                          OcShared& sh, int n_threads) {
  double2* ph = reinterpret_cast<double2*>(sm + D.L.ph);
  const double* ev = reinterpret_cast<const double*>(sm + D.L.ev);
  const int lane = threadIdx.x & 31;
  double t = sh.t0;
  int cur = 0;
  oc_bar(1, n_threads);               // the start
  if (sh.skip) return;
  for (;;) {
    const int stage = sh.S[cur].stage;
    if (stage == 5) break;
    double dt = sh.ti.dt;
    if (at && t + dt >= sh.t_end) dt = sh.t_end - t;
    if (stage == 0 || stage == 2) {
      double2* o = ph + (stage == 0 ? d.n_e : 0);
      const double tn = t + (stage == 0 ? dt * 0.5 : dt);
      for (int e = lane; e < d.n_e; e += 32) {
        double sn, co;
        sincos(ev[e] * tn, &sn, &co);
        o[e] = make_double2(co, -sn);
      }
    }
    if (stage == 3) t += dt;
    __syncwarp();
    oc_bar(1, n_threads);             // (B)
    cur = cur == 2 ? 0 : cur + 1;
  }
  if (at) oc_bar(1, n_threads);
}

// T: threads of a CTA at most (144 registers a thread with 448, 80 with 768).
template <bool at, int T>
__global__ void __launch_bounds__(T, 1) oc_kernel(PropDev d, OcDev D) {
  extern __shared__ __align__(16) unsigned char oc_sm[];
  __shared__ OcShared sh;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_threads = blockDim.x, row_warps = n_threads / 32 - 2;
  const int N = d.N;
  double2* ph = reinterpret_cast<double2*>(oc_sm + D.L.ph);
  double* ev = reinterpret_cast<double*>(oc_sm + D.L.ev);
  double* Rg = reinterpret_cast<double*>(oc_sm + D.L.rg);
  double* Rih = reinterpret_cast<double*>(oc_sm + D.L.ih);
  double* Rc5 = reinterpret_cast<double*>(oc_sm + D.L.c5);
  const OcGrid grid{Rg, Rih, Rc5, d.nR};
  for (int i = tid; i < d.nR; i += n_threads) {
    const double x = d.R[i], h = i + 1 < d.nR ? d.R[i + 1] - x : 1.0;
    Rg[i] = x;
    Rih[i] = 1.0 / h;
    Rc5[i] = (h * h) / 6.0;
  }
  for (int e = tid; e < d.n_e; e += n_threads) ev[e] = d.e_val[e];
  int key = -1, key_blk = -1;   // the interval (and, coupled states, the m-block) in K
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      const int t = atomicAdd(D.queue, 1);
      sh.tr = t;
      if (t < D.n_traj) {
        sh.ti = D.init[t];
        sh.t0 = sh.t_end = 0.0;
        if (at) {
          sh.t0 = d.at_rec[8 * d.at_off[t]];
          sh.t_end = d.at_rec[8 * (d.at_off[t] + d.at_n[t] - 1)];
        }
      }
    }
    __syncthreads();
    const int tr = sh.tr;
    if (tr >= D.n_traj) break;
    OcRows rw;
    rw.s_int = d.inv_perm[sh.ti.s_st - 1];
    const int blk = d.cs ? d.st_blk[rw.s_int] : -1;
    rw.lo = blk >= 0 ? d.blk_s0[blk] : 0;
    rw.n = blk >= 0 ? d.blk_n[blk] : N;
    rw.sq_lo = blk >= 0 ? D.sq0[blk] : 0;
    if (blk != key_blk) {
      key = -1;
      key_blk = blk;
    }
    // the initial time's phases (buffer 0)
    for (int e = tid; e < d.n_e; e += n_threads) {
      double sn, co;
      sincos(ev[e] * sh.t0, &sn, &co);
      ph[e] = make_double2(co, -sn);
    }
    if (warp < row_warps) oc_rows<at>(d, D, oc_sm, sh, rw, n_threads, key);
    else if (warp == row_warps) oc_classical<at>(d, D, oc_sm, sh, rw, n_threads, grid);
    else oc_phases<at>(d, D, oc_sm, sh, n_threads);
    // states outside the coupled states' block keep zero amplitude; a trajectory that is not
    // propagated returns its initial unit vector
    const bool skip = sh.skip != 0;
    double* amp = D.amp + (size_t)tr * 2 * N;
    for (int i = tid; i < N; i += n_threads)
      if (skip || i < rw.lo || i >= rw.lo + rw.n) {
        amp[d.perm[i]] = skip && i == rw.s_int ? 1.0 : 0.0;
        amp[N + d.perm[i]] = 0.0;
      }
    if (skip && tid == 0) {
      double* cl = D.cls + (size_t)tr * 6;
      cl[0] = sh.ti.r_start;
      cl[1] = cl[2] = cl[3] = cl[4] = cl[5] = 0.0;
      double* dg = D.diag + (size_t)tr * 8;
      dg[0] = dg[1] = dg[2] = dg[3] = dg[5] = dg[6] = dg[7] = 0.0;
      dg[4] = 2.0;
    }
  }
}

// ---------------------------------------------------------------- host
struct OcEngine {
  DevBuf<int> sq0, sq_slot, queue;
  int n_sq = 0, n_max = 0;
  size_t smem = 0;
  OcSmem L{};
  bool ready = false, ok = false;
};

OcEngine* oc_create() { return new OcEngine(); }
void oc_destroy(OcEngine* e) { delete e; }

constexpr int OC_T1 = 448;

static const void* oc_fn(bool at, bool wide) {
  return at ? (wide ? (const void*)oc_kernel<true, 32 * OC_MAX_WARPS>
                    : (const void*)oc_kernel<true, OC_T1>)
            : (wide ? (const void*)oc_kernel<false, 32 * OC_MAX_WARPS>
                    : (const void*)oc_kernel<false, OC_T1>);
}

// Lays the tables out once and reports whether they fit: the squares of the m-blocks, 32 B an
// element, in one SM's shared memory, and at most 704 rows.
bool oc_usable(OcEngine* e, const PropDev& d, const std::vector<int>& blk_n,
               const std::vector<int>& blk_s0, const std::vector<int64_t>& blk_slot0,
               cudaStream_t st) {
  if (e->ready) return e->ok;
  e->ready = true;
  int64_t n_sq = 0;
  for (int n : blk_n) {
    n_sq += (int64_t)n * n;
    e->n_max = std::max(e->n_max, n);
  }
  int dev = 0, optin = 0;
  cudaFuncAttributes fa{};
  if (d.N > 32 * (OC_MAX_WARPS - 2) || n_sq > (1 << 20) || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess )
    return false;
  e->L = oc_layout(n_sq, d.N, d.n_e, d.nR);
  e->smem = (size_t)e->L.total;
  for (int f = 0; f < 4; ++f)
    if (cudaFuncGetAttributes(&fa, oc_fn(f & 1, f & 2)) != cudaSuccess ||
        e->smem + fa.sharedSizeBytes > (size_t)optin ||
        cudaFuncSetAttribute(oc_fn(f & 1, f & 2), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin - (int)fa.sharedSizeBytes) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  std::vector<int> sq0, slot;
  for (size_t b = 0; b < blk_n.size(); ++b) {
    sq0.push_back((int)slot.size());
    const int n = blk_n[b];
    for (int j = 0; j < n; ++j)
      for (int i = 0; i < n; ++i) {
        const int hi = std::max(i, j), lo = std::min(i, j);
        slot.push_back((int)(blk_slot0[b] + (int64_t)hi * (hi + 1) / 2 + lo));
      }
  }
  e->n_sq = (int)n_sq;
  if (e->sq0.upload(sq0, st) != cudaSuccess || e->sq_slot.upload(slot, st) != cudaSuccess ||
      e->queue.alloc(1) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  e->ok = true;
  return true;
}

int oc_run(OcEngine* e, const PropDev& d, int n_sm, cudaStream_t st, cudaEvent_t ev0,
           cudaEvent_t ev1, const mqct_traj_init_t* d_init, int n_traj, double* amp, double* cls,
           double* diag) {
  // One thread per row, two for a coupled-states block, whose few rows leave the SM idle: 400
  // steps of 48 trajectories, tables of 165 states (blocks of up to 25), 2.53 ms with one, 2.60
  // with two; coupled states 1.89 and 1.55; 600 trajectories 12.4 / 12.8 and 9.2 / 7.6.  The
  // 80-register form costs a tenth to a fifth (2.79, 1.86), so only CTAs of more threads take it.
  const int rows = d.cs ? e->n_max : d.N;
  const int tpr = d.cs && 2 * rows <= OC_T1 - 64 ? 2 : 1;
  const int threads = 32 * ((rows * tpr + 31) / 32 + 2);
  const bool wide = threads > OC_T1;
  OcDev D{};
  D.L = e->L;
  D.init = d_init;
  D.n_traj = n_traj;
  D.tpr = tpr;
  D.n_sq = e->n_sq;
  D.sq0 = e->sq0.p;
  D.sq_slot = e->sq_slot.p;
  D.queue = e->queue.p;
  D.amp = amp;
  D.cls = cls;
  D.diag = diag;
  int per_sm = 1;
  const void* fn = oc_fn(d.mode == MQCT_MODE_AT, wide);
  MQCT_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, e->smem));
  const unsigned grid = (unsigned)std::min<int64_t>(n_traj, (int64_t)n_sm * std::max(1, per_sm));
  PropDev dv = d;
  void* args[] = {&dv, &D};
  MQCT_CUDA_TRY(cudaMemsetAsync(e->queue.p, 0, sizeof(int), st));
  MQCT_CUDA_TRY(cudaEventRecord(ev0, st));
  MQCT_CUDA_TRY(cudaLaunchKernel(fn, dim3(grid), dim3(threads), args, e->smem, st));
  MQCT_CUDA_TRY(cudaEventRecord(ev1, st));
  return MQCT_OK;
}

}  // namespace mqct
