// VortexArraysSystemPtr neighbour passes (plain FP64), the reference's second
// model (DynamicalSystems/VortexArraysSystemPtr.cpp).
//
// Per candidate pair the model needs the exact distance dr = sqrt(dx^2 + dy^2)
// and, for cohesion, the bearing of j from i: pass 1 sums the alignment (dr <=
// xi_a), anti-alignment (xi_a < dr <= rho) and cohesion (dr <= xi_r) terms with
// their counts (:472-488); pass 2 (the stochastic Runge-Kutta form) sums the
// additional derivative (:695-728) from the pass-1 rates of both particles.
//
// One lane takes one particle, as in the particle-per-lane passes (spc_lane.cuh):
// a float test drops candidates beyond max(rho, xi_r) for certain, the rest
// become bits, and the lanes walk their bits together (the reference's visiting
// order; all of the system's particles in index order when rho > L/4,
// :164-183).  The pair terms are FP64 with few operations of that pipe, which
// bounds these passes:
//  * the cutoffs compare dr^2 with the largest square whose root is within the
//    cutoff (the rounded root is monotonic, so the sets are those of dr);
//  * the minimum image of two positions of neighbouring cells is dx or dx -+ L;
//  * sin and cos of phi_j - phi_i and of the bearing minus phi_i come from the
//    particles' cos and sin, (dx, dy) / dr and the angle-difference identities
//    (a small sine or cosine is evaluated as the reference writes it, as in
//    add_pair; phi_j - phi_i by the differences of cos and sin and with what
//    their roundings left), and the strengths from their polynomials'
//    coefficients;
//  * the quotients by the counts are taken once of each sum.
// 19 operations a pair in pass 1 and 36 in pass 2, where sincos, atan2, quotients
// and minimum images took about 100 and 60 with 32 bytes a pair kept between the
// passes.  N = 12,800, L = 4, rho = 0.2: 149 and 288 us, before 1,338 and 1,143.
#pragma once

#include "spc_lane.cuh"

namespace spc {

// Per-particle results of a pass.
struct VAAcc {
  double align, coh;      // pass 1: (anti-)alignment, cohesion
  int c01, c2;            // their partners
  double a0, a1, b0, b1;  // pass 2: the additional terms, (anti-)alignment and cohesion
};

// Fused epilogue of the vortex-arrays passes for the particle at cell-order
// slot p, pool slot q.
template <int KIND>
__device__ void va_epilogue(const KArgs &a, int epi, const SysDesc &sd, int p, int q, double2 cs,
                            const VAAcc &r) {
  const SysConst &sc = sd.sc;
  const bool live = a.step_off < sd.budget;
  const int i = q - sd.pool_p0;
  const unsigned long long step = sd.step + (unsigned long long)a.step_off;
  const double dt = a.dt;
  double z0 = 0.0, z1 = 0.0;
  const bool draws = (epi == kEpiEulerPtr || epi == kEpiSrk2) && !a.noise && live;
  // velocity components (VortexArraysSystemPtr.cpp:491-504)
  const double d0 = dmul(sc.v0, cs.x), d1 = dmul(sc.v0, cs.y);
  if (draws) philox_normal2(sd.seed, sd.system_id, step, (uint32_t)i, z0, z1);
  if constexpr (KIND == kKindSin) {
    // k_next / derivative: velocity components always; the phase rate only
    // when there are (anti-)alignment partners, then the cohesion mean added
    // on top
    auto rate_from = [&](double prev) {
      double v = prev;
      const Count n1 = count_of(r.c01), n2 = count_of(r.c2);
      if (r.c01 > 0) v = ddiv_by(r.align, n1.n, n1.r);
      if (r.c2 > 0) v = dadd(v, ddiv_by(r.coh, n2.n, n2.r));
      return v;
    };
    if (epi == kEpiSrk1) {
      a.dphi_s[p] = rate_from(0.0);  // the stepper zero-fills derivative
      a.cnt_s[p] = r.c01;
      a.va_cnt2[p] = r.c2;
    } else if (epi == kEpiEulerPtr) {
      if (!live) return;
      // StochasticEulerStepperPtr.hpp:56-76
      const double rate = rate_from(0.0);
      const double dW = dmul(a.sdt, noise_at(a, q, 0, z0, z1));
      const double xs = dadd(a.x[q], dmul(d0, dt));
      const double ys = dadd(a.y[q], dmul(d1, dt));
      a.phi[q] = dadd(a.phi[q], dadd(dmul(rate, dt), dmul(sc.s2D, dW)));
      a.x[q] = wrap_1d(xs, sc.rL, sc.L);
      a.y[q] = wrap_1d(ys, sc.rL, sc.L);
    } else if (epi == kEpiRkK || epi == kEpiRk4Combine) {
      if (!live) return;
      const int k = a.kq_out;
      a.kx[k][q] = d0;
      a.ky[k][q] = d1;
      a.kphi[k][q] = rate_from(a.kphi[k][q]);  // the persistent k keeps a stale rate (H5)
      if (epi == kEpiRk4Combine) {
        // RungeKutta4StepperPtr.cpp:57-61
        const double sx_ = dadd(dadd(dadd(a.kx[0][q], dmul(2.0, a.kx[1][q])), dmul(2.0, a.kx[2][q])), a.kx[3][q]);
        const double sy_ = dadd(dadd(dadd(a.ky[0][q], dmul(2.0, a.ky[1][q])), dmul(2.0, a.ky[2][q])), a.ky[3][q]);
        const double sp_ =
            dadd(dadd(dadd(a.kphi[0][q], dmul(2.0, a.kphi[1][q])), dmul(2.0, a.kphi[2][q])), a.kphi[3][q]);
        const double xs = dadd(a.x[q], ddiv(dmul(sx_, dt), 6.0));
        const double ys = dadd(a.y[q], ddiv(dmul(sy_, dt), 6.0));
        a.phi[q] = dadd(a.phi[q], dmul(ddiv(sp_, 6.0), dt));
        a.x[q] = wrap_1d(xs, sc.rL, sc.L);
        a.y[q] = wrap_1d(ys, sc.rL, sc.L);
      }
    }
  } else {
    // additional_derivative[i][0] *= sqrt(2 D) (VortexArraysSystemPtr.cpp:732)
    // the neighbours within a cutoff are those the first pass counted
    const int c01 = a.cnt_s[p], c2 = a.va_cnt2[p];
    const Count n1 = count_of(c01), n2 = count_of(c2);
    double s0 = 0.0, A1 = 0.0;
    if (c01 > 0) {
      s0 = ddiv_by(r.a0, n1.n, n1.r);
      A1 = ddiv_by(r.a1, n1.n, n1.r);
    }
    if (c2 > 0) {
      s0 = dadd(s0, ddiv_by(r.b0, n2.n, n2.r));
      A1 = dadd(A1, ddiv_by(r.b1, n2.n, n2.r));
    }
    const double A0 = dmul(s0, sc.s2D);
    const double d2 = a.dphi_s[p];
    if (epi == kEpiSrk2Out) {
      a.out_d[3 * (size_t)q] = d0;
      a.out_d[3 * (size_t)q + 1] = d1;
      a.out_d[3 * (size_t)q + 2] = d2;
      a.out_a[2 * (size_t)q] = A0;
      a.out_a[2 * (size_t)q + 1] = A1;
    } else {
      if (!live) return;
      // StochasticRungeKuttaStepperPtr.hpp:70-96 (no natural frequencies)
      const double U1 = noise_at(a, q, 0, z0, z1), U2 = noise_at(a, q, 1, z0, z1);
      const double sdt = a.sdt;
      const double dW = dmul(U1, sdt);
      const double dZ = dmul(dmul(dmul(0.5, dt), sdt), dadd(U1, ddiv_by(U2, kSqrt3, kRcpSqrt3)));
      const double D = sc.D;
      const double s2D = sc.s2D;
      const double dtdt_x = dmul(dmul(dmul(0.5, dadd(dmul(d2, d1), dmul(D, d0))), dt), dt);
      const double xs = dadd(a.x[q], dsub(dsub(dmul(d0, dt), dmul(dmul(s2D, d1), dZ)), dtdt_x));
      const double dtdt_y = dmul(dmul(dmul(0.5, dsub(dmul(d2, d0), dmul(D, d1))), dt), dt);
      const double ys = dadd(a.y[q], dadd(dadd(dmul(d1, dt), dmul(dmul(s2D, d0), dZ)), dtdt_y));
      const double ps = dadd(a.phi[q], dadd(dadd(dadd(dmul(d2, dt), dmul(s2D, dW)), dmul(A0, dZ)),
                                            dmul(dmul(dmul(0.5, A1), dt), dt)));
      a.x[q] = wrap_1d(xs, sc.rL, sc.L);
      a.y[q] = wrap_1d(ys, sc.rL, sc.L);
      a.phi[q] = ps;
    }
  }
}


// a <= b for doubles that are not negative (b not NaN), by their bit patterns
__device__ __forceinline__ bool le_bits(double a, double b) {
  return (unsigned long long)__double_as_longlong(a) <= (unsigned long long)__double_as_longlong(b);
}

// xj - xi by minimum image (PeriodicBoundaryConditions.cpp:22-35).  `near`: the
// pair passed the float test of a cell list with both cutoffs up to L/4, so the
// difference is within L/4 of 0 or of -+L, and the reference's truncated
// quotient is 0 or +-1, but +-2 at a difference of L itself (a copy that wraps
// to exactly L, against x = 0), which the general form takes.
__device__ __forceinline__ double va_image(const SysConst &sc, double xj, double xi, bool near) {
  const double d = dsub(xj, xi);
  const int hi = __double2hiint(d) & 0x7fffffff;
  if (!near || hi >= __double2hiint(sc.L)) return min_image_1d(d, sc.rL, sc.L);
  return hi > __double2hiint(sc.va_hL) ? dsub(d, copysign(sc.L, d)) : d;
}

__device__ __noinline__ double va_bearing(double dx, double dy, double phi) { return dsub(atan2(dy, dx), phi); }
__device__ __noinline__ double sin_library(double v) { return sin(v); }
__device__ __noinline__ double cos_library(double v) { return cos(v); }

// dr2 < 2^-900 (0 among them): its root, and (dx, dy) over it, would not have a
// double's precision by the short forms.
__device__ __forceinline__ bool va_tiny(double dr2) { return __double2hiint(dr2) < 0x07b00000; }

// sin and cos of (bearing - phi_i)
__device__ __forceinline__ void va_bearing_sincos(double dx, double dy, double dr, bool tiny, double2 ci, double phii,
                                                  double &s, double &c) {
  if (tiny) {
    const double t = va_bearing(dx, dy, phii);
    s = sin_library(t);
    c = cos_library(t);
    return;
  }
  s = ddiv(__fma_rn(dy, ci.x, -dmul(dx, ci.y)), dr);
  c = ddiv(__fma_rn(dx, ci.x, dmul(dy, ci.y)), dr);
  if (small_term(s)) s = sin_library(va_bearing(dx, dy, phii));
  if (small_term(c)) c = cos_library(va_bearing(dx, dy, phii));
}

// What one pair adds: pass 1 (anti-)alignment x and cohesion u, pass 2 x and y
// to the additional terms, u and v of cohesion.
struct VATerm {
  bool term, coh;
  double x, y, u, v;
};

// G lanes per particle: one, or a group of four, three of which test a row of
// the stencil each (or a third of an all-pairs system) and all of which form
// pair terms side by side.  The terms are added in the reference's order either
// way, so both give the same bits.  Few particles take groups: SRK step of N =
// 12,800, L = 4 652 us with one lane, 456 with four; N = 25,600 820
// and 943; N = 51,200 1,348 and 1,656.
constexpr int kVAGroupMax = 19200;

template <int KIND, int G>
__global__ void __launch_bounds__(kLaneThreads) k_va_pass(KArgs a, int epi) {
  __shared__ uint32_t s_bits[kLaneWords][kLaneThreads];
  __shared__ int s_slot[kLaneWords][kLaneThreads];
  const int tid = threadIdx.x, g = tid % G, lead = tid % kWarp - g;
  const int p_own = a.lane_p1 + (blockIdx.x * blockDim.x + tid) / G;
  if (G == 1 && p_own >= a.va_p1) return;  // no barrier below
  // groups: the warps stay whole, lanes past the end repeat the last particle
  const int p = min(p_own, a.va_p1 - 1);
  const int cell = cell_of_slot(a, p);
  const SysDesc &sd = a.sys[a.sys_of_c[cell]];
  const SysConst &sc = sd.sc;
  const bool ap = sc.allpairs != 0, near = !ap && sc.va_near;
  const double xi = a.sx[p], yi = a.sy[p], phii = a.sphi[p];
  const double2 ci = a.dcs[p];
  const double ddi = KIND == kKindCos2 ? a.dphi_s[p] : 0.0;
  const uint32_t ri = a.rest[p], rest_from = (ri & 0xf000u) - (2u << 12);
  const int rest_own = (int)(ri & 0xfffu);
  VAAcc r{0.0, 0.0, 0, 0, 0.0, 0.0, 0.0, 0.0};

  auto term_of = [&](int j, bool wanted) {
    VATerm t{false, false, 0.0, 0.0, 0.0, 0.0};
    const double dx = va_image(sc, a.sx[j], xi, near), dy = va_image(sc, a.sy[j], yi, near);
    const double dr2 = dadd(dmul(dx, dx), dmul(dy, dy));
    const bool align = le_bits(dr2, sc.va_t_xia), rho_pair = le_bits(dr2, sc.va_t_rho);
    t.term = wanted && (KIND == kKindSin ? align || rho_pair : rho_pair);
    t.coh = wanted && le_bits(dr2, sc.va_t_xir);
    const bool tiny = va_tiny(dr2);
    const double dr = tiny ? dsqrt(dr2) : sqrt_pos(dr2);
    const double2 cj = a.dcs[j];
    // AlignmentStrength (:737-749) and, over dr, AlignmentStrengthDerivative (:751-763)
    const bool in1 = !le_bits(sc.va_s_xia, dr2), in2 = !in1 && !le_bits(sc.va_s_rho, dr2);
    const double f = in1 ? __fma_rn(dr2, -sc.va_c1, sc.mu_plus)
                         : (in2 ? dmul(dmul(sc.va_c2, dsub(dr, sc.xi_a)), dsub(sc.rho, dr)) : 0.0);
    // the products of the differences round like the small sine of aligned phases
    // does; what the rounded cosines and sines lack is added (see sine_rest)
    const double ex = dsub(cj.x, ci.x), ey = dsub(cj.y, ci.y);
    double sp = __fma_rn(ey, ci.x, -dmul(ex, ci.y));
    const uint32_t rj = a.rest[j];
    if (((rj - rest_from) & 0xffffu) < kRestNear)
      sp = __fma_rn((double)((int)(rj & 0xfffu) - rest_own), 0x1p-64, sp);
    if (wanted && small_term(sp)) sp = sin_of_difference(a.sphi[j], phii, 0.0);
    if constexpr (KIND == kKindSin) {
      t.x = dmul(f, sp);  // VortexArraysSystemPtr.cpp:475-485
      if (t.coh) {        // :486-488
        double s, c;
        va_bearing_sincos(dx, dy, dr, tiny, ci, phii, s, c);
        t.u = dmul(-sc.kappa, s);
      }
    } else {
      // VortexArraysSystemPtr.cpp:706-728
      double cp = __fma_rn(cj.x, ci.x, dmul(cj.y, ci.y));
      if (wanted && small_term(cp)) cp = cos_of_difference(a.sphi[j], phii, 0.0);
      // ex, ey times v0: the velocity difference
      // the strength's derivative over dr, times v0; at dr = 0 the reference divides 0 by 0
      double gr = in1 ? -sc.va_g1 : 0.0;
      if (in2) gr = ddiv(dmul(sc.va_g2, __fma_rn(-2.0, dr, sc.va_xr)), dr);
      if (dr == 0.0) gr = __longlong_as_double(0x7ff8000000000000ll);
      const double q = __fma_rn(__fma_rn(ex, dx, dmul(ey, dy)), gr, dmul(-sc.va_2D, f));
      t.x = dmul(f, cp);
      t.y = __fma_rn(dsub(a.dphi_s[j], ddi), t.x, dmul(q, sp));
      if (t.coh) {
        double s, c;
        va_bearing_sincos(dx, dy, dr, tiny, ci, phii, s, c);
        const double turn = ddiv(dmul(sc.v0, __fma_rn(ey, dx, -dmul(ex, dy))), dr2);
        t.u = dmul(sc.kappa, c);
        t.v = __fma_rn(dmul(-sc.kappa, dsub(turn, ddi)), c, dmul(dmul(sc.kappa, sc.D), s));
      }
    }
    return t;
  };
  auto add = [&](bool term, bool coh, double x, double y, double u, double v) {
    if constexpr (KIND == kKindSin) {
      if (term) {
        r.align = dadd(r.align, x);
        ++r.c01;
      }
      if (coh) {
        r.coh = dadd(r.coh, u);
        ++r.c2;
      }
    } else {
      if (term) {
        r.a0 = dsub(r.a0, x);
        r.a1 = dadd(r.a1, y);
      }
      if (coh) {
        r.b0 = dadd(r.b0, u);
        r.b1 = dadd(r.b1, v);
      }
    }
  };

  int nw = 0;         // words listed
  bool full = false;  // G > 1: the row has more words than the list
  auto walk = [&]() {  // this lane's words, in order
    uint32_t bits = 0u;
    int slot = 0;
    for (int w = 0;;) {
      if (bits == 0u) {
        if (w == nw) break;
        bits = s_bits[w][tid];
        slot = s_slot[w][tid];
        ++w;
      }
      const int t = __clz(bits);
      bits ^= 0x80000000u >> t;
      const VATerm v = term_of(slot + t, true);
      add(v.term, v.coh, v.x, v.y, v.u, v.v);
    }
    nw = 0;
  };
  auto put = [&](uint32_t bits, int slot) {
    if ((unsigned)(p - slot) < (unsigned)kWarp) bits &= ~(0x80000000u >> (p - slot));  // not itself
    if (bits == 0u) return;
    s_bits[nw][tid] = bits;
    s_slot[nw][tid] = slot;
    ++nw;
  };

  const int nc = sc.nc, cl = cell - sd.c0, cy = cl / nc, cx = cl - cy * nc;
  const LaneRuns rn = lane_runs(cx, nc);
  const float2 fi = ap ? make_float2(0.0f, 0.0f) : a.fxy[p];
  const float xa = fi.x - (float)rn.sa * sc.cell_f, xb = fi.x - (float)rn.sb * sc.cell_f;
  // rows [k0, k1) of the stencil, or thirds of an all-pairs system; flush: walk
  // the list when it is full
  auto rows = [&](int k0, int k1, bool flush) {
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const float y = fi.y - (float)(k - 1) * sc.cell_f;
      const int *row = a.cell_start + sd.c0 + (ap ? 0 : adjust_cell(cy + k - 1, nc) * nc);
#pragma unroll 1
      for (int run = 0; run < (ap ? 1 : 2); ++run) {
        int j0, j1;
        if (ap) {
          const long long m = row[1] - row[0];
          j0 = row[0] + (int)(m * k / 3);
          j1 = row[0] + (int)(m * (k + 1) / 3);
        } else {
          j0 = row[run ? rn.b0 : rn.a0];
          j1 = row[run ? rn.b1 : rn.a1];
        }
        const float x = run ? xb : xa;
        for (int base = j0; base < j1; base += kWarp) {
          const int cnt = min(kWarp, j1 - base);
          uint32_t bits = 0xffffffffu;
          if (!ap) {
            // sign of d^2 - va_r2 (rounded outwards): beyond rho and xi_r for certain when clear
            int done = 0;
            for (; done < cnt; done += 4) {
              const float2 *f = a.fxy + base + done;
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const float2 d = add2(f[u], make_float2(-x, -y));
                bits = __funnelshift_l(__float_as_uint(cutoff_offset(d.x, d.y, -sc.va_r2)), bits, 1);
              }
            }
            bits <<= kWarp - done;
          }
          put(bits & first_bits(cnt), base);
          if (nw == kLaneWords) {
            if (flush) {
              walk();
            } else {
              full = true;
              return;
            }
          }
        }
      }
    }
  };

  if constexpr (G == 1) {
    rows(0, 3, true);
    walk();
  } else {
    constexpr unsigned kAll = 0xffffffffu;
    if (g < 3) rows(g, g + 1, false);
    __syncwarp();
    const bool alone = ((__ballot_sync(kAll, full) >> lead) & ((1u << G) - 1u)) != 0u;  // a very long row
    GroupWords words(nw, lead, alone);
    uint32_t bits = 0u;
    int slot = 0;
    while (true) {
      words.next(s_bits, s_slot, tid - g, bits, slot);
      const int m = __popc(bits);
      if (!__any_sync(kAll, m > 0)) break;
      const int j = group_pick(bits, slot, g, m, p);
      const VATerm t = term_of(j, g < m);
      __syncwarp();
      const unsigned terms = __ballot_sync(kAll, t.term) >> lead, all_cohs = __ballot_sync(kAll, t.coh);
      const unsigned cohs = all_cohs >> lead;
#pragma unroll
      for (int u = 0; u < G; ++u) {
        const double x = __shfl_sync(kAll, t.x, lead + u);
        const double y = KIND == kKindCos2 ? __shfl_sync(kAll, t.y, lead + u) : 0.0;
        double cu = 0.0, cv = 0.0;
        if (all_cohs != 0u) {  // the same for the whole warp
          cu = __shfl_sync(kAll, t.u, lead + u);
          if constexpr (KIND == kKindCos2) cv = __shfl_sync(kAll, t.v, lead + u);
        }
        add((terms >> u) & 1u, (cohs >> u) & 1u, x, y, cu, cv);
      }
    }
    if (g != 0 || p_own >= a.va_p1) return;
    if (alone) {  // the first lane walks as it tests
      nw = 0;
      rows(0, 3, true);
      walk();
    }
  }
  va_epilogue<KIND>(a, epi, sd, p, a.pidx[p], ci, r);
}

}  // namespace spc
