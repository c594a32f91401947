// mc_fp64.cuh -- the FP64 transport steps of the stochastic backward Monte
// Carlo, included by mc_device.cuh.  The same program, draws and decisions as the
// templates there (which carry the FP32 transport), arranged for the FP64 pipe:
// one FP64 warp instruction takes an SM partition 64 cycles, whatever the number
// of active lanes, so a step costs what its FP64 instructions cost.
//  - A logarithm is taken once per energy: the step's energy serves the physics
//    grid, the MIXED kernel's grid and the hard-scattering path, and an energy
//    that came from an inverse lookup keeps the interval and offset it was
//    formed from.
//  - Inverse lookups walk from the step's own interval (a step is at most 1 % of
//    the range) instead of taking the logarithm of the range.
//  - Interval widths are inverted once per medium (the columns pack_derived
//    appends to the FP64 media); other divisions, roots and elementary functions
//    are those of fp64_math.cuh; comparisons of positive numbers are integer.
//  - Quotients that only enter a comparison are compared as products.
// About 300 FP64 instructions per straggled and scattered step against about
// 1050.  run_backward_mc through 100 m of rock, 1-100 GeV: 10^2 histories 22.1 ->
// 10.4 ms, 10^4 67.0 -> 22.1 ms, 10^5 182.7 -> 72.6 ms; a direction of 256
// histories 13.3 -> 5.9 ms.  Histories agree with the templates' form to 5e-10.

// Derived columns of an FP64 medium: inverse interval widths of log E, the CSDA
// range and the restricted range after the transport paths, and of the MIXED
// kernel's energies after its columns.
enum { X_ILE = 0, X_ICR, X_IMR, X_NCOL };
constexpr int K_IE = K_NCOL;
constexpr double kMagic = 6755399441055744.0;  // 1.5 2^52: adding it rounds to an integer

__device__ __forceinline__ const double* xcol(const Med<double>& m, int k) {
  return m.col(MC_LB1 + 2 * m.slots + k);
}
__device__ __forceinline__ bool positive_finite(double x) {  // x > 0 and finite
  return (unsigned long long)(__double_as_longlong(x) - 1) < 0x7fefffffffffffffull;
}

// Interval of x on the physics grid, lx = log x.
__device__ __forceinline__ Loc<double> locate_log(const Med<double>& m, double x, double lx) {
  Loc<double> L{0, 0, 0.0};
  const double* E = m.col(MC_E);
  if (!f64::lt_pos(E[0], x)) {
    L.edge = -1;
    return L;
  }
  if (!f64::lt_pos(x, E[m.n - 1])) {
    L.edge = 1;
    return L;
  }
  const double *lE = m.col(MC_LE), *inv = xcol(m, X_ILE);
  int i;
  if (m.uniform) {
    i = __double2loint(fma(lx - m.lE0, m.inv_dlE, kMagic));
    i = i < 0 ? 0 : (i > m.n - 2 ? m.n - 2 : i);
  } else {
    i = bisect_r(lE, m.n, lx);
  }
  L.t = f64::grid_offset(lE, inv, m.n, lx, i);
  L.i = i;
  return L;
}
__device__ __forceinline__ Loc<double> locate(const Med<double>& m, double x) {
  return locate_log(m, x, log64(x));
}
// Energy at the range X of a range column, walking from interval i; *L its place
// on the grid.
__device__ __forceinline__ double energy_at(const Med<double>& m, int col, double X, int i, Loc<double>* L) {
  const double *Rc = m.col(col), *lE = m.col(MC_LE);
  const int n = m.n;
  *L = Loc<double>{0, 0, 0.0};
  if (!f64::lt_pos(Rc[0], X)) {
    L->edge = -1;
    return m.col(MC_E)[0];
  }
  if (!f64::lt_pos(X, Rc[n - 1])) {
    L->edge = 1;
    return m.col(MC_E)[n - 1];
  }
  while (i < n - 2 && !f64::lt_pos(X, Rc[i + 1])) ++i;
  while (i > 0 && f64::lt_pos(X, Rc[i])) --i;
  L->i = i;
  L->t = (X - Rc[i]) * xcol(m, col == MC_CR ? X_ICR : X_IMR)[i];
  return exp64(fma(L->t, lE[i + 1] - lE[i], lE[i]));
}
// MIXED kernel location of x, lx = log x (klocate_e).
__device__ __forceinline__ KLoc<double> klocate_log(const Med<double>& m, double x, double lx, int* status) {
  const double* xs = m.kcol(K_E);
  const int n = m.nk;
  KLoc<double> L{0, 0, 0.0};
  if (!m.kuniform) return klocate(xs, n, x, status);
  if (f64::lt_pos(x, xs[0])) {
    *status |= ST_DOMAIN_LO;
    L.edge = -1;
    return L;
  }
  if (f64::lt_pos(xs[n - 1], x)) {
    *status |= ST_DOMAIN_HI;
    L.edge = 1;
    return L;
  }
  int i = __double2loint(fma(lx - m.lE0, m.kinv_dlE, kMagic));
  i = i < 0 ? 0 : (i > n - 2 ? n - 2 : i);
  while (i > 0 && f64::lt_pos(x, xs[i])) --i;
  while (i < n - 2 && !f64::lt_pos(x, xs[i + 1])) ++i;
  L.i = i;
  L.f = (x - xs[i]) * m.kcol(K_IE)[i];
  return L;
}
__device__ __forceinline__ KLoc<double> klocate_e(const Med<double>& m, double x, int* status) {
  return klocate_log(m, x, log64(x), status);
}
// Location of x on the kernel's range or hazard axis, walking from node i.
__device__ __forceinline__ KLoc<double> klocate_from(const Med<double>& m, int xcol_, double x, int i,
                                                     int* status) {
  const double* xs = m.kcol(xcol_);
  const int n = m.nk;
  KLoc<double> L{0, 0, 0.0};
  if (f64::lt_pos(x, xs[0])) {
    *status |= ST_DOMAIN_LO;
    L.edge = -1;
    return L;
  }
  if (f64::lt_pos(xs[n - 1], x)) {
    *status |= ST_DOMAIN_HI;
    L.edge = 1;
    return L;
  }
  while (i < n - 2 && !f64::lt_pos(x, xs[i + 1])) ++i;
  while (i > 0 && f64::lt_pos(x, xs[i])) --i;
  const double d = xs[i + 1] - xs[i];
  L.i = i;
  L.f = d == 0.0 ? 0.0 : f64::div(x - xs[i], d);
  return L;
}
// Hazard rate per grammage at an energy.
__device__ __forceinline__ double rate_at(const Med<double>& m, double x, double lx, int* status) {
  return kat(m.kcol(K_SIG), m.nk, klocate_log(m, x, lx, status));
}

__device__ __forceinline__ double transport_path(const Med<double>& m, const Loc<double>& L) {
  if (m.nm == 1) return at(m, L, MC_LB1);
  double inv = 0.0;
  for (int j = 0; j < m.nm; ++j) {
    const double lp = at(m, L, MC_LB1 + j);
    if (lp > 0.0) inv += f64::div(m.frac[j], lp);
  }
  return inv > 0.0 ? f64::rcp(inv) : 1e9;
}
// Hard-scattering path (ehs_path) as num / den, at the place L of the energy K.
__device__ __forceinline__ void ehs_ratio(const Med<double>& m, double K, const Loc<double>& L, double mass,
                                          double elastic_ratio, double* num, double* den) {
  const double p2 = K * (K + 2.0 * mass);
  *den = 1.0;
  if (m.nm == 1) {
    const double Lb = at(m, L, m.lbe(0));
    if (!f64::lt_pos(K, 1e-3) && Lb > 0.0 && Lb < kEhsPathMax * p2) {
      *num = Lb;
      *den = p2;
    } else {
      *num = ehs_single(m, 0, K, L, mass, elastic_ratio);
    }
    return;
  }
  double inv = 0.0;
  for (int j = 0; j < m.nm; ++j) {
    const double Lb = at(m, L, m.lbe(j));
    if (!f64::lt_pos(K, 1e-3) && Lb > 0.0 && Lb < kEhsPathMax * p2) {
      inv += f64::div(m.frac[j] * p2, Lb);
    } else {
      const double lp = ehs_single(m, j, K, L, mass, elastic_ratio);
      if (lp > 0.0 && lp < kEhsPathMax) inv += f64::div(m.frac[j], lp);
    }
  }
  if (inv > 0.0) {
    *num = 1.0;
    *den = inv;
  } else {
    *num = kEhsPathMax;
  }
}

// rotate_direction (src/Straggling.jl:645-710).
static __device__ __noinline__ void rotate(State<double>& s, double mu, Stream& g) {
  const double ct = 1.0 - 2.0 * mu, st2 = 4.0 * mu * (1.0 - mu);
  if (st2 <= 0.0) return;
  const double st = f64::sqrt(st2), d0 = s.ux, d1 = s.uy, d2 = s.uz;
  const double ax = fabs(d0), ay = fabs(d1), az = fabs(d2);
  // a unit vector normal to the direction, from its two components that leave
  // out the smallest one or the y and z axes
  const bool xz = f64::lt_pos(ay, ax) && f64::lt_pos(az, ax), xy = !f64::lt_pos(ay, ax) && f64::lt_pos(az, ay);
  const double p = xz || xy ? d0 : d1, q = xy ? d1 : d2, nrm = f64::rsqrt(fma(p, p, q * q));
  const double u0x = xz ? -d2 * nrm : (xy ? d1 * nrm : 0.0);
  const double u0y = xz ? 0.0 : (xy ? -d0 * nrm : d2 * nrm);
  const double u0z = xz ? d0 * nrm : (xy ? 0.0 : -d1 * nrm);
  const double u1x = u0y * d2 - u0z * d1, u1y = u0z * d0 - u0x * d2, u1z = u0x * d1 - u0y * d0;
  double cp, sp;
  f64::sincospi(1.0 - 2.0 * uni<double>(g), &sp, &cp);
  const double a = st * cp, b = st * sp;
  double nx = fma(ct, d0, fma(a, u0x, b * u1x));
  double ny = fma(ct, d1, fma(a, u0y, b * u1y));
  double nz = fma(ct, d2, fma(a, u0z, b * u1z));
  const double n2 = fma(nx, nx, fma(ny, ny, nz * nz));
  if (n2 > 0.0) {
    const double r = f64::rsqrt(n2);
    nx *= r;
    ny *= r;
    nz *= r;
  }
  s.ux = nx;
  s.uy = ny;
  s.uz = nz;
}

// sample_soft_scattering (src/Straggling.jl:539-590, :1204-1253) over the
// grammage dX: ilb1 = dX / 4 (1/lb0 + 1/lb1).
__device__ __forceinline__ double soft_angle(const Med<double>& m, double lb0, const Loc<double>& L1, double k1,
                                             double dX, Stream& g) {
  if (!(dX > 0.0)) return 0.0;
  const double lb1 = k1 > 0.0 ? transport_path(m, L1) : lb0;
  if (!(lb0 > 0.0) && !(lb1 > 0.0)) return 0.0;
  double ilb1 = 0.25 * dX;
  if (lb0 > 0.0 && lb1 > 0.0) ilb1 *= f64::div(lb0 + lb1, lb0 * lb1);
  else ilb1 *= f64::rcp(lb0 > 0.0 ? lb0 : lb1);
  if (f64::lt_pos(ilb1, 1e-12)) return 0.0;
  if (f64::lt_pos(1.0, ilb1)) ilb1 = 1.0;
  for (int it = 0; it < 1000; ++it) {
    const double u = uni<double>(g);
    if (u == 0.0) continue;
    const double mu = -ilb1 * log64(u);
    if (mu <= 1.0) return fmax(mu, 0.0);
  }
  return ilb1;
}

// The step's end (straggled_end): lckf = log ckf, irho = 1 / density.
__device__ __forceinline__ double straggled_end64(const Med<double>& m, const Consts& C, State<double>& s,
                                                  const Loc<double>& Li, double lb0, double ki, double kf,
                                                  double ckf, double lckf, double dX, double dw, int proc, int elem,
                                                  bool del, bool ehs, double k_ehs, double irho, double step,
                                                  bool shortened, bool scattering, Stream& g) {
  const double mass = C.mass;
  // the reference's dX / density: the requested length unless shortened
  const double astep = shortened ? dX * irho : step, oz = s.uz;
  const Loc<double> Lc = locate_log(m, ckf, lckf);
  if (scattering) {
    if (del && proc > 0) {
      double mu;
      if (proc == 1 || proc == 2) mu = polar_brems(mass, kf, ckf, m.el[kElStride * elem + 4], g);
      else mu = proc == 3 ? polar_photo(mass, kf, ckf, g) : polar_ioni(mass, kf, ckf);
      if (mu > 0.0) rotate(s, mu, g);
    }
    if (ehs) {
      const double mu = scattering_angle(m, mass, k_ehs, g);
      if (mu > 0.0) rotate(s, mu, g);
    }
    const double mu = soft_angle(m, lb0, Lc, ckf, dX, g);
    if (mu > 0.0) rotate(s, mu, g);
  }
  const double pt = 0.5 * astep * mass *
                    (f64::rsqrt(ki * (ki + 2.0 * mass)) + f64::rsqrt(ckf * (ckf + 2.0 * mass)));
  s.z = fma(-astep, oz, s.z);
  s.w = s.w * f64::div(at(m, Lc, MC_MS), at(m, Li, MC_MS)) * exp64(-f64::div(pt, C.ctau)) * dw;
  s.E = kf;
  return astep;
}
__device__ __forceinline__ double straggled_end(const Med<double>& m, const Consts& C, State<double>& s,
                                                const Loc<double>& Li, double lb0, double ki, double kf,
                                                double ckf, double dX, double dw, int proc, int elem, bool del,
                                                bool ehs, double k_ehs, double density, double step,
                                                bool shortened, bool scattering, Stream& g) {
  return straggled_end64(m, C, s, Li, lb0, ki, kf, ckf, log64(ckf), dX, dw, proc, elem, del, ehs, k_ehs,
                         f64::rcp(density), step, shortened, scattering, g);
}
__device__ __forceinline__ double straggled_end_in(const Med<double>& m, const Consts& C, State<double>& s,
                                                   const Loc<double>& Li, double lb0, double ki, double kf,
                                                   double ckf, double dX, double dw, int proc, int elem, bool del,
                                                   bool ehs, double k_ehs, double density, double step,
                                                   bool shortened, bool scattering, Stream& g) {
  return straggled_end(m, C, s, Li, lb0, ki, kf, ckf, dX, dw, proc, elem, del, ehs, k_ehs, density, step,
                       shortened, scattering, g);
}

// A straggled step (src/Geometry.jl:148-357) up to its hard-event decision; true
// when it suspended on the event's DCS sum.  lki = log of the step's energy.
template <bool MOVED>
__device__ __forceinline__ bool straggled_step64(const Med<double>& m, const Consts& C, State<double>& s,
                                                 const Loc<double>& Li, double lki, double lb0, double density,
                                                 double step, Stream& g, bool scattering, double energy_limit,
                                                 Cont<double>& x) {
  const double ki = s.E, irho = f64::rcp(density), Xi = at(m, Li, MC_MR);
  double dX = step * density;
  bool shortened = false;
  Loc<double> L1;
  double k1 = energy_at(m, MC_MR, Xi + dX, Li.i, &L1);
  // fluctuate_energy_loss, backward (src/Straggling.jl:103-173): ratio = rn / rd
  double kf = k1, rn = 1.0, rd = 1.0;
  if (ki > 0.001) {
    const double dk0 = fabs(ki - k1);
    if (k1 > 0.0 && dk0 > 0.0) {
      double dk12 = 0.5 * dX * (at(m, Li, MC_STRAG) + at(m, L1, MC_STRAG));
      if (dX > 0.05 * Xi) dk12 *= 1.0 - f64::div(dX, dk0) * (at(m, L1, MC_MS) - at(m, Li, MC_MS));
      const double dk1 = dk12 > 0.0 ? f64::sqrt(dk12) : 0.0;
      if (dk1 > 0.0) {
        if (dk0 >= 3.0 * dk1) {
          k1 = fma(truncated_randn<double>(g), dk1, k1);
        } else if (dk0 >= 1.7320508 * dk1) {
          k1 = fma(1.7320508 * (1.0 - 2.0 * uni<double>(g)), dk1, k1);
        } else {
          const double dk32 = 3.0 * dk12, dk02 = dk0 * dk0;
          const double a = 1.0 - f64::div(dk32 - dk02, dk32 + 3.0 * dk02);
          if (uni<double>(g) <= a) {
            const double b = f64::div(0.5 * (dk32 + 3.0 * dk02), dk0);
            k1 = fma(b, uni<double>(g), ki);
            if (k1 < 0.0) k1 = 0.0;
          } else {
            k1 = ki;
          }
        }
      }
      rn = fabs(ki - k1);
      rd = dk0;
      if (rn == 0.0) rn = rd;  // a ratio of zero counts as one
    }
    kf = k1 > ki ? k1 : ki;
  }
  if (energy_limit > 0.0 && kf >= energy_limit) {
    const double dk = fabs(ki - kf);
    if (dk > 0.0) {
      dX = dX * f64::div(fabs(energy_limit - ki), dk);
      kf = energy_limit;
      shortened = true;
    }
  }
  const double lkf = log64(kf);
  bool del = false, ehs = false;
  double X_del = CUDART_INF, k_del = 0.0, X_ehs = CUDART_INF, k_ehs = 0.0;
  const double rate = fmax(rate_at(m, ki, lki, &s.status), rate_at(m, kf, lkf, &s.status));
  if (rate > 0.0) {
    const double e = expo<double>(g);
    if (e < dX * rate) {
      const double cand = f64::div(e, rate);
      Loc<double> Lh;
      const double kh = energy_at(m, MC_MR, Xi + cand, Li.i, &Lh);
      const double pre = fma(f64::div(rn, rd), fabs(kh - ki), ki);
      if (pre > 0.0 && uni<double>(g) * rate <= rate_at(m, pre, log64(pre), &s.status)) {
        del = true;
        X_del = cand;
        k_del = pre;
      }
    }
  }
  if (scattering) {
    // sample_ehs_event, backward (src/Straggling.jl:373-434); kf >= ki
    const bool swap = f64::lt_pos(ki, 0.001);
    const double k0 = swap ? kf : ki;
    const Loc<double> L0 = swap ? locate_log(m, kf, lkf) : Li;
    double num, den;
    ehs_ratio(m, k0, L0, C.mass, C.elastic_ratio, &num, &den);
    if (num > 0.0 && num < kEhsPathMax * den) {
      const double zeta = uni<double>(g);
      if (zeta > 0.0) {
        const double lz = -log64(zeta) * num;
        if (lz < dX * den) {
          const double X = f64::div(lz, den);
          Loc<double> Lh;
          const double kh = energy_at(m, MC_MR, Xi + X, Li.i, &Lh);
          const double k = fma(f64::div(rn, rd), fabs(ki - kh), ki);
          if (k > 0.0) {
            double n2, d2;
            ehs_ratio(m, k, locate(m, k), C.mass, C.elastic_ratio, &n2, &d2);
            // r = lbk / lb > 0; the candidate stands with probability 1 / r
            if (n2 > 0.0 && n2 < kEhsPathMax * d2) {
              const double a = n2 * den, b = num * d2;
              if (uni<double>(g) * a <= b) {
                ehs = true;
                X_ehs = X;
                k_ehs = k;
              }
            }
          }
        }
      }
    }
  }
  if (del && ehs) {
    if (X_del <= X_ehs) ehs = false;
    else del = false;
  }
  double dw = 1.0, ckf = kf, lckf = lkf;
  int proc = 0, elem = -1;
  if (del) {
    DelOut d;
    if (del_start(m, C, k_del, g, &s.status, &d, x)) {
      x.details = 1;
      x.a = step;
      x.r0 = ki;
      x.r1 = k_del;
      x.r2 = X_del;
      x.r3 = density;
      x.flag = scattering;
      return true;
    }
    ckf = k_del;
    lckf = log64(ckf);
    kf = d.energy;
    dw = d.weight;
    proc = d.process;
    elem = d.element;
    dX = X_del;
    shortened = true;
  }
  if (ehs) {
    kf = ckf = k_ehs;
    lckf = log64(ckf);
    dX = X_ehs;
    shortened = true;
  }
  const double moved = straggled_end64(m, C, s, Li, lb0, ki, kf, ckf, lckf, dX, dw, proc, elem, del, ehs, k_ehs,
                                       irho, step, shortened, scattering, g);
  if (MOVED) x.moved = moved;
  return false;
}

// The event loop of a mixed step from x.event (src/MixedTransport.jl:144-200);
// true when it suspended on a DCS sum.  A kernel energy that came from a range
// or a hazard keeps its place: all columns are linear in that place.
__device__ __forceinline__ bool mixed_run64(const Med<double>& m, const Consts& C, State<double>& s,
                                            Cont<double>& x, Stream& g, double energy_limit) {
  const int nk = m.nk;
  const double *kE = m.kcol(K_E), *kR = m.kcol(K_R), *kH = m.kcol(K_H);
  const double Emax = kE[nk - 1], mass = C.mass, irho = f64::rcp(x.c);
  for (; x.event < C.event_cap; ++x.event) {
    const double k = x.r0;
    if (x.a <= x.d || k >= x.r2) {
      mixed_end(s, x, Emax, energy_limit, false);
      return false;
    }
    const KLoc<double> Lk = klocate_e(m, k, &s.status);
    const double ri = kat(kR, nk, Lk), hi = kat(kH, nk, Lk);
    // the ceiling's place, then the endpoint's
    KLoc<double> Le{nk - 2, 1, 0.0};
    if (x.r2 < Emax) Le = klocate_e(m, x.r2, &s.status);
    const double rtc = fmax(0.0, kat(kR, nk, Le) - ri);
    double eg = rtc, pre = x.r2;
    if (x.a < rtc) {
      eg = x.a;
      Le = klocate_from(m, K_R, ri + eg, Lk.i, &s.status);
      pre = kat(kE, nk, Le);
      if (pre < k) {
        pre = k;
        Le = Lk;
      }
    }
    const double eventh = hi + expo<double>(g);
    const bool occurs = eventh < kat(kH, nk, Le);
    double dx = eg;
    if (occurs) {
      Le = klocate_from(m, K_H, eventh, Lk.i, &s.status);
      pre = kat(kE, nk, Le);
      if (pre < k) {
        pre = k;
        Le = Lk;
      }
      dx = fmax(0.0, kat(kR, nk, Le) - ri);
    }
    double dt;
    if (dx <= 8.0 * ulp_up(fabs(ri)) || pre - k <= 8.0 * ulp_up(fabs(k)))
      dt = 0.5 * dx * irho * mass * (f64::rsqrt(k * (k + 2.0 * mass)) + f64::rsqrt(pre * (pre + 2.0 * mass)));
    else
      dt = (kat(m.kcol(K_T), nk, Le) - kat(m.kcol(K_T), nk, Lk)) * irho;
    x.r1 *= f64::div(kat(m.kcol(K_S), nk, Le), kat(m.kcol(K_S), nk, Lk)) * exp64(-f64::div(dt, C.ctau));
    x.b += dx;
    x.a = fmax(0.0, x.a - dx);
    x.r0 = pre;
    if (!occurs) {
      mixed_end(s, x, Emax, energy_limit, false);
      return false;
    }
    DelOut d;
    if (del_start(m, C, pre, g, &s.status, &d, x)) {
      x.details = 0;
      return true;
    }
    if (mixed_event(s, x, d)) {
      mixed_end(s, x, Emax, energy_limit, false);
      return false;
    }
  }
  mixed_end(s, x, Emax, energy_limit, true);
  return false;
}

// Deterministic CSDA step on a medium (src/Geometry.jl:424-457).
__device__ __forceinline__ void csda_step(const Med<double>& m, const Consts& C, State<double>& s,
                                          const Loc<double>& Li, double density, double step) {
  const double mass = C.mass, ki = s.E;
  Loc<double> Lf;
  const double kf = energy_at(m, MC_CR, at(m, Li, MC_CR) + step * density, Li.i, &Lf);
  double d;
  const double dt = step * f64::inv_beta_gamma(0.5 * (ki + kf) / mass, &d);
  s.z = fma(-step, s.uz, s.z);
  s.w = s.w * f64::div(at(m, Lf, MC_CS), at(m, Li, MC_CS)) * exp64(-f64::div(dt, C.ctau));
  s.E = kf;
}
