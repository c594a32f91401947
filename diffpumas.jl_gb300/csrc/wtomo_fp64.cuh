// wtomo_fp64.cuh -- the FP64 instance of the water-fraction CSDA walk and its
// kernel (wtomo.cu).  Same walk, branches and derivatives as the reference's
// (src/Tomography.jl:444-551), arranged for the FP64 pipe, which issues one
// warp instruction per 64 cycles and SM partition and bounds everything here:
//  - S(E) at the end of a step serves the next step's start (the reference
//    evaluates it again at the same energy), so a Heun step locates two
//    energies instead of three;
//  - the weight's stopping-power ratios S(E')/S(E) telescope over a segment and
//    its decay factors multiply to exp(-sum ds/(beta gamma c tau)): one division
//    per segment and one exponential per path instead of three and one per step;
//  - tangents are written out per step (d log S/d log E of the interval times
//    dE/E) instead of carried through every operation as dual numbers;
//  - interval searches start at the step's last interval and compare signs and
//    exponents of the offset, the elementary functions are those of
//    fp64_math.cuh, and the straggling and hard-loss increments are formed only
//    where the correction that reads them is on.
//  - the lanes of a warp step together: a finished lane repeats its last state
//    without keeping it, and every step ends in a warp barrier.  Lanes left to
//    end their loops by themselves drifted apart (2.3 of 32 lanes per
//    instruction, four times slower than the dual numbers).
// About 75 FP64 instructions per air step and lane against about 550 for the dual
// numbers.  A direction is one warp, so one-warp CTAs put each on an SM
// partition of its own.  192 directions, 32 nodes, with the Jacobian: 49.2 ->
// 9.6 ms.

namespace dp {
namespace wt64 {

using wt::Lane;
using wt::Params;
using wt::kMaxChunks;
constexpr int kThreads = 32;

// Columns derived in shared memory: inverse interval widths of log E, and the
// differences of the CSDA stopping powers over the intervals.
enum { D_INV = 0, D_R, D_W, D_P, D_A, kDerived };

struct Tables {
  const double* c[wt::kSlots];
  const double* d[kDerived];
  int n;
  long long lo, hi;  // bit patterns of the grid's end energies
};
struct Run {
  double half_inv_m, inv_ctau;
};

// Place of an energy on the grid: offset t in interval i, inverse width il (0
// at the clamped ends, where the derivative vanishes).
struct Pos {
  int i;
  double t, il;
};
__device__ __forceinline__ Pos locate(const Tables& tb, double E, int i) {
  const long long b = __double_as_longlong(E);
  Pos p{0, 0.0, 0.0};
  if (b >= tb.hi) {
    p = Pos{tb.n - 2, 1.0, 0.0};
  } else if (b > tb.lo) {
    const double lE = f64::log(E);
    const double* inv = tb.d[D_INV];
    p.t = f64::grid_offset(tb.c[wt::S_LE], inv, tb.n, lE, i);
    p.i = i;
    p.il = inv[i];
  }
  __syncwarp();
  return p;
}
// First interval of a walk (bisection on the energies).
__device__ __forceinline__ int first_interval(const Tables& tb, double E) {
  int lo = 0, hi = tb.n - 1;
  while (lo < hi - 1) {
    const int mid = (lo + hi) >> 1;
    if (f64::lt_pos(E, tb.c[wt::S_E][mid])) hi = mid; else lo = mid;
  }
  return lo;
}

// A property at a place: value, derivative in log E and in the water fraction.
struct Val {
  double v, sl, sw;
};
// One material's column and its interval differences.
struct OneMaterial {
  const double *y, *d;
  __device__ __forceinline__ Val at(const Pos& p) const {
    return Val{fma(p.t, d[p.i], y[p.i]), d[p.i] * p.il, 0.0};
  }
};
// A cell of water fraction w: (1 - w) r + w q with r the rock, or half rock and
// half porous material in the porous top layer (src/Tomography.jl:303-352).
struct CellMix {
  const double *r, *dr, *q, *dq, *p, *dp;  // p: null without the porous layer
  double w;
  __device__ __forceinline__ Val at(const Pos& o) const {
    double yr = r[o.i], er = dr[o.i];
    if (p) {
      yr = 0.5 * (yr + p[o.i]);
      er = 0.5 * (er + dp[o.i]);
    }
    const double a = fma(o.t, er, yr), e = dq[o.i], b = fma(o.t, e, q[o.i]) - a;
    return Val{fma(w, b, a), fma(w, e - er, er) * o.il, b};
  }
};
// The same for a column whose differences are not tabulated.
__device__ __forceinline__ Val mix_at(const double* r, const double* q, const double* p, double w,
                                      const Pos& o) {
  double y0 = r[o.i], y1 = r[o.i + 1];
  if (p) {
    y0 = 0.5 * (y0 + p[o.i]);
    y1 = 0.5 * (y1 + p[o.i + 1]);
  }
  const double er = y1 - y0, e = q[o.i + 1] - q[o.i];
  const double a = fma(o.t, er, y0), b = fma(o.t, e, q[o.i]) - a;
  return Val{fma(w, b, a), fma(w, e - er, er) * o.il, b};
}

// A walk in flight: energy, its place and tangents (n = 0: the segment's
// entry energy, n = 1: its water fraction), S there and its tangents, and the
// segment's sum of ds / (beta gamma).
template <int N>
struct Walk {
  double E, iE, S, tau;
  double dE[N], dS[N], dtau[N];
  int i;
};
template <int N, class M>
__device__ __forceinline__ void begin(const Tables& tb, const M& m, Walk<N>& k) {
  const Pos p = locate(tb, k.E, k.i);
  const Val v = m.at(p);
  k.i = p.i;
  // (of a normal energy; zero, subnormal and negative ones lie below the grid, where no
  // derivative uses it)
  k.iE = f64::hi32(k.E) >= 0x00100000 ? f64::rcp(k.E) : 0.0;
  k.S = v.v;
  k.tau = 0.0;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    k.dE[n] = n == 0 ? 1.0 : 0.0;
    k.dS[n] = v.sl * k.iE * k.dE[n] + (n == 1 ? v.sw : 0.0);
    k.dtau[n] = 0.0;
  }
}
__device__ __forceinline__ bool positive_finite(double x) {
  return uint32_t(f64::hi32(x) - 1) < 0x7fefffffu;
}
// One Heun step of length ds and grammage gx (src/Tomography.jl:455-471) from
// k to k; false on an invalid step (k is then not to be kept).
template <int N, class M>
__device__ __forceinline__ bool heun(const Tables& tb, const Run& R, const M& m, Walk<N>& k, double ds,
                                     double gx, const double (&dds)[N], const double (&dgx)[N]) {
  const double Ep = fma(k.S, gx, k.E);
  const Pos p1 = locate(tb, Ep, k.i);
  const Val v1 = m.at(p1);
  const double a1 = v1.sl * f64::rcp(Ep);
  const double sum = k.S + v1.v, h = 0.5 * gx, En = fma(sum, h, k.E);
  const bool valid = (unsigned long long)__double_as_longlong(En) < 0x426d1a94a2000000ull;  // 1e12
  const Pos p2 = locate(tb, En, k.i);
  const Val v2 = m.at(p2);
  const double iEn = f64::rcp(En), a2 = v2.sl * iEn;
  double dib;
  const double x = (k.E + En) * R.half_inv_m, ib = f64::inv_beta_gamma(x, &dib);
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const double dEp = fma(k.S, dgx[n], fma(k.dS[n], gx, k.dE[n]));
    const double dS1 = fma(a1, dEp, n == 1 ? v1.sw : 0.0);
    const double dEn = fma(0.5 * sum, dgx[n], fma(k.dS[n] + dS1, h, k.dE[n]));
    k.dtau[n] += fma(dds[n], ib, ds * dib * ((k.dE[n] + dEn) * R.half_inv_m));
    k.dE[n] = dEn;
    k.dS[n] = fma(a2, dEn, n == 1 ? v2.sw : 0.0);
  }
  k.tau = fma(ds, ib, k.tau);
  k.E = En;
  k.iE = iEn;
  k.i = p2.i;
  k.S = v2.v;
  return valid;
}
// The grammage of a 2 % energy gain, at least `least`, and its relative tangents.
template <int N>
__device__ __forceinline__ double gain_limit(const Walk<N>& k, double least, double (&rel)[N]) {
  const bool small = f64::lt_pos(k.E, 1e-6);
  const double iS = f64::rcp(k.S), g = wt::kMaxGain * (small ? 1e-6 : k.E) * iS;
  const bool clamp = f64::lt_pos(g, least);
#pragma unroll
  for (int n = 0; n < N; ++n)
    rel[n] = clamp ? 0.0 : (small ? 0.0 : k.dE[n] * k.iE) - k.dS[n] * iS;
  return clamp ? least : g;
}
// Closes a segment: the weight factor S_end / S_start and d log(weight).
template <int N>
__device__ __forceinline__ void finish(const Walk<N>& k, const Run& R, double iS0, const double (&g0)[N],
                                       double& ratio, double& tau, double (&g)[N]) {
  const double iS = f64::rcp(k.S);
  ratio *= k.S * iS0;
  tau += k.tau;
#pragma unroll
  for (int n = 0; n < N; ++n) g[n] = k.dS[n] * iS - g0[n] - k.dtau[n] * R.inv_ctau;
}

// propagate_csda_cell_segment / propagate_csda_uniform_segment (:444-509):
// density rho with d log rho / d w = lrho.  k.E and k.i enter and leave; ratio
// and tau accumulate the weight, g receives d log(weight).  All lanes of the
// warp call it; ok: the lane's walk is valid so far, and on return still is.
template <int N, class M>
__device__ __forceinline__ void solid_segment(const Tables& tb, const Run& R, const M& m, double rho,
                                              double irho, double lrho, double distance, Walk<N>& k,
                                              double& ratio, double& tau, double (&g)[N], bool& ok) {
  if (!(distance > 1e-8)) {  // no step (the same for the whole warp): nothing of the cell enters
#pragma unroll
    for (int n = 0; n < N; ++n) {
      k.dE[n] = n == 0 ? 1.0 : 0.0;
      g[n] = 0.0;
    }
    return;
  }
  begin(tb, m, k);
  const double iS0 = f64::rcp(k.S);
  double g0[N], drem[N];
#pragma unroll
  for (int n = 0; n < N; ++n) {
    g0[n] = k.dS[n] * iS0;
    drem[n] = 0.0;
  }
  double rem = distance;
  for (int guard = 0;; ++guard) {
    bool on = ok && f64::lt_pos(1e-8, rem);
    if (!__any_sync(0xffffffffu, on)) break;
    if (on && (guard > 10000000 || !positive_finite(k.S))) on = ok = false;
    double rel[N], dds[N], dgx[N];
    const double gl = gain_limit(k, 1e-6, rel), c = gl * irho;
    const bool whole = !f64::lt_pos(wt::kMaxStep, rem);
    const double len = whole ? rem : wt::kMaxStep;
    const bool gain = f64::lt_pos(c, len);  // the energy gain limits the step
    const double ds = gain ? c : len, gx = gain ? gl : len * rho;
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const double r = n == 1 ? rel[n] - lrho : rel[n];
      dds[n] = gain ? ds * r : (whole ? drem[n] : 0.0);
      dgx[n] = n == 1 ? fma(dds[n], rho, gx * lrho) : dds[n] * rho;
    }
    Walk<N> next = k;
    const bool valid = heun(tb, R, m, next, ds, gx, dds, dgx);
    if (on && !valid) on = ok = false;
    if (on) {
      k = next;
      rem -= ds;
#pragma unroll
      for (int n = 0; n < N; ++n) drem[n] -= dds[n];
    }
    __syncwarp();
  }
  finish(k, R, iS0, g0, ratio, tau, g);
}

// propagate_csda_air_segment (:516-551).  Nearly all steps are the 60 m limit
// of every lane, with no tangent in their length: the density at the middle of
// such a step then serves both the limit and the step, it follows from the last
// one by a constant factor (anew from the altitude every 8 steps, so that the
// factors' rounding stays below that of the exponential), and neither the gain
// limit nor any tangent of length or density is formed.
__device__ __forceinline__ void air_segment(const Tables& tb, const Run& R, double base, double cos_t,
                                            double distance, Walk<1>& k, double& ratio, double& tau,
                                            double (&g)[1], bool& ok) {
  const OneMaterial m{tb.c[wt::A_CS], tb.d[D_A]};
  begin(tb, m, k);
  const double iS0 = f64::rcp(k.S), g0[1] = {k.dS[0] * iS0};
  const double b0 = base * (-1.0 / 12e3), c0 = cos_t * (-1.0 / 12e3);
  const double fall = f64::exp(c0 * wt::kMaxStep);  // density ratio of 60 m
  double rem = distance, trav = 0.0, dtrav = 0.0, rho = 0.0;
  int run = 0;  // steps since the density was formed from the altitude
  for (int guard = 0;; ++guard) {
    bool on = ok && f64::lt_pos(1e-8, rem);
    if (!__any_sync(0xffffffffu, on)) break;
    if (on && (guard > 10000000 || !positive_finite(k.S))) on = ok = false;
    const bool whole = !f64::lt_pos(wt::kMaxStep, rem);
    double ds = whole ? rem : wt::kMaxStep, dds[1] = {0.0}, dgx[1] = {0.0};
    const bool chain = run > 0 && run < 8 && !__any_sync(0xffffffffu, on && whole);
    rho = chain ? rho * fall : 1.205 * f64::exp(fma(c0, fma(0.5, ds, trav), b0));
    run = chain ? run + 1 : 1;
    double gx = ds * rho;
    // grel / rho < ds: the energy gain limits the step
    const bool gain = wt::kMaxGain * f64::max_pos(k.E, 1e-6) < k.S * (f64::max_pos(rho, 1e-12) * ds);
    const bool varies = gain || (whole && f64::lt_pos(ds, 1e-3)) || dtrav != 0.0;
    if (__any_sync(0xffffffffu, on && varies)) {
      double rel[1], drho;
      const double gl = gain_limit(k, 0.0, rel);
      dds[0] = whole ? -dtrav : 0.0;
      if (gain) {
        const bool thin = f64::lt_pos(rho, 1e-12);
        const double ir = f64::rcp(thin ? 1e-12 : rho);
        drho = rho * (c0 * fma(0.5, dds[0], dtrav));
        ds = gl * ir;
        dds[0] = ds * (rel[0] - (thin ? 0.0 : drho * ir));
      }
      if (f64::lt_pos(ds, 1e-3)) {
        ds = 1e-3;
        dds[0] = 0.0;
      }
      rho = 1.205 * f64::exp(fma(c0, fma(0.5, ds, trav), b0));
      drho = rho * (c0 * fma(0.5, dds[0], dtrav));
      gx = ds * rho;
      dgx[0] = fma(dds[0], rho, ds * drho);
      run = 0;
    }
    __syncwarp();
    Walk<1> next = k;
    const bool valid = heun(tb, R, m, next, ds, gx, dds, dgx);
    if (on && !valid) on = ok = false;
    if (on) {
      k = next;
      trav += ds;
      dtrav += dds[0];
      rem -= ds;
    }
    __syncwarp();
  }
  finish(k, R, iS0, g0, ratio, tau, g);
}

// cell_density (:303-310): density, its inverse and d log rho / d w, and the
// cell's stopping power.
struct CellMedium {
  CellMix S;
  double rho, irho, lrho;
};
__device__ __forceinline__ CellMedium cell_medium(const Params& P, const Tables& tb, int cell) {
  CellMedium c;
  const bool porous = wt::cell_porous(P, cell);
  c.S = CellMix{tb.c[wt::R_CS], tb.d[D_R], tb.c[wt::W_CS], tb.d[D_W],
                porous ? tb.c[wt::P_CS] : nullptr, tb.d[D_P], P.wf[cell]};
  double drho;
  c.rho = wt::density64(P, cell, &drho);
  c.irho = f64::rcp(c.rho);
  c.lrho = drho * c.irho;
  return c;
}
// Straggling and hard-loss increments of a segment of grammage gx at its mean
// energy (src/Tomography.jl:598-617), with tangents.
template <int N>
__device__ __forceinline__ void vh_increments(const Tables& tb, const double* qS, const double* qM,
                                              const double* qT, const double* pS, const double* pM,
                                              const double* pT, double w, double gx, double lgx,
                                              double E_in, const Walk<N>& k, double& v, double& h,
                                              double (&dv)[N], double (&dh)[N]) {
  const double e = 0.5 * (E_in + k.E);
  const Pos o = locate(tb, e, k.i);
  const Val s = mix_at(tb.c[wt::R_ST], qT, pT, w, o);
  const Val a = mix_at(tb.c[wt::R_CS], qS, pS, w, o), b = mix_at(tb.c[wt::R_MS], qM, pM, w, o);
  const double ie = f64::rcp(e);
  v = s.v * gx;
  h = (a.v - b.v) * gx;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    const double de = 0.5 * ((n == 0 ? 1.0 : 0.0) + k.dE[n]) * ie;
    dv[n] = (s.sl * de + (n == 1 ? s.sw : 0.0)) * gx + (n == 1 ? v * lgx : 0.0);
    dh[n] = ((a.sl - b.sl) * de + (n == 1 ? a.sw - b.sw : 0.0)) * gx + (n == 1 ? h * lgx : 0.0);
  }
}
template <int N>
__device__ __forceinline__ void vh_cell(const Params& P, const Tables& tb, const CellMedium& c, double len,
                                        double E_in, const Walk<N>& k, double& v, double& h,
                                        double (&dv)[N], double (&dh)[N]) {
  const bool p = c.S.p != nullptr;
  vh_increments(tb, tb.c[wt::W_CS], tb.c[wt::W_MS], tb.c[wt::W_ST], p ? tb.c[wt::P_CS] : nullptr,
                p ? tb.c[wt::P_MS] : nullptr, p ? tb.c[wt::P_ST] : nullptr, c.S.w, len * c.rho, c.lrho,
                E_in, k, v, h, dv, dh);
}

// Running sums over the segments of a path: the prefix product of dE_out/dE_in
// and the energy derivatives of the log weight, V and H referred to the start.
struct Sums {
  double P = 1.0, s = 0.0, v = 0.0, h = 0.0;
  __device__ __forceinline__ void add(double dg, double dv, double dh, double dE) {
    s = fma(dg, P, s);
    v = fma(dv, P, v);
    h = fma(dh, P, h);
    P *= dE;
  }
};

// Pass 1: flux of one sample and its end-of-path adjoint constants (zeros where
// the walk is invalid or the lane has no sample: ok false).
static __device__ __noinline__ Lane pass1(const Params& P, const Run& R, const Tables& tb, long b,
                                          double E0, double q, bool ok) {
  Lane out{0.0, 0.0, 0.0, 0.0};
  const double ct = P.cos_t[b];
  Walk<1> k;
  k.E = E0;
  k.i = first_interval(tb, E0);
  double ratio = 1.0, tau = 0.0, V = 0.0, H = 0.0, g[1];
  Sums S;
  const int64_t s0 = P.seg_ptr[b], s1 = P.seg_ptr[b + 1];
  for (int64_t j = s0; j < s1; ++j) {
    const CellMedium c = cell_medium(P, tb, P.seg_cell[j]);
    const double len = P.seg_len[j], E_in = k.E;
    solid_segment(tb, R, c.S, c.rho, c.irho, 0.0, len, k, ratio, tau, g, ok);
    // (a NaN length, which takes no step, leaves the path without a Jacobian)
    double v = 0.0, h = 0.0, dv[1] = {0.0 * len}, dh[1] = {0.0};
    if (P.corr) vh_cell(P, tb, c, len, E_in, k, v, h, dv, dh);
    S.add(g[0], dv[0], dh[0], k.dE[0]);
    V += v;
    H += h;
  }
  if (P.rem[b] > 1e-8) {
    const OneMaterial m{tb.c[wt::R_CS], tb.d[D_R]};
    const double E_in = k.E;
    solid_segment(tb, R, m, P.rho_rock, f64::rcp(P.rho_rock), 0.0, P.rem[b], k, ratio, tau, g, ok);
    double v = 0.0, h = 0.0, dv[1] = {0.0}, dh[1] = {0.0};
    if (P.corr)  // rock alone: no water in the mix
      vh_increments(tb, tb.c[wt::R_CS], tb.c[wt::R_MS], tb.c[wt::R_ST], nullptr, nullptr, nullptr, 0.0,
                    P.rem[b] * P.rho_rock, 0.0, E_in, k, v, h, dv, dh);
    S.add(g[0], dv[0], dh[0], k.dE[0]);
    V += v;
    H += h;
  }
  {
    const double air = fmax(0.0, P.primary - P.exit_z[b]) / fmax(ct, 1e-3);
    air_segment(tb, R, P.det_elev + P.exit_z[b], ct, air, k, ratio, tau, g, ok);
    S.add(g[0], 0.0, 0.0, k.dE[0]);
  }
  if (!ok) return out;
  const double cs = cos_theta_star(ct), cs129 = pow(cs, 1.29), E = k.E;
  double dlogF;
  const double F = gccly_flux(cs, cs129, E, q, &dlogF);
  double corr = 1.0, dcorr = 0.0;
  if (P.corr) {
    // csda_var_correction (:384-391)
    const double e = fmax(E, 1.0);
    double bi, dbi;
    wt::spectral_index(e, cs, cs129, &bi, &dbi);
    const double cstr = 0.5 * bi * (bi + 1.0), Hp = fmax(H, 0.0);
    corr = exp(P.ks * cstr * V / (e * e) - P.kh * Hp / e);
    out.aV = P.ks * cstr / (e * e);
    out.aH = H > 0.0 ? -P.kh / e : 0.0;
    if (E > 1.0)
      dcorr = P.ks * V * ((bi + 0.5) * dbi / (e * e) - 2.0 * cstr / (e * e * e)) + P.kh * Hp / (e * e);
  }
  out.f = ratio * exp(-tau * R.inv_ctau) * corr * F;
  out.A = (dlogF + dcorr) * S.P + S.s + out.aV * S.v + out.aH * S.h;
  return out;
}

__global__ void __launch_bounds__(kThreads) wtomo_kernel(const __grid_constant__ Params P) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
  double* cols = reinterpret_cast<double*>(smem + 16);
  if (!stage_columns(cols, P.col, P.staged, P.col_bytes, bar, P.wait_iters)) {
    if (threadIdx.x == 0) atomicExch(P.err_flag, 1);
    return;
  }
  const int ld = int(P.col_bytes / 8), n = P.tv.n, lane = threadIdx.x;
  Tables tb;
#pragma unroll
  for (int s = 0; s < wt::kSlots; ++s)
    tb.c[s] = s < wt::kWalkSlots || P.staged == wt::kSlots ? cols + size_t(s) * ld : P.col[s];
  double* der = cols + size_t(P.staged) * ld;
#pragma unroll
  for (int s = 0; s < kDerived; ++s) tb.d[s] = der + size_t(s) * ld;
  for (int i = lane; i < n - 1; i += kThreads) {
    auto diff = [&](int s) { return cols[size_t(s) * ld + i + 1] - cols[size_t(s) * ld + i]; };
    der[size_t(D_INV) * ld + i] = 1.0 / diff(wt::S_LE);
    der[size_t(D_R) * ld + i] = diff(wt::R_CS);
    der[size_t(D_W) * ld + i] = diff(wt::W_CS);
    der[size_t(D_P) * ld + i] = diff(wt::P_CS);
    der[size_t(D_A) * ld + i] = diff(wt::A_CS);
  }
  __syncwarp();
  tb.n = n;
  tb.lo = __double_as_longlong(cols[size_t(wt::S_E) * ld]);
  tb.hi = __double_as_longlong(cols[size_t(wt::S_E) * ld + n - 1]);
  const Run R{0.5 / P.mass, 1.0 / P.ctau};
  const int n_chunks = (P.n_e + 31) / 32;
  // bins are handed out one at a time as warps finish (path lengths differ widely)
  auto next_bin = [&]() -> long {
    unsigned long long v = 0;
    if (lane == 0) v = atomicAdd(P.next_bin, 1ull);
    return long(__shfl_sync(0xffffffffu, v, 0));
  };
  for (long b = next_bin(); b < P.n_bins; b = next_bin()) {
    const int64_t s0 = P.seg_ptr[b], s1 = P.seg_ptr[b + 1];
    const double ct = P.cos_t[b];
    // device-array calls: cells outside the water-fraction vector end the call
    bool bad = false;
    for (int64_t j = s0 + lane; j < s1; j += 32) bad |= P.seg_cell[j] < 0 || P.seg_cell[j] >= P.n_cells;
    if (__any_sync(0xffffffffu, bad)) {
      if (lane == 0) {
        P.flux[b] = CUDART_NAN;
        atomicExch(P.err_flag, 3);
      }
      continue;
    }
    if ((P.valid && !P.valid[b]) || !(ct > 0.0)) {
      if (lane == 0) P.flux[b] = CUDART_NAN;
      if (P.jac)
        for (int64_t j = s0 + lane; j < s1; j += 32) P.jac[j] = 0.0;
      continue;
    }
    Lane L[kMaxChunks];
    double sum = 0.0;
#pragma unroll
    for (int ch = 0; ch < kMaxChunks; ++ch) {
      L[ch] = Lane{0.0, 0.0, 0.0, 0.0};
      const int s = ch * 32 + lane;
      if (ch < n_chunks) {
        const bool in = s < P.n_e;
        L[ch] = pass1(P, R, tb, b, in ? P.E[s] : 1.0, in ? P.q[s] : 0.0, in);
        L[ch].f *= in ? 2.0 * P.ew[s] : 0.0;
      }
      sum += L[ch].f;
    }
    sum = wt::warp_sum(sum);
    // geometric and material multipliers (:405-412, :557-579)
    double Lsum = 0.0, water = 0.0, mass = 0.0;
    for (int64_t j = s0 + lane; j < s1; j += 32) {
      const int cell = P.seg_cell[j];
      const double gx = P.seg_len[j] * wt::density64(P, cell);
      Lsum += P.seg_len[j];
      water += P.wf[cell] * gx;
      mass += gx;
    }
    Lsum = wt::warp_sum(Lsum);
    water = wt::warp_sum(water);
    mass = wt::warp_sum(mass) + P.rem[b] * P.rho_rock;
    double G = 1.0;
    if (P.corr && (P.ra != 0.0 || P.rb != 0.0 || P.rc != 0.0 || P.rd != 0.0)) {
      const double lL = log(fmax(P.rem[b] + Lsum, 1.0));
      G = exp(P.ra + P.rb * lL + P.rc * lL * lL + P.rd * ct);
    }
    const double qf = water / fmax(mass, 1e-30);
    const double M = P.mcorr ? exp(P.lin * qf + P.quad * qf * qf) : 1.0;
    const double flux = G * M * sum / double(P.n_e);
    if (lane == 0) P.flux[b] = flux;
    if (!P.jac) continue;

    // pass 2: d log f / d w per cell segment, summed over the samples
    const double scale = G * M / double(P.n_e);
    for (int ch = 0; ch < n_chunks; ++ch) {
      const int s = ch * 32 + lane;
      const Lane& l = L[ch];
      bool ok = s < P.n_e && l.f != 0.0;
      Walk<2> k;
      k.E = ok ? P.E[s] : 1.0;
      k.i = first_interval(tb, k.E);
      double ratio = 1.0, tau = 0.0;
      Sums S;
      for (int64_t j = s0; j < s1; ++j) {
        const CellMedium c = cell_medium(P, tb, P.seg_cell[j]);
        const double len = P.seg_len[j], E_in = k.E;
        double g[2], v, h, dv[2] = {0.0, 0.0}, dh[2] = {0.0, 0.0};
        solid_segment(tb, R, c.S, c.rho, c.irho, c.lrho, len, k, ratio, tau, g, ok);
        if (P.corr) vh_cell(P, tb, c, len, E_in, k, v, h, dv, dh);
        S.add(g[0], dv[0], dh[0], k.dE[0]);
        const double lam = f64::div(l.A - S.s - l.aV * S.v - l.aH * S.h, S.P);
        // not ok: no sample or flux, or (not reached) an invalid walk
        double gk = ok ? l.f * (lam * k.dE[1] + g[1] + l.aV * dv[1] + l.aH * dh[1]) : 0.0;
        gk = wt::warp_sum(gk);
        if (lane == 0) P.jac[j] = (ch ? P.jac[j] : 0.0) + scale * gk;
      }
    }
    // d M / d w through the column water fraction q (:557-579)
    if (P.mcorr) {
      const double dlogM = P.lin + 2.0 * P.quad * qf, mm = fmax(mass, 1e-30);
      __syncwarp();
      for (int64_t j = s0 + lane; j < s1; j += 32) {
        const int cell = P.seg_cell[j];
        double dgx;
        const double gx = P.seg_len[j] * wt::density64(P, cell, &dgx);
        dgx *= P.seg_len[j];
        const double dwater = gx + P.wf[cell] * dgx;
        const double dq = mass > 1e-30 ? (dwater * mm - water * dgx) / (mm * mm) : dwater / mm;
        P.jac[j] += flux * dlogM * dq;
      }
    }
  }
}

}  // namespace wt64
}  // namespace dp
