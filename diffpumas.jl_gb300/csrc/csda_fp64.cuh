// csda_fp64.cuh -- the FP64 CSDA histories of run_backward_mc
// (straggling = scattering = false) with their density tangent, in two forms of
// one step program (src/Geometry.jl:534-672 with transport_backward_step,
// :424-457, and the step limit, :461-476).
//
// FP64 warp instructions bound both (one per 64 cycles and SM partition, with
// one lane active as with 32), and a history is a chain of 10^2-10^3 dependent
// steps.  A step costs one exponential and one reciprocal square root: the range
// at its end is carried into the next one (the reference recomputes it from the
// energy: R(K(Y)) = Y to rounding), the stopping-power ratios of consecutive
// steps in one material telescope, the decay factors multiply to
// exp(-sum dt / c tau), and tangents are written out.
//
//  - csda_thread_kernel, one history per lane: the fewest instructions per
//    history where there are histories for every lane of the chip.
//  - csda_warp_kernel, one history per warp: up to 32 steps of it at once.  In
//    the rock the step limit is 1 % of the range, so the ranges of the next
//    steps are X 1.01^j and their altitudes follow; in the air at the altitude
//    limit the steps have one length, and the ranges are prefix sums of the
//    densities; in between (thin air, low energy) only the altitudes form a
//    chain.  Each lane then inverts one step's range and forms its flight time.
//    The lanes commit up to the first step that the reference would have cut
//    otherwise (a boundary, the energy ceiling, a table end), which all lanes
//    then take as one ordinary step.
//
// Every branch the reference takes is the same, and the results agree with its
// operation-by-operation program to rounding (~1e-13).  compute_flux_gradient
// of one history 0.95 -> 0.11 ms, 10^4 histories of 1-100 GeV through 100 m at
// 45 deg 2.72 -> 0.79 ms, 10^5 13.4 -> 6.0 ms; 10^5 through 5 m (by thread) 5.9
// -> 3.9 ms, host copies included.

enum { S_E = 0, S_LOGE, S_RS, S_RR, S_AS, S_AR, S_NCOL };
enum { D_RINV = 0, D_RSLO, D_AINV, D_ASLO, D_NCOL };
constexpr int kCsdaThreads = 128;

// One material's columns: range, stopping power, 1 / dR and d log E / d R per
// interval.
struct CsdaMat {
  const double *R, *S, *rinv, *slo;
};
struct CsdaTables {
  const double *E, *lE;
  CsdaMat mat[2];  // rock, air
  int n;
};
struct CsdaConst {
  double ceiling;     // threshold - eps
  double half_inv_m;
  int cap;
};

// Geometry of a history as its steps use it.
struct CsdaWalk {
  double thick, rho, top, rock_top;  // top: H - eps; rock_top: the rock ends there or at H
  double H, uz, inv_uz, air_limit;
  double c, cd, irho;      // rock step limit per range and its tangent, 1 / rho
};
__device__ __forceinline__ CsdaWalk csda_walk(double thick, double rho, double H, double uz, double air_limit) {
  CsdaWalk w;
  w.thick = thick;
  w.rho = rho;
  w.H = H;
  w.top = H - kEps64;
  w.rock_top = w.top < thick ? w.top : thick;
  w.uz = uz;
  w.air_limit = air_limit;
  w.inv_uz = uz > kEps64 || uz < -kEps64 ? 1.0 / uz : 0.0;
  const bool thin = !(rho >= 1e-6);  // max(rho, 1e-6)
  w.irho = 1.0 / (thin ? 1e-6 : rho);
  w.c = 0.01 * w.irho;
  w.cd = thin ? 0.0 : -w.c * w.irho;
  return w;
}

// A history: energy, range, altitude and proper time with their tangents, the
// weight of the materials it has left and the stopping power at the entry of
// its present one (m: 0 rock, 1 air, -1 none yet), its energy interval and
// whether the energy is clamped at a table end (edge).
struct CsdaHist {
  double E, Ed, X, Xd, z, zd, tau, taud, w, wd, S0, S0d;
  int m, i, edge, steps;
};
__device__ __forceinline__ void csda_start(CsdaHist& h, double E0) {
  h.E = E0;
  h.Ed = h.X = h.Xd = h.z = h.zd = h.tau = h.taud = h.wd = h.S0d = 0.0;
  h.w = h.S0 = 1.0;
  h.m = -1;
  h.i = h.edge = h.steps = 0;
}
// Weight factor S(here) / S(entry) of the present material.
__device__ __forceinline__ void csda_leave(const CsdaTables& T, CsdaHist& h) {
  if (h.m < 0) return;
  const CsdaMat& M = T.mat[h.m];
  double S, Sd = 0.0;
  if (h.edge) {
    S = M.S[h.edge < 0 ? 0 : T.n - 1];
  } else {
    const double d = (M.S[h.i + 1] - M.S[h.i]) * M.rinv[h.i];
    S = fma(h.X - M.R[h.i], d, M.S[h.i]);
    Sd = d * h.Xd;
  }
  const double q = S / h.S0, qd = (Sd - q * h.S0d) / h.S0;
  h.wd = fma(h.wd, q, h.w * qd);
  h.w *= q;
}
// Enters material m: its range and stopping power at the present energy,
// log-linear on the shared energy grid (src/Physics.jl:660-687).
__device__ __forceinline__ void csda_enter(const CsdaParams& P, const CsdaTables& T, CsdaHist& h, int m) {
  csda_leave(T, h);
  const CsdaMat& M = T.mat[m];
  double t, td = 0.0;
  if (h.m < 0) {
    t = 0.0;
    h.edge = h.E <= T.E[0] ? -1 : (h.E >= T.E[T.n - 1] ? 1 : 0);
    if (!h.edge) {
      const double lE = f64::log(h.E);
      h.i = P.tab.uniform ? uniform_interval(T.lE, T.n, lE, P.tab.lE0, P.tab.inv_dlE) : bisect(T.lE, T.n, lE);
      t = (lE - T.lE[h.i]) / (T.lE[h.i + 1] - T.lE[h.i]);
    } else {
      h.i = h.edge < 0 ? 0 : T.n - 2;
    }
  } else {
    const CsdaMat& O = T.mat[h.m];
    t = (h.X - O.R[h.i]) * O.rinv[h.i];
    td = O.rinv[h.i] * h.Xd;
  }
  h.m = m;
  if (h.edge) {
    const int j = h.edge < 0 ? 0 : T.n - 1;
    h.X = M.R[j];
    h.S0 = M.S[j];
    h.Xd = h.S0d = 0.0;
  } else {
    const double dR = M.R[h.i + 1] - M.R[h.i], dS = M.S[h.i + 1] - M.S[h.i];
    h.X = fma(t, dR, M.R[h.i]);
    h.S0 = fma(t, dS, M.S[h.i]);
    h.Xd = dR * td;
    h.S0d = dS * td;
  }
}
// Interval of the range Y inside (R[0], R[n-1]), walking from i.
__device__ __forceinline__ int csda_interval(const double* R, int n, double Y, int i) {
  while (i < n - 2 && !f64::lt_pos(Y, R[i + 1])) ++i;
  while (i > 0 && f64::lt_pos(Y, R[i])) --i;
  return i;
}
__device__ __forceinline__ bool csda_on(const CsdaConst& C, const CsdaWalk& W, const CsdaHist& h) {
  return h.steps < C.cap && h.E < C.ceiling && !(h.z < 0.0) && h.z < W.top;
}
// Distance to the boundary ahead of altitude z.
__device__ __forceinline__ double csda_ahead(const CsdaWalk& W, bool air, double z) {
  const double to = air ? (W.inv_uz > 0.0 ? W.H : W.thick) : (W.inv_uz > 0.0 ? W.thick : 0.0);
  return W.inv_uz != 0.0 ? (to - z) * W.inv_uz : 1000.0;
}

// One step of the reference's program.
__device__ __forceinline__ void csda_step(const CsdaParams& P, const CsdaTables& T, const CsdaConst& C,
                                          const CsdaWalk& W, CsdaHist& h) {
  const int m = h.z >= W.thick ? 1 : 0;
  if (m != h.m) csda_enter(P, T, h, m);
  const CsdaMat& M = T.mat[m];
  const double ahead = csda_ahead(W, m != 0, h.z);
  double dens, densd, lim, limd;
  if (m == 0) {
    dens = W.rho;
    densd = 1.0;
    lim = h.X * W.c;
    limd = fma(h.Xd, W.c, h.X * W.cd);
  } else {
    dens = 1.205 * f64::exp(h.z * (-1.0 / 12e3));
    densd = dens * (-1.0 / 12e3) * h.zd;
    const bool thin = dens < 1e-6;
    const double inv = f64::rcp(thin ? 1e-6 : dens);
    lim = 0.01 * h.X * inv;
    limd = inv * fma(thin ? 0.0 : -lim, densd, 0.01 * h.Xd);
    if (W.air_limit < lim) {
      lim = W.air_limit;
      limd = 0.0;
    }
  }
  double step = ahead + 1e-7, stepd = -h.zd * W.inv_uz;
  if (lim < step) {
    step = lim;
    stepd = limd;
  }
  if (step < kStepMin || step > 1000.0) {
    step = step < kStepMin ? kStepMin : 1000.0;
    stepd = 0.0;
  }
  // inverse range at Y (src/Physics.jl:833-867), clamped at the table ends
  const double Y = fma(step, dens, h.X), Yd = fma(step, densd, fma(stepd, dens, h.Xd));
  double En, End = 0.0;
  if (Y <= M.R[0]) {
    h.i = 0;
    h.edge = -1;
    En = T.E[0];
  } else if (Y >= M.R[T.n - 1]) {
    h.i = T.n - 2;
    h.edge = 1;
    En = T.E[T.n - 1];
  } else {
    h.i = csda_interval(M.R, T.n, Y, h.i);
    h.edge = 0;
    const double slo = M.slo[h.i];
    En = f64::exp(fma(Y - M.R[h.i], slo, T.lE[h.i]));
    End = En * slo * Yd;
  }
  // proper time of the step at the mean Lorentz factor
  double dib;
  const double ib = f64::inv_beta_gamma((h.E + En) * C.half_inv_m, &dib);
  h.tau = fma(step, ib, h.tau);
  h.taud += fma(stepd, ib, step * dib * ((h.Ed + End) * C.half_inv_m));
  h.z = fma(step, W.uz, h.z);
  h.zd = fma(stepd, W.uz, h.zd);
  h.X = Y;
  h.Xd = Yd;
  h.E = En;
  h.Ed = End;
  ++h.steps;
}

// Weight and acceptance of an ended history: w * flux and its tangent.
__device__ __forceinline__ void csda_flux(const CsdaParams& P, const CsdaConst& C, const CsdaGeo& G,
                                          const CsdaHist& h, double q, double w, double* f, double* df) {
  const double e = exp(-h.tau / P.ctau), v = h.w * e, vd = e * (h.wd - h.w * h.taud / P.ctau);
  *f = *df = 0.0;
  if (h.steps >= C.cap) {
    atomicExch(P.err_flag, 4);
  } else if (h.z >= G.H - 1.0 && h.E < P.threshold && G.cos_final > 0.0) {
    double dlogf;
    const double F = gccly_flux(G.cs, G.cs129, h.E, q, &dlogf);
    *f = w * (v * F);
    *df = w * (vd * F + v * F * dlogf * h.Ed);
  }
}

// Start of history i: its geometry and sample.
__device__ __forceinline__ CsdaGeo csda_sample(const CsdaParams& P, long i, double* E0, double* q, double* w) {
  CsdaGeo G = P.geo;
  if (P.los) {
    long lo = 0, hi = P.n_los;
    while (hi - lo > 1) {
      const long mid = (lo + hi) >> 1;
      if (P.los_off[mid] <= i) lo = mid; else hi = mid;
    }
    const dp_los& L = P.los[lo];
    const double H = L.air_height > 0.0 ? L.thickness + L.air_height
                                        : (L.primary_altitude > 0.0 ? L.primary_altitude : 3e4);
    G = csda_geo(L.thickness, L.density, L.elevation, H);
    mc_sample(P.seed, uint64_t(i), L.energy_min, L.energy_max > L.energy_min ? L.energy_max : L.energy_min, E0,
              q, w);
  } else if (P.use_philox) {
    mc_sample(P.seed, uint64_t(i), P.emin, P.emax, E0, q, w);
  } else {
    *E0 = P.E[i];
    *q = P.q[i];
    *w = P.w[i];
  }
  return G;
}

// Stages the columns and derives the per-interval ones; false when the staging
// wait gave up.
__device__ __forceinline__ bool csda_tables(const CsdaParams& P, double* smem, uint64_t* mbar, CsdaTables& T) {
  const int ld = P.tab.ld, n = P.tab.n;
  const double* src[S_NCOL] = {P.tab.col(0, DP_COL_E),          P.tab.col(0, DP_COL_LOGE),
                               P.tab.col(P.rock, DP_COL_CSDA_S), P.tab.col(P.rock, DP_COL_CSDA_R),
                               P.tab.col(P.air, DP_COL_CSDA_S),  P.tab.col(P.air, DP_COL_CSDA_R)};
  if (!stage_columns(smem, src, S_NCOL, uint32_t(ld * sizeof(double)), mbar, P.wait_iters)) {
    if (threadIdx.x == 0) atomicExch(P.err_flag, 1);
    return false;
  }
  double* der = smem + S_NCOL * ld;
  T.E = smem + S_E * ld;
  T.lE = smem + S_LOGE * ld;
  T.n = n;
  T.mat[0] = CsdaMat{smem + S_RR * ld, smem + S_RS * ld, der + D_RINV * ld, der + D_RSLO * ld};
  T.mat[1] = CsdaMat{smem + S_AR * ld, smem + S_AS * ld, der + D_AINV * ld, der + D_ASLO * ld};
  for (int k = threadIdx.x; k < n - 1; k += blockDim.x) {
    const double dle = T.lE[k + 1] - T.lE[k];
    const double r = 1.0 / (T.mat[0].R[k + 1] - T.mat[0].R[k]), a = 1.0 / (T.mat[1].R[k + 1] - T.mat[1].R[k]);
    der[D_RINV * ld + k] = r;
    der[D_RSLO * ld + k] = dle * r;
    der[D_AINV * ld + k] = a;
    der[D_ASLO * ld + k] = dle * a;
  }
  __syncthreads();
  return true;
}
__device__ __forceinline__ CsdaConst csda_const(const CsdaParams& P) {
  return CsdaConst{P.threshold - kEps64, 0.5 / P.mass, P.step_cap};
}

__global__ void __launch_bounds__(kCsdaThreads) csda_thread_kernel(CsdaParams P) {
  extern __shared__ __align__(16) double smem[];
  __shared__ uint64_t mbar;
  CsdaTables T;
  if (!csda_tables(P, smem, &mbar, T)) return;
  const CsdaConst C = csda_const(P);
  const long stride = long(gridDim.x) * blockDim.x;
  // warp-uniform loop: the lanes of a warp step together
  for (long i0 = blockIdx.x * long(blockDim.x) + (threadIdx.x & ~31); i0 < P.n; i0 += stride) {
    const long i = i0 + (threadIdx.x & 31);
    const bool in = i < P.n;
    double E0, q, w;
    const CsdaGeo G = csda_sample(P, in ? i : i0, &E0, &q, &w);
    const CsdaWalk W = csda_walk(G.thickness, G.rho, G.H, G.uz, G.air_limit);
    CsdaHist h;
    csda_start(h, E0);
    for (;;) {
      const bool on = in && csda_on(C, W, h);
      if (!__any_sync(0xffffffffu, on)) break;
      if (on) csda_step(P, T, C, W, h);
      __syncwarp();
    }
    csda_leave(T, h);
    double f, df;
    if (in) {
      csda_flux(P, C, G, h, q, w, &f, &df);
      P.contrib[i] = f;
      if (P.dcontrib) P.dcontrib[i] = df;
      if (P.steps) P.steps[i] = h.steps;
    }
    __syncwarp();
  }
}

// The warp form's batch: lane j holds step j (from altitude z, length `step`,
// end range Y).  Commits the leading run of steps for which `fits` holds (the
// step's limit and length are the batch's, it starts in the batch's medium and
// ends inside the table) and which start below the energy ceiling; returns
// their number.  zn, znd: altitude after the step.
__device__ __forceinline__ int csda_commit(const CsdaTables& T, const CsdaConst& C, CsdaHist& h, int lane,
                                           bool fits, double step, double stepd, double Y, double Yd, double zn,
                                           double znd, double& tau, double& taud) {
  const CsdaMat& M = T.mat[h.m];
  fits = fits && f64::lt_pos(M.R[0], Y) && f64::lt_pos(Y, M.R[T.n - 1]) && h.steps + lane < C.cap;
  const double Yc = fits ? Y : h.X;  // a lane past the run repeats the start
  const int i = csda_interval(M.R, T.n, Yc, h.i);
  __syncwarp();
  const double slo = M.slo[i], En = f64::exp(fma(Yc - M.R[i], slo, T.lE[i])), End = En * slo * Yd;
  double E = __shfl_up_sync(0xffffffffu, En, 1), Ed = __shfl_up_sync(0xffffffffu, End, 1);
  if (lane == 0) {
    E = h.E;
    Ed = h.Ed;
  }
  fits = fits && E < C.ceiling;
  const unsigned ok = __ballot_sync(0xffffffffu, fits);
  const int k = ok == 0xffffffffu ? 32 : __ffs(~ok) - 1;
  if (k == 0) return 0;
  double dib;
  const double ib = f64::inv_beta_gamma((E + En) * C.half_inv_m, &dib);
  if (lane < k) {
    tau = fma(step, ib, tau);
    taud += fma(stepd, ib, step * dib * ((Ed + End) * C.half_inv_m));
  }
  const int from = k - 1;
  h.E = __shfl_sync(0xffffffffu, En, from);
  h.Ed = __shfl_sync(0xffffffffu, End, from);
  h.X = __shfl_sync(0xffffffffu, Y, from);
  h.Xd = __shfl_sync(0xffffffffu, Yd, from);
  h.z = __shfl_sync(0xffffffffu, zn, from);
  h.zd = __shfl_sync(0xffffffffu, znd, from);
  h.i = __shfl_sync(0xffffffffu, i, from);
  h.edge = 0;
  h.steps += k;
  return k;
}
// Whether a step of length s at altitude z is cut by nothing but its limit.
__device__ __forceinline__ bool csda_free(const CsdaWalk& W, bool air, double z, double s) {
  return s < csda_ahead(W, air, z) + 1e-7 && s >= kStepMin && s <= 1000.0 && z >= (air ? W.thick : 0.0) &&
         z < (air ? W.top : W.rock_top);
}

__global__ void __launch_bounds__(kCsdaThreads) csda_warp_kernel(CsdaParams P, int group) {
  extern __shared__ __align__(16) double smem[];
  __shared__ uint64_t mbar;
  CsdaTables T;
  if (!csda_tables(P, smem, &mbar, T)) return;
  const CsdaConst C = csda_const(P);
  const int lane = threadIdx.x & 31;
  const double2 p0 = f64::kPow101[lane], p1 = f64::kPow101[lane + 1];
  const double jd = f64::from_int(lane), air_k = -1.0 / 12e3;
  const long warps = long(gridDim.x) * (blockDim.x >> 5);
  // groups of `group` histories, neighbouring warps on different SMs
  for (long b = (long(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * group; b < P.n; b += warps * group) {
    const int m = int(P.n - b < group ? P.n - b : group);
    // lane l: sample and geometry of history b + l, and its end state
    const bool mine = lane < m;
    double E0, q, w;
    const CsdaGeo G = csda_sample(P, b + (mine ? lane : 0), &E0, &q, &w);
    CsdaHist end;
    csda_start(end, E0);
    for (int l = 0; l < m; ++l) {
      auto get = [&](double v) { return __shfl_sync(0xffffffffu, v, l); };
      const CsdaWalk W = csda_walk(get(G.thickness), get(G.rho), get(G.H), get(G.uz), get(G.air_limit));
      CsdaHist h;  // the same in every lane but for the flight time
      csda_start(h, get(E0));
      double tau = 0.0, taud = 0.0;  // this lane's share of it
      const double s_air = W.air_limit < 1000.0 ? W.air_limit : 1000.0;
      const bool dense = W.rho >= 1e-6;
      while (csda_on(C, W, h)) {
        const bool air = h.z >= W.thick;
        if (int(air) != h.m) csda_enter(P, T, h, air ? 1 : 0);
        int k = 0;
        if (!h.edge && !air && dense) {
          // ranges X 1.01^j, altitudes z + u_z (X_j - X) / rho
          const double a = W.uz * h.X * W.irho, ad = (W.uz * h.Xd - a) * W.irho;
          const double Xj = h.X * p0.x, z = fma(a, p0.y, h.z), step = Xj * W.c;
          k = csda_commit(T, C, h, lane, csda_free(W, false, z, step), step, fma(h.Xd * p0.x, W.c, Xj * W.cd),
                          h.X * p1.x, h.Xd * p1.x, fma(a, p1.y, h.z), fma(ad, p1.y, h.zd), tau, taud);
        } else if (!h.edge && air) {
          const double d0 = 1.205 * f64::exp(h.z * air_k);
          if (0.01 * h.X > s_air * (d0 < 1e-6 ? 1e-6 : d0)) {
            // steps of one length: ranges by prefix sums of the grammages
            const double z = fma(jd, s_air * W.uz, h.z), dens = 1.205 * f64::exp(z * air_k), gx = s_air * dens;
            double sum = gx;
            for (int o = 1; o < 32; o <<= 1) {
              const double v = __shfl_up_sync(0xffffffffu, sum, o);
              if (lane >= o) sum += v;
            }
            const double Y = h.X + sum;
            const bool fits = csda_free(W, true, z, s_air) && 0.01 * (Y - gx) > s_air * (dens < 1e-6 ? 1e-6 : dens);
            k = csda_commit(T, C, h, lane, fits, s_air, 0.0, Y, fma(h.zd * air_k, sum, h.Xd),
                            fma(jd + 1.0, s_air * W.uz, h.z), h.zd, tau, taud);
          } else if (d0 >= 1e-6) {
            // 1 % of the range at the local density: ranges X 1.01^j, the
            // altitudes one after the other
            double z = h.z, zd = h.zd, step = 0.0, stepd = 0.0, zn = 0.0, znd = 0.0;
            bool fits = false;
            for (int j = 0; j < 32; ++j) {
              const double2 pj = f64::kPow101[j];
              const double inv = f64::rcp(1.205 * f64::exp(z * air_k));
              const double s = 0.01 * (h.X * pj.x) * inv, sd = fma(0.01 * (h.Xd * pj.x), inv, -s * (air_k * zd));
              const bool f = s <= W.air_limit && inv <= 1e6 && csda_free(W, true, z, s);
              const double z1 = fma(s, W.uz, z), zd1 = fma(sd, W.uz, zd);
              if (j == lane) {
                fits = f;
                step = s;
                stepd = sd;
                zn = z1;
                znd = zd1;
              }
              z = z1;
              zd = zd1;
              if (!f) break;
            }
            k = csda_commit(T, C, h, lane, fits, step, stepd, h.X * p1.x, h.Xd * p1.x, zn, znd, tau, taud);
          }
        }
        if (k < 32 && csda_on(C, W, h)) csda_step(P, T, C, W, h);
        __syncwarp();
      }
      csda_leave(T, h);
      for (int o = 16; o > 0; o >>= 1) {
        tau += __shfl_xor_sync(0xffffffffu, tau, o);
        taud += __shfl_xor_sync(0xffffffffu, taud, o);
      }
      h.tau += tau;
      h.taud += taud;
      if (lane == l) end = h;
    }
    if (mine) {
      double f, df;
      csda_flux(P, C, G, end, q, w, &f, &df);
      P.contrib[b + lane] = f;
      if (P.dcontrib) P.dcontrib[b + lane] = df;
      if (P.steps) P.steps[b + lane] = end.steps;
    }
    __syncwarp();
  }
}
