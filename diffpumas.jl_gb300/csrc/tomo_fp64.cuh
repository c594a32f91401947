// tomo_fp64.cuh -- the FP64 evaluation kernel of the voxel-density tomography
// (tomo.cu): per-ray flux and, with ADJ, d flux / d density of every segment.
// One warp per ray, one lane per energy node.
//
// Bound by the FP64 pipe (one warp instruction per 64 cycles and SM partition),
// so the arithmetic per segment and lane is what this kernel is made of:
//  - the range is carried from segment to segment (the reference recomputes
//    R(E) after each inversion: R(K(Y)) = Y to rounding), so a segment costs one
//    exponential instead of three logarithms and one exponential;
//  - the stopping-power ratios telescope to S(E_N)/S(E_0) and the decay factors
//    to one exponential of the summed L / (beta gamma c tau);
//  - the adjoint is carried as nu_k = lambda_k dE_k/dY_k, the derivative of
//    log f in the range: nu_k = nu_(k+1) + a_k K_k with the forward sweep's
//    K_k = dE_k/dY_k and half decay slopes, which it keeps in `work`: four
//    operations per segment in place of an inversion, two table slopes and a
//    decay term;
//  - the lanes' contributions to a segment are summed 32 segments at a time
//    through shared memory (one addition per lane and segment, not five).
// About 37 FP64 instructions per segment and lane (forward and adjoint) against
// about 450.  4096 rays of the 64x64x32 grid, 32 nodes, flux and J^T r: kernel
// 6.94 -> 0.75 ms.

// Shared memory: the staged columns (all six, or the three that the segments read,
// the others then in global memory), two derived ones, then per warp the lengths and
// grammages of the ray's segments and (ADJ) the 32 x 33 tile.
enum { T_E = 0, T_LOGE, T_RR, T_SEGCOL, T_RS = T_SEGCOL, T_AS, T_AR, T_NCOL };
constexpr int kTile = 32 * 33;
inline size_t eval64_smem(int staged, int ld, int seg_cap, int warps, bool adj) {
  return (size_t(staged + 2) * ld + size_t(warps) * (2 * size_t(seg_cap) + (adj ? kTile : 0))) * sizeof(double);
}
__device__ __forceinline__ bool is_nan_bits(double x) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}

template <bool ADJ>
__global__ void __launch_bounds__(kWarps * 32) eval64_kernel(EvalP P) {
  extern __shared__ __align__(16) double smem[];
  __shared__ uint64_t mbar;
  const int ld = P.tab.ld, n = P.tab.n;
  const double* src[T_NCOL] = {P.tab.col(0, DP_COL_E),          P.tab.col(0, DP_COL_LOGE),
                               P.tab.col(P.rock, DP_COL_CSDA_R), P.tab.col(P.rock, DP_COL_CSDA_S),
                               P.tab.col(P.air, DP_COL_CSDA_S),  P.tab.col(P.air, DP_COL_CSDA_R)};
  if (!stage_columns(smem, src, P.staged, uint32_t(ld * sizeof(double)), &mbar, P.wait_iters)) {
    if (threadIdx.x == 0) atomicExch(P.err_flag, 1);
    return;
  }
  const bool all = P.staged == T_NCOL;
  const double *tE = smem + T_E * ld, *tlE = smem + T_LOGE * ld, *rR = smem + T_RR * ld;
  const double* rS = all ? smem + T_RS * ld : src[T_RS];
  const double *aS = all ? smem + T_AS * ld : src[T_AS], *aR = all ? smem + T_AR * ld : src[T_AR];
  double *rinv = smem + P.staged * ld, *dle = rinv + ld;
  for (int i = threadIdx.x; i < n - 1; i += blockDim.x) {
    rinv[i] = 1.0 / (rR[i + 1] - rR[i]);
    dle[i] = tlE[i + 1] - tlE[i];
  }
  __syncthreads();
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cap = P.seg_cap;
  double* sL = dle + ld + size_t(warp) * (2 * size_t(cap) + (ADJ ? kTile : 0));
  double* sG = sL + cap;    // grammage rho L
  double* tile = sG + cap;  // [segment & 31][lane]
  double2* work = ADJ ? P.work + (size_t(blockIdx.x) * warps + warp) * size_t(cap) * 32 + lane : nullptr;
  const double Emax = tE[n - 1], Rlo = rR[0], Rhi = rR[n - 1];
  const double half_inv_m = 0.5 / P.mass, inv_ctau = 1.0 / P.ctau, half_inv_mct = 0.5 / (P.mass * P.ctau);
  for (long q = blockIdx.x * long(warps) + warp; q < P.n_rays; q += long(gridDim.x) * warps) {
    const long r = P.order[q];
    const int64_t off = P.row_ptr[r];
    const int nseg = int(P.row_ptr[r + 1] - off);
    for (int s = lane; s < nseg; s += 32) {
      const double L = P.len[off + s];
      sL[s] = L;
      sG[s] = L * seg_density(P, P.cell[off + s]);
    }
    __syncwarp();
    const double cs_safe = fmax(fabs(P.rays[r].cos_theta), 0.01), inv_cs = 1.0 / cs_safe;
    const double Lair = (P.H - P.zmax) * inv_cs;
    const double Gair = fmax((1.205 * 12e3 * inv_cs) * P.air_dexp, 0.0);
    const double cs = P.star[r].x, cs129 = P.star[r].y;
    double fsum = 0.0;
    for (int base = 0; base < P.n_nodes; base += 32) {
      const int nd = base + lane;
      // (a NaN node energy ends its node at the first segment: it takes no part)
      const bool active = nd < P.n_nodes && !(nseg > 0 && is_nan_bits(P.nE[nd]));
      const double E0 = active ? P.nE[nd] : 1.0;
      // the node's place: interval i, offset t in log E; edge: clamped there
      int i = 0;
      double t = 0.0;
      bool edge = true;
      if (E0 >= Emax) {
        i = n - 2;
        t = 1.0;
      } else if (E0 > tE[0]) {
        const double lE = f64::log(E0);
        i = P.tab.uniform ? uniform_interval(tlE, n, lE, P.tab.lE0, P.tab.inv_dlE) : bisect(tlE, n, lE);
        t = (lE - tlE[i]) / dle[i];
        edge = false;
      }
      __syncwarp();
      double Y = fma(t, rR[i + 1] - rR[i], rR[i]);
      const double S0 = fma(t, rS[i + 1] - rS[i], rS[i]);
      double E = E0, dsum = 0.0, K = edge ? 0.0 : E0 * dle[i] * rinv[i];
      bool ok = active;
      for (int s = 0; s < nseg; ++s) {
        const double L = sL[s], Yn = Y + sG[s];
        double En;
        // clamped at a table end; a NaN (of either sign: the comparisons are of bits)
        // arrives at one of them too and ends the node
        if (!f64::lt_pos(Yn, Rhi)) {
          ok = ok && !is_nan_bits(Yn);
          i = n - 2;
          t = 1.0;
          Y = Rhi;
          En = Emax;
          K = 0.0;
          edge = true;
        } else if (!f64::lt_pos(Rlo, Yn)) {
          ok = ok && !is_nan_bits(Yn);
          i = 0;
          t = 0.0;
          Y = Rlo;
          En = tE[0];
          K = 0.0;
          edge = true;
        } else {
          while (i < n - 2 && !f64::lt_pos(Yn, rR[i + 1])) ++i;
          while (i > 0 && f64::lt_pos(Yn, rR[i])) --i;
          t = (Yn - rR[i]) * rinv[i];
          Y = Yn;
          En = f64::exp(fma(t, dle[i], tlE[i]));
          K = ADJ ? En * (dle[i] * rinv[i]) : 0.0;
          edge = false;
        }
        __syncwarp();
        ok = ok && (unsigned long long)__double_as_longlong(En) < 0x426d1a94a2000000ull;  // 1e12
        double dib;
        const double ib = f64::inv_beta_gamma((E + En) * half_inv_m, &dib);
        dsum = fma(L, ib, dsum);
        // K = dE/dY and half of the segment's decay slope a in its mean energy
        if (ADJ) work[size_t(s) * 32] = double2{K, -(L * half_inv_mct * dib)};
        E = En;
      }
      // the air column from the place on the shared energy grid
      const double dar = aR[i + 1] - aR[i], das = aS[i + 1] - aS[i], drs = rS[i + 1] - rS[i];
      const double Ya = fma(t, dar, aR[i]) + Gair;
      int j = i;
      double tj, Ef;
      bool edgeF = true;
      if (Ya >= aR[n - 1]) {
        j = n - 2;
        tj = 1.0;
        Ef = Emax;
      } else if (Ya <= aR[0]) {
        j = 0;
        tj = 0.0;
        Ef = tE[0];
      } else {
        j = walk_up(aR, n, Ya, i);
        tj = (Ya - aR[j]) / (aR[j + 1] - aR[j]);
        Ef = f64::exp(fma(tj, dle[j], tlE[j]));
        edgeF = false;
      }
      __syncwarp();
      const double SN = fma(t, drs, rS[i]), SaN = fma(t, das, aS[i]);
      const double dasF = aS[j + 1] - aS[j], SaF = fma(tj, dasF, aS[j]);
      double diba;
      const double iba = f64::inv_beta_gamma((E + Ef) * half_inv_m, &diba);
      const double w = f64::div(SN * SaF, S0 * SaN) * f64::exp(-fma(Lair, iba, dsum) * inv_ctau);
      double dlogF = 0.0;
      const double F = gccly_flux(cs, cs129, Ef, active ? P.nq[nd] : 0.0, ADJ ? &dlogF : nullptr);
      const double f = ok ? w * F : 0.0, coef = ok ? 2.0 * P.nw[nd] / P.n_nodes : 0.0;
      fsum += coef * f;
      if (ADJ) {
        // d log f / d Y_N, times the node's weight and flux
        double nu = 0.0;
        const double cf = coef * f;
        if (coef != 0.0 && f != 0.0 && !edge) {
          const double hA = -(Lair * half_inv_mct * diba);
          const double iE = f64::rcp(E * dle[i]), dSr = drs * iE / SN, dSaN = das * iE / SaN;
          double lam = dSr - dSaN + hA;
          if (!edgeF) {
            const double dEf = Ef * dle[j] / (aR[j + 1] - aR[j]) * (dar * iE);
            lam += dEf * (dasF / (SaF * Ef * dle[j]) + hA + dlogF);
          }
          nu = cf * lam * K;
        }
        __syncwarp();
        double2 cur = nseg > 0 ? work[size_t(nseg - 1) * 32] : double2{0.0, 0.0};
        for (int s = nseg - 1; s >= 0; --s) {
          const double2 prev = s > 0 ? work[size_t(s - 1) * 32] : double2{0.0, 0.0};
          const double h = cf * cur.y;
          nu = fma(h, cur.x, nu);
          tile[(s & 31) * 33 + lane] = nu * sL[s];
          // a clamped start has no derivative
          nu = f64::hi32(prev.x) == 0 ? 0.0 : fma(h, prev.x, nu);
          cur = prev;
          if ((s & 31) == 0) {
            __syncwarp();
            if (lane < nseg - s) {
              double v = 0.0;
              for (int k = 0; k < 32; ++k) v += tile[lane * 33 + k];
              double* J = P.jval64 + off + s + lane;
              *J = base == 0 ? v : *J + v;
            }
            __syncwarp();
          }
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) fsum += __shfl_xor_sync(0xffffffffu, fsum, o);
    if (lane == 0) P.flux[r] = fsum;
    __syncwarp();
  }
}
