// stx_rok4w.cu -- the ROK4 integration (kernels_gpu.F90:10360-11205) with one
// warp per state vector, for the batched 0-D reactors and for small grids.
//
// The thread-per-cell kernels suit large grids: 32 cells per warp amortise the
// Krylov algebra.  A batch of reactors or a grid of a few thousand cells is
// different: a launch lasts as long as its slowest state, and a thread takes
// some 1e5 cycles for a step of one state.  Here a warp integrates one state:
//  * lane m holds component m of every vector (state, Krylov basis, stages);
//    dot products and norms sum the lanes' products in component order, by
//    shuffles that do not depend on one another and a chain of adds, one per
//    component, so every lane has the bits of the thread kernels' loops (a
//    butterfly would take five rounds, in another order);
//  * the right-hand side evaluates the reaction rates one reaction per lane
//    (the per-reaction arithmetic of chem_source_rec or chem_source_sp), then
//    lane k sums its species' terms in ascending reaction order from shared
//    memory (the species-major lists t.sk_*);
//  * the temperature Newton iteration and the 4 x 4 Krylov algebra run
//    redundantly in every lane.
// So a state gets the bits of the thread kernels.  Compiled without FMA
// contraction, like the other chemistry kernels.
#include <mutex>
#include <set>
#include <utility>

#include "stx_chem.cuh"

#define WFULL 0xffffffffu
#define WNRMAX 64          // reactions per mechanism the warp kernels take (two per lane)

// sum_m a_m b_m over the first N lanes, in lane order
template <int N>
__device__ __forceinline__ double wdot(double a, double b) {
  const double x = a * b;
  double s = 0.0;
#pragma unroll
  for (int m = 0; m < N; m++) s = s + __shfl_sync(WFULL, x, m);
  return s;
}

// Warp ROK4 of one state of NV <= 32 components (lane m holds component m;
// lanes >= NV hold 0).  f.rhs(y, T, lane) returns the lane's component of the
// right-hand side; f.accept / f.done as in rok4_core.
template <int NV, class FN>
__device__ void rok4_core_w(const DevCtx &c, FN &f, double &v, double T_iter, double fls, double dttry,
                            double time_start, double time_end, int simpler, int maxsteps, int lane) {
  const double gam = 0.572816062482135;
  const double alpha[4][3] = {{0, 0, 0},
                              {0.432364435748567, 0, 0},
                              {-0.514211316876170, 1.382271144617360, 0},
                              {-0.514211316876170, 1.382271144617360, 0.0}};
  const double gmc[4][3] = {{0, 0, 0},
                            {-0.602765307997356, 0, 0},
                            {-1.389195789724843, 1.072950969011413, 0},
                            {0.992356412977094, -1.390032613873701, -0.440875890223325}};
  const double bsv[4] = {0.194335256262729, 0.483167813989227, 0.0, 0.322496929748044};
  const double btv[4] = {-0.217819895945721, 1.03130847478467, 0.186511421161047, 0.0};
  double V[STX_MMAX + 1], Ks[STX_NSTAGE], inv[STX_MMAX * STX_MMAX];
  int mA = 0;
#pragma unroll
  for (int q = 0; q < STX_MMAX * STX_MMAX; q++) inv[q] = 0.0;
#pragma unroll
  for (int q = 0; q < STX_NSTAGE; q++) Ks[q] = 0.0;
  double time = time_start, dt = dttry, errn = 1.0;
  int it = 0;
  while (time < (time_end - 1.0e-12)) {
    dt = dmin_(dt, time_end - time);
    it = it + 1;
    // ---- arnoldi (:10664-10792)
    double raw, rs;                   // f(VEC), and less fl_sav with the simpler splitting
    {
      const double TOL = 1e-6, eps = 1.0e-08;
      double HH[(STX_MMAX + 1) * STX_MMAX], HI[STX_MMAX * STX_MMAX], prj[STX_MMAX], lam[STX_MMAX];
#pragma unroll
      for (int q = 0; q < (STX_MMAX + 1) * STX_MMAX; q++) HH[q] = 0.0;
#pragma unroll
      for (int q = 0; q < STX_MMAX * STX_MMAX; q++) HI[q] = 0.0;
#pragma unroll
      for (int q = 0; q <= STX_MMAX; q++) V[q] = 0.0;
#pragma unroll
      for (int q = 0; q < STX_MMAX; q++) prj[q] = 0.0;
      mA = 0;
      raw = f.rhs(v, T_iter, lane);
      rs = simpler == 1 ? raw - fls : raw;
      double nrm = sqrt(wdot<NV>(rs, rs));
      V[0] = rs / nrm;
#pragma unroll
      for (int kk = 1; kk <= STX_MMAX; kk++) {
        double jac = f.rhs(v + (eps * V[kk - 1]), T_iter, lane);
        if (simpler == 1) jac = jac - fls;
        jac = (jac - rs) / eps;
#pragma unroll
        for (int jj = 1; jj <= kk; jj++) {
          double dot = wdot<NV>(V[jj - 1], jac);
          HH[(kk - 1) * (STX_MMAX + 1) + jj - 1] = dot;
          jac = jac - (dot * V[jj - 1]);
        }
        double hn = sqrt(wdot<NV>(jac, jac));
        HH[(kk - 1) * (STX_MMAX + 1) + kk] = hn;
        V[kk] = jac / hn;
        prj[kk - 1] = wdot<NV>(V[kk - 1], rs);   // the earlier projections stand
#pragma unroll
        for (int n = 1; n <= kk; n++)
#pragma unroll
          for (int nn = 1; nn <= kk; nn++) {
            double h = -(dt * gam * HH[(nn - 1) * (STX_MMAX + 1) + n - 1]);
            if (n == nn) h = h + 1.0;
            HI[(nn - 1) * STX_MMAX + n - 1] = h;
          }
#pragma unroll
        for (int n = kk + 1; n <= STX_MMAX; n++) HI[(n - 1) * STX_MMAX + n - 1] = 1.0;
        inv_matrix_k(HI, kk);
#pragma unroll
        for (int ll = 1; ll <= STX_MMAX; ll++) {
          double s = 0.0;
#pragma unroll
          for (int jj = 1; jj <= STX_MMAX; jj++) s = s + HI[(jj - 1) * STX_MMAX + ll - 1] * prj[jj - 1];
          lam[ll - 1] = s;
        }
        if (fabs(dt * gam * hn) * fabs(lam[kk - 1]) < TOL) {
          mA = kk;
#pragma unroll
          for (int q = 0; q < STX_MMAX * STX_MMAX; q++) inv[q] = HI[q];
          break;
        }
      }
    }
    // ---- stages: B F = A (Vb^T F), this lane's row of A from V and inv
    double vb[STX_MMAX];
#pragma unroll
    for (int q = 0; q < STX_MMAX; q++) vb[q] = (q < mA) ? V[q] : 0.0;
#pragma unroll
    for (int ii = 1; ii <= STX_NSTAGE; ii++) {
      double ys = v;
#pragma unroll
      for (int jj = 1; jj <= ii - 1; jj++) ys = ys + dt * alpha[ii - 1][jj - 1] * Ks[jj - 1];
      double F = ii == 1 ? raw : f.rhs(ys, T_iter, lane);
      double GK = 0.0;
#pragma unroll
      for (int jj = 1; jj <= ii - 1; jj++) GK = GK + gmc[ii - 1][jj - 1] / gam * Ks[jj - 1];
      F = F + GK;
      if (simpler == 1) F = F - fls;
      double s = 0.0;
#pragma unroll
      for (int kk = 0; kk < STX_MMAX; kk++) {
        double pf = (kk < mA) ? wdot<NV>(V[kk], F) : 0.0;
        double a = vb[0] * ((kk == 0 ? 1.0 : 0.0) - inv[kk * STX_MMAX + 0]);
#pragma unroll
        for (int jj = 1; jj < STX_MMAX; jj++) a = a + vb[jj] * ((jj == kk ? 1.0 : 0.0) - inv[kk * STX_MMAX + jj]);
        s = s + a * pf;
      }
      Ks[ii - 1] = F - s - GK;
    }
    double a = v, b = v;
#pragma unroll
    for (int ii = 0; ii < STX_NSTAGE; ii++) {
      a = a + dt * bsv[ii] * Ks[ii];
      b = b + dt * btv[ii] * Ks[ii];
    }
    double errv = (b - a) / ((1.0e-4) * a + 1.0e-8);
    double errmax = sqrt(wdot<NV>(errv, errv));
    double fac = 0.625 * pow(errn, 0.1) / pow(errmax, 0.175);
    double dtnext = dt * dmin_(5.0, dmax_(0.2, fac));
    if (errmax < 1.0) {
      time = time + dt;
      v = a;
      f.accept(v, time, T_iter, time_end, lane);
    }
    dt = dtnext;
    errn = errmax;
    if (it > maxsteps) {
      if (lane == 0) set_status(c.p, STX_ST_ROS_STEPS_CAP);
      break;
    }
  }
  f.done(time, T_iter, it);
}

// Production rate of this lane's species (0 beyond NS) at T = tt from the
// concentrations in sm[0..NS), written by the lanes just before.  sm: per-warp
// shared scratch of NS + 1 + WNRMAX doubles (concentrations, a 1, then the
// reaction rates).
template <int NS, bool DD>
__device__ __forceinline__ double production_w(const DevTab &t, double tt, double *sm, int lane) {
  double *conc = sm, *qr = sm + NS + 1;
  if (lane == 0) conc[NS] = 1.0;
  __syncwarp();
  const int nr = t.nr;
  double Rtti = 1.0 / (t.Ru * tt);
  int itt;
  double dtt;
  kc_pos(t, tt, itt, dtt);
  double lh = 0.0, ll = 0.0;
  if (DD && rec_range(t, tt)) log_dd(tt, lh, ll);
  if (rec_range(t, tt)) {
    for (int lr = lane; lr < nr; lr += 32) {
      const double2 *rec = (const double2 *)t.rec + (long long)lr * (REC_N / 2);
      const double2 c0 = __ldg(rec), c1 = __ldg(rec + 1), c2 = __ldg(rec + 2), c3 = __ldg(rec + 3);
      const uint4 ix = __ldg((const uint4 *)(rec + 7));
      const double *kc0 = t.kc_r + (long long)(itt - 1) * nr + lr;
      const double ka = ldg(kc0), kc = ka + (ldg(kc0 + nr) - ka) * dtt;
      const int fl = __double2loint(c3.y), cls = fl & 255;
      double tbs = 1.0;
      if (cls != REC_PLAIN) {
        tbs = 0.0;
        const double *ef = t.rec + (nr * REC_N + lr * rec_es(NS));
#pragma unroll
        for (int k = 0; k < NS; k++) tbs = tbs + ldg(ef + k) * conc[k];
      }
      const double kf = rec_kf<DD>(t, lr, cls, c0, c1, c2, c3.x, tt, Rtti, lh, ll, tbs);
      const double kb = (fl >> 8) & 255 ? kf / kc : 0.0;
      const double q1 = conc[ix.x & 255] * conc[(ix.x >> 8) & 255] * conc[(ix.x >> 16) & 255];
      const double q2 = conc[ix.x >> 24] * conc[ix.y & 255] * conc[(ix.y >> 8) & 255];
      const double tb = cls == REC_TB ? tbs : 1.0;
      qr[lr] = tb * (kf * q1 - kb * q2);
    }
  } else {
  for (int lr = lane; lr < nr; lr += 32) {
    int ty = __ldg(t.reac_ty + lr);
    double tbs = 1.0;
    if (ty != 0) {
      tbs = 0.0;
#pragma unroll 1
      for (int k = 0; k < NS; k++) tbs = tbs + ldg(t.tb_eff + (long long)k * nr + lr) * conc[k];
    }
    double kf, kb;
    rate_consts<false>(t, lr, ty, tt, Rtti, itt, dtt, tbs, kf, kb);
    const int cnt = __ldg(t.sp_cnt + lr);
    const unsigned char *ix = t.sp_idx + (long long)lr * STX_SPW;
    const double *cf = t.sp_coef + (long long)lr * STX_SPW;
    double q1 = 1.0, q2 = 1.0;
#pragma unroll 1
    for (int n = 0; n < (cnt & 255); n++) {
      double x = conc[__ldg(ix + n)], e = ldg(cf + n);
      if (e == 1.0) q1 = q1 * x;
      else q1 = q1 * stoich_pow(x, e);
    }
#pragma unroll 1
    for (int n = 0; n < ((cnt >> 8) & 255); n++) {
      double x = conc[__ldg(ix + STX_SPR + n)], e = ldg(cf + STX_SPR + n);
      if (e == 1.0) q2 = q2 * x;
      else q2 = q2 * stoich_pow(x, e);
    }
    double tb = (ty == 1) ? tbs : 1.0;
    qr[lr] = tb * (kf * q1 - kb * q2);
  }
  }
  __syncwarp();
  double acc = 0.0;
  if (lane < NS) {
    const double mwk = ldg(t.mw + lane);
    const int n0 = __ldg(t.sk_ptr + lane), n1 = __ldg(t.sk_ptr + lane + 1);
#pragma unroll 1
    for (int n = n0; n < n1; n++) {
      double wdtkj = ldg(t.sk_c + n) * qr[__ldg(t.sk_r + n)];
      acc = acc + wdtkj * mwk;
    }
  }
  __syncwarp();
  return acc;
}

// Right-hand side of the constant-pressure reactor (cp_rhs) for the state held
// one component per lane; returns this lane's component.
template <int NS>
__device__ __noinline__ double cp_rhs_w(const DevCtx &c, double y, double T_iter, double h, double p, double *sm,
                                        int lane) {
  const DevTab &t = c.t;
  double Yc[NS];
#pragma unroll
  for (int k = 0; k < NS; k++) {
    double yk = __shfl_sync(WFULL, y, k);
    Yc[k] = yk > 0.0 ? yk : 0.0;
  }
  double tt = temp_from_poly<NS>(t, t.cp, c.p, h, T_iter, Yc);
  double rm = 0.0;
#pragma unroll
  for (int k = 0; k < NS; k++) rm = rm + ldg(t.rgas + k) * Yc[k];
  double rho = p / (rm * tt);
  if (lane < NS) sm[lane] = rho * (y > 0.0 ? y : 0.0) / ldg(t.mw + lane);
  const double acc = production_w<NS, true>(t, tt, sm, lane);
  return lane < NS ? acc / rho : 0.0;
}

// Right-hand side of a flow cell (krylov_rhs), the species densities one per
// lane; m0..m3 the momentum components and the energy.  Lanes beyond NS return 0.
template <int NS, bool DD>
__device__ __noinline__ double flow_rhs_w(const DevCtx &c, double y, double m0, double m1, double m2, double m3,
                                          double T_iter, double *sm, int lane) {
  const DevTab &t = c.t;
  const double yc = y > 0.0 ? y : 0.0;
  double Y[NS];
#pragma unroll
  for (int k = 0; k < NS; k++) Y[k] = __shfl_sync(WFULL, yc, k);
  double rho = Y[0];
#pragma unroll
  for (int k = 1; k < NS; k++) rho = rho + Y[k];
  const double ri = 1.0 / rho;
#pragma unroll
  for (int k = 0; k < NS; k++) Y[k] = Y[k] * ri;
  if (lane < NS) sm[lane] = rho * (yc * ri) / ldg(t.mw + lane);
  const double uu = m0 * ri, vv = m1 * ri, ww = m2 * ri;
  const double qq = 0.5 * (uu * uu + vv * vv + ww * ww);
  const double ee = (m3 * ri) - qq;
  const double tt = temp_from_e<NS>(t, c.p, ee, T_iter, Y);
  return production_w<NS, DD>(t, tt, sm, lane);
}

// The flow cell, one component per lane.  FULL: the state is (rho Y_k, rho u,
// rho v, rho w, rho E) as in Rok4Flow; otherwise the species densities alone, the
// other four fixed in mom, as in Rok4FlowSpecies.
template <int NS, bool FULL>
struct Rok4FlowW {
  const DevCtx &c;
  double mom[4];
  double *sm;
  __device__ __forceinline__ double rhs(double y, double T_iter, int lane) const {
    double m[4];
#pragma unroll
    for (int q = 0; q < 4; q++) m[q] = FULL ? __shfl_sync(WFULL, y, NS + q) : mom[q];
    return flow_rhs_w<NS, !FULL>(c, y, m[0], m[1], m[2], m[3], T_iter, sm, lane);
  }
  __device__ __forceinline__ void accept(double v, double, double &T_iter, double &, int) const {
    double Y[NS], m[4];
#pragma unroll
    for (int k = 0; k < NS; k++) Y[k] = __shfl_sync(WFULL, v, k);
#pragma unroll
    for (int q = 0; q < 4; q++) m[q] = FULL ? __shfl_sync(WFULL, v, NS + q) : mom[q];
    double rho = Y[0];
#pragma unroll
    for (int k = 1; k < NS; k++) rho = rho + Y[k];
    const double ri = 1.0 / rho;
#pragma unroll
    for (int k = 0; k < NS; k++) Y[k] = Y[k] * ri;
    const double uu = m[0] * ri, vv = m[1] * ri, ww = m[2] * ri;
    const double qq = 0.5 * (uu * uu + vv * vv + ww * ww);
    const double ee = m[3] * ri - qq;
    T_iter = temp_from_e<NS>(c.t, c.p, ee, T_iter, Y);
  }
  __device__ __forceinline__ void done(double, double, int) const {}
};

// One warp per flow cell (k_rok4's work on a small grid).  Bound by the latency of
// a cell's chain of right-hand sides: the budget of four CTAs per SM (128 registers, some
// spilled outside the right-hand side) keeps 2368 cells resident at once.  4096
// H2/air cells: 309 us against 814 us with a thread per cell.  Budgets of 2, 3, 4, 5
// and 6 CTAs, one 2e-7 s window on a B200: 1024 H2/air cells 1.50, 1.55, 1.66, 1.77,
// 1.84 ms; 4096 4.98, 4.26, 3.95, 4.24, 4.41; 8192 8.86, 7.53, 7.36, 7.41, 7.52; 4096
// cells of 14 species 22.6, 20.0, 19.6, 22.4, 23.7.
template <int NS>
__global__ void __launch_bounds__(128, 4)
    k_rok4_w(DevCtx c, const DevCtx *__restrict__ cg, double *__restrict__ w, const double *__restrict__ wa,
             const double *__restrict__ fl_sav, double dttry, double t0, double t1, int simpler) {
  __shared__ double sm_all[4][NS + 1 + WNRMAX];
  const DevGrid &g = c.g;
  const double eps_Z = 5e-4;
  if (c.p.dt_d) dttry = dttry * *c.p.dt_d;   // captured CFL-driven step: dttry holds the splitting's factor
  if (c.p.time_d) {                 // captured step: the window starts at the device-held time
    t0 = *c.p.time_d;
    t1 = t0 + dttry;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long cell = (long long)blockIdx.x * 4 + wid;
  if (cell >= g.npi) return;
  const int i = 1 + (int)(cell % g.nx);
  const long long r = cell / g.nx;
  const int j = 1 + (int)(r % g.ny), k = 1 + (int)(r / g.ny);
  const long long p = gidx(g, i, j, k);
  const double Z = FG(wa, p, NS + 12);
  if (!(Z > eps_Z && Z < 1.0 - eps_Z)) return;
  const double T = FG(wa, p, NS + 5);
  double v = lane < NS + 4 ? FG(w, p, lane + 1) : 0.0;
  const int maxsteps = cg->p.ros_maxsteps;
  if (simpler != 1) {
    Rok4FlowW<NS, false> f{*cg, {}, sm_all[wid]};
#pragma unroll
    for (int q = 0; q < 4; q++) f.mom[q] = __shfl_sync(WFULL, v, NS + q);
    v = lane < NS ? v : 0.0;
    rok4_core_w<NS>(*cg, f, v, T, 0.0, dttry, t0, t1, 0, maxsteps, lane);
    if (lane < NS) FG(w, p, lane + 1) = v;
  } else {
    Rok4FlowW<NS, true> f{*cg, {}, sm_all[wid]};
    const double fls = lane < NS + 4 ? fl_sav[cell + (long long)lane * g.npi] : 0.0;
    rok4_core_w<NS + 4>(*cg, f, v, T, fls, dttry, t0, t1, 1, maxsteps, lane);
    if (lane < NS + 4) FG(w, p, lane + 1) = v;
  }
}

template <int NS>
static int rok4_w_t(const DevCtx &c, const DevCtx *cg, cudaStream_t s, double *w, const double *wa,
                    const double *fl_sav, double dttry, double t0, double t1, int simpler) {
  if constexpr (NS + 4 > 32) {
    return STX_E_UNSUPPORTED;
  } else {
    if (c.t.nr > WNRMAX) return STX_E_UNSUPPORTED;
    k_rok4_w<NS><<<(unsigned)((c.g.npi + 3) / 4), 128, 0, s>>>(c, cg, w, wa, fl_sav, dttry, t0, t1, simpler);
    STX_CUDA_TRY(cudaGetLastError());
    return STX_OK;
  }
}

bool rok4_warp_serves(const DevTab &t) {
  switch (t.ns) {
#define X(N) case N: return N + 4 <= 32 && t.nr <= WNRMAX;
    STX_FOR_NS(X)
#undef X
    default: return false;
  }
}

int launch_rok4_warp(const DevCtx &c, const DevCtx *cg, cudaStream_t s, double *w, const double *wa,
                     const double *fl_sav, double dttry, double t0, double t1, int simpler) {
  switch (c.t.ns) {
#define X(N) case N: return rok4_w_t<N>(c, cg, s, w, wa, fl_sav, dttry, t0, t1, simpler);
    STX_FOR_NS(X)
#undef X
    default: return STX_E_UNSUPPORTED;
  }
}

template <int NS>
struct Rok4ConstPW {
  const DevCtx &c;
  double h, p, T0, ign_factor, end_factor;
  double *sm;
  double t_ign, time_reached, T_final;
  int steps;
  __device__ __forceinline__ double rhs(double y, double T_iter, int lane) const {
    return cp_rhs_w<NS>(c, y, T_iter, h, p, sm, lane);
  }
  __device__ __forceinline__ void accept(double v, double time, double &T_iter, double &time_end, int) {
    double Yc[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) {
      double yk = __shfl_sync(WFULL, v, k);
      Yc[k] = yk > 0.0 ? yk : 0.0;
    }
    T_iter = temp_from_poly<NS>(c.t, c.t.cp, c.p, h, T_iter, Yc);
    if (t_ign < 0.0 && T_iter > ign_factor * T0) {
      t_ign = time;
      double te = end_factor * time;
      if (te < time_end) time_end = te;
    }
  }
  __device__ __forceinline__ void done(double time, double T_iter, int it) {
    time_reached = time;
    T_final = T_iter;
    steps = it;
  }
};

// One warp per reactor, reactors claimed from the work-stealing counter.
template <int NS>
__global__ void __launch_bounds__(128) k_batch0d_w(DevCtx c, int n, const double *__restrict__ T0,
                                                   const double *__restrict__ p0, const double *__restrict__ Y0,
                                                   double t_max, double dttry, double ign_factor, double end_factor,
                                                   double *__restrict__ Y, double *__restrict__ T,
                                                   double *__restrict__ t_ign, double *__restrict__ t_end,
                                                   int *__restrict__ nsteps, unsigned int *counter) {
  __shared__ double sm_all[4][NS + 1 + WNRMAX];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double *sm = sm_all[wid];
  for (;;) {
    unsigned int r0 = 0;
    if (lane == 0) r0 = atomicAdd(counter, 1u);
    const long long r = (long long)__shfl_sync(WFULL, r0, 0);
    if (r >= n) break;
    double v = lane < NS ? Y0[(long long)lane * n + r] : 0.0;
    const double T0r = T0[r];
    double h = 0.0;
#pragma unroll 1
    for (int k = 0; k < NS; k++) h = h + Y0[(long long)k * n + r] * species_poly_int(c.t, c.t.cpi, T0r, k + 1);
    Rok4ConstPW<NS> f{c, h, p0[r], T0r, ign_factor, end_factor, sm, -1.0, 0.0, T0r, 0};
    rok4_core_w<NS>(c, f, v, T0r, 0.0, dttry, 0.0, t_max, 0, c.p.ros_maxsteps, lane);
    if (lane < NS) Y[(long long)lane * n + r] = v;
    if (lane == 0) {
      T[r] = f.T_final;
      t_ign[r] = f.t_ign;
      t_end[r] = f.time_reached;
    }
    // nsteps last, after every lane's outputs are visible system-wide: a caller
    // whose outputs are mapped host memory polls it to collect finished reactors
    __threadfence_system();
    __syncwarp();
    if (lane == 0) nsteps[r] = f.steps;
  }
}

template <int NS>
static int batch0d_w_t(const DevCtx &c, cudaStream_t s, int n, const double *T0, const double *p0, const double *Y0,
                       double t_max, double dttry, double ign, double endf, double *Y, double *T, double *t_ign,
                       double *t_end, int *nsteps, unsigned int *counter, int force) {
  if constexpr (NS > 32) {
    return STX_E_UNSUPPORTED;
  } else {
  if (c.t.nr > WNRMAX) return STX_E_UNSUPPORTED;
  int dev = 0, nsm = 148, per = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void *)k_batch0d_w<NS>, 128, 0);
  long long nb = (long long)nsm * (per < 1 ? 1 : per);
  long long need = ((long long)n + 3) / 4;      // four reactors (warps) per CTA
  // More reactors than resident warps: a thread per reactor finishes the batch
  // sooner (all of them run at once); the warp kernel only where every reactor
  // gets its own warp from the start, unless forced.
  if (!force && need > nb) return STX_E_UNSUPPORTED;
  STX_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned int), s));
  if (nb > need) nb = need;
  if (c.p.batch_ctas_max > 0 && nb > c.p.batch_ctas_max) nb = c.p.batch_ctas_max;   // after the choice of kernel
  k_batch0d_w<NS><<<(int)nb, 128, 0, s>>>(c, n, T0, p0, Y0, t_max, dttry, ign, endf, Y, T, t_ign, t_end, nsteps,
                                          counter);
  STX_CUDA_TRY(cudaGetLastError());
  return STX_OK;
  }
}

// The warp-per-reactor kernel (the one small, served batches take) is persistent
// and can stay resident for seconds.
// An SM holding one of their CTAs keeps its shared-memory/L1 split until the CTA
// exits, and a kernel that needs a larger shared-memory share (the staged
// convective sweeps, ~90 KB per CTA) cannot start a CTA there meanwhile; on a
// server that runs grid solves beside reactor launches those solves then wait
// for the reactors.  So the warp kernel asks for the largest shared-memory split,
// which every other kernel fits beside.  (The thread-per-reactor kernel, for
// large batches, keeps the default: its local working set needs the L1.)
template <int NS>
static void batch0d_carveout_t() {
  cudaFuncSetAttribute(k_batch0d_w<NS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                       (int)cudaSharedmemCarveoutMaxShared);
}

int launch_batch0d_setup(int ns) {
  static std::mutex mu;
  static std::set<std::pair<int, int>> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({dev, ns})) return STX_OK;
  switch (ns) {
#define X(N) case N: batch0d_carveout_t<N>(); break;
    STX_FOR_NS(X)
#undef X
    default: break;
  }
  done.insert({dev, ns});
  return cudaGetLastError() == cudaSuccess ? STX_OK : STX_E_CUDA;
}

int launch_batch0d_warp(const DevCtx &c, cudaStream_t s, int n, const double *T0, const double *p0, const double *Y0,
                        double t_max, double dttry, double ign, double endf, double *Y, double *T, double *t_ign,
                        double *t_end, int *nsteps, unsigned int *counter, int force) {
  switch (c.t.ns) {
#define X(N) case N: return batch0d_w_t<N>(c, s, n, T0, p0, Y0, t_max, dttry, ign, endf, Y, T, t_ign, t_end, nsteps, counter, force);
    STX_FOR_NS(X)
#undef X
    default: return STX_E_UNSUPPORTED;
  }
}
