// plain_fused.cu -- the RK4 stages of the FP64 plain form as one launch per stage (compiled
// with -fmad=false).
//
// Within a step the positions, the neighbour lists and (without the continuity equation) the
// densities are constant, so everything a pair sum takes from them alone is formed once, by
// k_pprep, with the operations the reference repeats in every stage:
//   hW   (m/rho) W of every entry (a stress-point's wall entry: 1 - beta of the wall velocity)
//   hG   (G m)/rho of a stress-point's entries, both components
//   norm the sum of W m / rho of a target, and its reciprocal
//   AE   the CSPM moments of a target
// A stage then reads them instead of recomputing: 4 + 10 FP64 operations an entry on the
// stress-point side and 8 + 21 on the node side, against 12 + 22 and 18 + 21; the
// multiplications among them (2 + 4 and 4 + 12) run on the integer pipes (mul_int).
//
// k_pstage runs a whole stage of both kinds (blocks of stress-points first, then blocks of
// nodes): stress_point_update, adapt_stress2 and the BCs, get_derivatives, the rates, their
// RK accumulation, and the state of the next stage.  The values a stage reads from its
// neighbours (node velocities pv, stress-point stresses ps and stress/rho^2 pa) are double
// buffered, so the two kinds need no order between them.  k_pfinish interpolates the final
// state and moves the particles.  Results are bit-identical to the separate kernels of
// plain_step.cu, which remain for the options that change densities or node stresses between
// the two halves of a stage (Ctx::fused).
//
// What bounds it: the additions on the FP64 pipe (2 lanes a clock and SM) at large sizes; at small ones the
// serial chain of a target's sums, which LS and LN lanes a target share by component (one
// velocity component a lane, one stress component a lane), each component still summed in
// list order by one lane.
#include <cuda_runtime.h>

#include <algorithm>

#include "ctx.cuh"
#include "stage_tail.cuh"

namespace sps {

namespace {

// adapt_stress2 (the plain form's stress_return of plain_step.cu)
__device__ __forceinline__ void ret(const Real& M, double& a, double& b, double& c, double& d) {
  if (M.ncrit != 12) return;
  if (inside_cone_f32(M.alpha2f, M.kcf, a, b, c, d)) return;
  adapt_stress(M.alpha2, M.kc, M.kc_shift, a, b, c, d);
}

// a / b with y = RN(1/b): the corrected product for a numerator of ordinary exponent (the
// range in which no step of div_rcp leaves the normal numbers, |b| within 2^+-200), else the
// IEEE division
__device__ __forceinline__ double div_pre(double a, double b, double y) {
  const int ex = (int)((__double_as_longlong(a) >> 52) & 0x7FF);
  if (ex > 400 && ex < 1640) return div_rcp(a, b, y);
  if ((__double_as_longlong(a) << 1) == 0) return a * y;  // a signed zero
  return a / b;
}

// the state of a stress-point at the start of a stage from its rates' result (a, b, c, d):
// return and BCs; that is what the nodes interpolate (ps), and returned once more (the
// reference returns every stress again after the interpolation) it enters get_derivatives
// (pa = sigma / rho^2)
__device__ __forceinline__ void sp_publish(const Dev& D, const Real& M, const StepScalars& sc,
                                           int t, int buf, double a, double b, double c, double d,
                                           bool with_pa, double* fin) {
  double vx = 0.0, vy = 0.0;
  ret(M, a, b, c, d);
  apply_bcs(D, sc, t, vx, vy, a, b, c, d);
  const size_t i = (size_t)(t - D.NN);
  st4(D.ps[buf] + 4 * i, a, b, c, d);
  ret(M, a, b, c, d);
  apply_bcs(D, sc, t, vx, vy, a, b, c, d);
  if (with_pa) {
    const double r2 = D.rho2[t], y = D.rinv2[t];
    st4(D.pa[buf] + 4 * i, div_pre(a, r2, y), div_pre(b, r2, y), div_pre(c, r2, y), D.mass[t]);
  }
  if (fin) {
    fin[0] = a;
    fin[1] = b;
    fin[2] = c;
    fin[3] = d;
  }
}

// a stress-point's entry: its constants, and unless its partner is a wall (true) its terms of
// the norm and of the CSPM moments
struct Terms {
  double norm, e[4];
};
template <bool CSPM>
__device__ __forceinline__ bool sp_entry(const Dev& D, int k, int j, double xt, double yt,
                                         Terms& T) {
  const int ns = D.NT - D.NN;
  const int4 e = D.cross[ell(j, k, D.N2)];
  const int u = e.x;
  const double Gx = f64_of(__int_as_float(e.z)), Gy = f64_of(__int_as_float(e.w));
  const double mu = D.mass[u], ru = D.rho[u], iu = D.rinv[u];
  const bool wall = e.y < 0;
  double h, h1, h2;
  if (!wall) {
    const double w = f64_of(__int_as_float(e.y));
    h = mul_int(D.vol[u], w);
    T.norm = div_rcp(mul_int(w, mu), ru, iu);
    h1 = div_rcp(mul_int(Gx, mu), ru, iu);
    h2 = div_rcp(mul_int(Gy, mu), ru, iu);
    if (CSPM) {
      const double xu = D.px[u] - xt, yu = D.py[u] - yt;
      T.e[0] = xu * h1;
      T.e[1] = yu * h1;
      T.e[2] = xu * h2;
      T.e[3] = yu * h2;
    }
  } else {
    const double wp = (double)D.wallpos[u];
    double da, db;
    if (D.horiz[u] == 1.0f) {
      da = fabs(yt - wp);
      db = fabs(D.py[u] - wp);
    } else {
      da = fabs(xt - wp);
      db = fabs(D.px[u] - wp);
    }
    const double bq = 1.0 + db / da;
    const double beta = 1.5 < bq ? 1.5 : bq;
    h = 1.0 - beta;
    h1 = div_rcp(-Gx * mu, ru, iu);
    h2 = div_rcp(-Gy * mu, ru, iu);
  }
  D.hW[(size_t)j * D.NT + k] = h;
  D.hG[(size_t)j * ns + k] = make_double2(h1, h2);
  return wall;
}
// a node's entry: the same, and of a wall partner u the boundary force (fx, fy) if it has one
// (push)
template <bool CSPM>
__device__ __forceinline__ bool node_entry(const Dev& D, const Real& M, int t, int k, int j,
                                           double xt, double yt, Terms& T, int& u, bool& push,
                                           float& fx, float& fy) {
  const int4 e = D.cross[ell(j, k, D.N2)];
  u = e.x;
  push = false;
  if (e.y < 0) {
    push = D.inside && D.bound_from_lists && u >= M.dum0 && u < M.dum0 + M.ndum2 &&
           bound_term(D, M, t, u, fx, fy);
    return true;
  }
  const double w = f64_of(__int_as_float(e.y));
  const double mu = D.mass[u], ru = D.rho[u], iu = D.rinv[u];
  D.hW[(size_t)j * D.NT + k] = mul_int(D.vol[u], w);
  T.norm = div_rcp(mul_int(w, mu), ru, iu);
  if (CSPM) {
    const double dwx = -f64_of(__int_as_float(e.z)), dwy = -f64_of(__int_as_float(e.w));
    const double h1b = -div_rcp(dwx * mu, ru, iu), h2b = -div_rcp(dwy * mu, ru, iu);
    const double xu = D.px[u] - xt, yu = D.py[u] - yt;
    T.e[0] = xu * h1b;
    T.e[1] = yu * h1b;
    T.e[2] = xu * h2b;
    T.e[3] = yu * h2b;
  }
  return false;
}

// Once per step, per target: the constants of its list entries (file comment), the boundary
// force of a node, and the state of stage 0.  Bound by the integer pipes, which form the
// products and quotients, and by memory (494 us at 2 million particles, 1069 with FP64 products;
// the terms of the CSPM moments are compiled out without them, since FP64 instructions that a
// predicate switches off still occupy their pipe: 1292 -> 1069 then).  L = 8, for problems that cannot fill the chip with one lane a
// target: eight lanes form eight entries' constants and terms together, and every one of them
// adds the terms in list order (0.0 where an entry has none, which changes no sum: none of
// them is ever -0.0); 49 -> 18 us at 600 particles, soil failure example 53 -> 16.
template <int L, bool CSPM>
__global__ void __launch_bounds__(128) k_pprep(Dev D) {
  constexpr unsigned all = 0xffffffffu;
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / L, q = threadIdx.x & (L - 1);
  const bool act = i < D.NT;
  if (L == 1 && !act) return;
  const int k = act ? i : 0;
  const int ns = D.NT - D.NN;
  const bool sp = k < ns;
  const int t = D.colid[k];
  const Real* Mp;
  const StepScalars* scp;
  load_real(D, t, Mp, scp);
  const Real& M = *Mp;
  const int deg = act ? D.degC[k] : 0;
  if (D.walk_order && act && q == 0) put_target_walk_order(D, k, t, !sp);
  if (L > 1) __syncwarp();
  const double xt = D.px[t], yt = D.py[t];
  double norm = 0.0;
  double AE[4] = {0.0, 0.0, 0.0, 0.0};
  WallForce F;
  if (L == 1) {
    auto add = [&](const Terms& T) {
      norm = norm + T.norm;
      if (CSPM)
        for (int p = 0; p < 4; p++) AE[p] = AE[p] + T.e[p];
    };
    if (sp) {
      for (int j = 0; j < deg; j++) {
        Terms T;
        if (!sp_entry<CSPM>(D, k, j, xt, yt, T)) add(T);
      }
    } else {
      for (int j = 0; j < deg; j++) {
        Terms T;
        int u;
        bool push;
        float fx, fy;
        const bool wall = node_entry<CSPM>(D, M, t, k, j, xt, yt, T, u, push, fx, fy);
        if (!wall) add(T);
        else F.met(D, push, u, fx, fy);
      }
    }
  } else {
    const int nmax = __reduce_max_sync(all, deg);
    for (int j = 0; j < nmax; j += L) {
      Terms T = {0.0, {0.0, 0.0, 0.0, 0.0}};
      int u = 0;
      bool wall = false, push = false;
      float fx = 0.0f, fy = 0.0f;
      if (j + q < deg) {
        if (sp) sp_entry<CSPM>(D, k, j + q, xt, yt, T);
        else wall = node_entry<CSPM>(D, M, t, k, j + q, xt, yt, T, u, push, fx, fy);
      }
#pragma unroll
      for (int o = 0; o < L; o++) {
        norm = norm + __shfl_sync(all, T.norm, o, L);
        if (CSPM)
          for (int p = 0; p < 4; p++) AE[p] = AE[p] + __shfl_sync(all, T.e[p], o, L);
      }
      if (__any_sync(all, wall)) {
#pragma unroll
        for (int o = 0; o < L; o++) {
          const bool w = __shfl_sync(all, (int)wall, o, L), p = __shfl_sync(all, (int)push, o, L);
          const int v = __shfl_sync(all, u, o, L);
          const float x = __shfl_sync(all, fx, o, L), y = __shfl_sync(all, fy, o, L);
          if (w) F.met(D, p, v, x, y);
        }
      }
    }
  }
  if (q || !act) return;
  if (!sp) {
    F.store(D, M, t);
    D.bc_int[t] = F.bc_int;
  }
  D.norm[k] = norm;
  D.rnorm[k] = norm != 0.0 ? 1.0 / norm : 0.0;
  if (CSPM) {
    double A[5];
    cspm_moments<false>(D, AE, A);
    for (int p = 0; p < 5; p++) D.AE[(size_t)p * D.NT + k] = A[p];
  }
  // the state of stage 0 (RK4 starts from zero rates)
  if (sp) {
    const double a = D.s0[t], b = D.s1[t], c = D.s2[t], d = D.s3[t];
    st4(D.st0c + 4 * (size_t)k, a, b, c, d);
    sp_publish(D, M, *scp, t, 0, a + 0.0, b + 0.0, c + 0.0, d + 0.0, true, nullptr);
  } else {
    const double v0x = D.vx[t], v0y = D.vy[t];
    D.vx0[t] = v0x;
    D.vy0[t] = v0y;
    double vx = v0x + 0.0, vy = v0y + 0.0, a = 0.0, b = 0.0, c = 0.0, d = 0.0;
    if (norm == 0.0) {  // no stress-point in reach: RK4 clears the stress, nothing sets it
      ret(M, a, b, c, d);
      apply_bcs(D, *scp, t, vx, vy, a, b, c, d);
      D.s0[t] = a;
      D.s1[t] = b;
      D.s2[t] = c;
      D.s3[t] = d;
      vx = 0.0;
      vy = 0.0;
    }
    apply_bcs(D, *scp, t, vx, vy, a, b, c, d);
    reinterpret_cast<double2*>(D.pv[0])[t] = make_double2(vx, vy);
  }
}

// In the kernels below kP is the number of entries a pass whose list words and neighbour records
// are loaded before any is summed: more in flight where few warps are there to hide a
// latency, one where they are many.

// A wall's velocity seen by a stress-point: v - (v (1 - beta) + beta 0).  Rare, and out of line:
// as predicated instructions it would take the FP64 pipe for every entry.
static __device__ __noinline__ double wall_du64(double v, double ob) { return v - (v * ob + 0.0); }

// One stage of a stress-point; LS = 2: lane d of the pair sums velocity component d
template <int LS>
__device__ __forceinline__ void sp_stage(const Dev& D, int stage, int k, bool act, int q) {
  constexpr int kP = LS == 1 ? 1 : 4;
  const int ns = D.NT - D.NN, cur = stage & 1, nxt = cur ^ 1;
  const int t = D.colid[k];
  const double2* __restrict__ pv = reinterpret_cast<const double2*>(D.pv[cur]);
  const int deg = act ? D.degC[k] : 0;
  const double norm = D.norm[k], rn = D.rnorm[k];
  const Real* Mp;
  const StepScalars* scp;
  load_real(D, t, Mp, scp);
  const Real& M = *Mp;
  double v0 = 0.0, v1 = 0.0;
  for (int j = 0; j < deg; j += kP) {
    int4 e[kP];
    double h[kP];
    double2 v[kP];
#pragma unroll
    for (int i = 0; i < kP; i++) {
      e[i] = j + i < deg ? D.cross[ell(j + i, k, D.N2)] : make_int4(0, -1, 0, 0);
      h[i] = e[i].y >= 0 ? D.hW[(size_t)(j + i) * D.NT + k] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < kP; i++) v[i] = e[i].y >= 0 ? pv[e[i].x] : make_double2(0.0, 0.0);
#pragma unroll
    for (int i = 0; i < kP; i++)
      if (e[i].y >= 0) {
        if (LS == 1) {
          v0 = v0 + mul_int(v[i].x, h[i]);
          v1 = v1 + mul_int(v[i].y, h[i]);
        } else {
          v0 = v0 + (q ? v[i].y : v[i].x) * h[i];
        }
      }
  }
  double vt0 = 0.0, vt1 = 0.0;  // RK4 clears the velocity; no node in reach leaves it so
  if (norm != 0.0) {
    vt0 = div_pre(v0, norm, rn);
    if (LS == 1) vt1 = div_pre(v1, norm, rn);
  }
  if (LS == 2) {
    const double o = __shfl_xor_sync(0xffffffffu, vt0, 1);
    vt1 = q ? vt0 : o;
    vt0 = q ? o : vt0;
  }
  const d4 own = ld4(D.ps[cur] + 4 * (size_t)(t - D.NN));
  double st[4] = {own.a, own.b, own.c, own.d};
  ret(M, st[0], st[1], st[2], st[3]);
  apply_bcs(D, *scp, t, vt0, vt1, st[0], st[1], st[2], st[3]);
  double g[4] = {0.0, 0.0, 0.0, 0.0};  // grad1(a,b) at a + 2b
  const double vtq = LS == 2 && q ? vt1 : vt0;
  for (int j = 0; j < deg; j += kP) {
    int4 e[kP];
    double2 h[kP], v[kP];
#pragma unroll
    for (int i = 0; i < kP; i++) {
      e[i] = j + i < deg ? D.cross[ell(j + i, k, D.N2)] : make_int4(0, 0, 0, 0);
      h[i] = j + i < deg ? D.hG[(size_t)(j + i) * ns + k] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int i = 0; i < kP; i++) {
      v[i] = make_double2(0.0, 0.0);
      if (j + i < deg) {
        if (e[i].y >= 0) v[i] = pv[e[i].x];
        else v[i].x = D.hW[(size_t)(j + i) * D.NT + k];  // 1 - beta
      }
    }
#pragma unroll
    for (int i = 0; i < kP; i++)
      if (j + i < deg) {
        double du0, du1 = 0.0;
        if (e[i].y >= 0) {
          du0 = LS == 1 ? v[i].x - vt0 : (q ? v[i].y : v[i].x) - vtq;
          if (LS == 1) du1 = v[i].y - vt1;
        } else {
          du0 = wall_du64(vtq, v[i].x);
          if (LS == 1) du1 = wall_du64(vt1, v[i].x);
        }
        g[0] = g[0] + mul_int(du0, h[i].x);
        g[2] = g[2] + mul_int(du0, h[i].y);
        if (LS == 1) {
          g[1] = g[1] + mul_int(du1, h[i].x);
          g[3] = g[3] + mul_int(du1, h[i].y);
        }
      }
  }
  if (LS == 2) {
    g[1] = __shfl_xor_sync(0xffffffffu, g[0], 1);
    g[3] = __shfl_xor_sync(0xffffffffu, g[2], 1);
    if (q) return;
  }
  if (!act) return;
  if (D.cspm) {
    double A[5];
    for (int i = 0; i < 5; i++) A[i] = D.AE[(size_t)i * D.NT + k];
    cspm_correct<2, false>(A, g);
  }
  double rhs[4], der;
  sp_rates_f64(D, M, *scp, t, g, st, rhs, der);
  const double f2 = (stage == 1 || stage == 2) ? 2.0 : 1.0;  // RK4 weights 1, 2, 2, 1
  double rk[4] = {0.0, 0.0, 0.0, 0.0}, rd = 0.0;
  double* rks = D.rkc + 4 * (size_t)k;
  if (stage > 0) {
    const d4 o = ld4(rks);
    rk[0] = o.a;
    rk[1] = o.b;
    rk[2] = o.c;
    rk[3] = o.d;
    rd = D.RKd[k];
  }
  for (int i = 0; i < 4; i++) rk[i] = rk[i] + f2 * rhs[i];
  rd = rd + der * f2;
  const d4 s0 = ld4(D.st0c + 4 * (size_t)k);
  if (stage < 3) {
    st4(rks, rk[0], rk[1], rk[2], rk[3]);
    D.RKd[k] = rd;
    const double f1dt = (stage == 2 ? 1.0 : 0.5) * M.dt;  // RK4 nodes 1/2, 1/2, 1
    sp_publish(D, M, *scp, t, nxt, s0.a + f1dt * rhs[0], s0.b + f1dt * rhs[1],
               s0.c + f1dt * rhs[2], s0.d + f1dt * rhs[3], true, nullptr);
  } else {  // the end of RK4 (2_SPH_main_2018.f90:784-799) and update_strain
    const double dt6 = M.dt6;
    double f[4];
    sp_publish(D, M, *scp, t, nxt, s0.a + dt6 * rk[0], s0.b + dt6 * rk[1], s0.c + dt6 * rk[2],
               s0.d + dt6 * rk[3], false, f);
    D.s0[t] = f[0];
    D.s1[t] = f[1];
    D.s2[t] = f[2];
    D.s3[t] = f[3];
    const int ex = (int)((__double_as_longlong(rd) >> 52) & 0x7FF);
    const double dd = (ex > 64 && ex < 1980) ? div_rcp(rd, 6.0, 1.0 / 6.0)
                      : (__double_as_longlong(rd) << 1) == 0 ? rd : rd / 6.0;
    D.Ddev[t] = dd;
    D.iv1[t] = D.iv1[t] + M.dt * dd;
  }
}

// artificial_viscosity's pair value for target t and neighbour u (2_SPH_main_2018.f90:
// 826-904): the FP32 products visc dW; the quotient by the pair's density uses the
// reciprocal of the last density met (the pairs of a uniform material share one)
struct ViscT {
  double xt, yt, vtx, vty, ht, rt, a600, beta;
  float hf, rf;
  double yrho;
  float yfor;
};
__device__ __forceinline__ float2 visc_pair(const Dev& D, ViscT& T, const int4& e, double2 vu) {
  const int u = e.x;
  const float xij = f32_rn(T.xt - D.px[u]), yij = f32_rn(T.yt - D.py[u]);
  const double hu = D.hsml[u], ru = D.rho[u];
  // 0.5 (h + h) = h exactly
  const float h = __double_as_longlong(hu) == __double_as_longlong(T.ht) ? T.hf
                                                                          : (float)(0.5 * (T.ht + hu));
  const float rho2 = __double_as_longlong(ru) == __double_as_longlong(T.rt)
                         ? T.rf
                         : (float)(0.5 * (T.rt + ru));
  float div_u = f32_rn(f64_of(xij) * (T.vtx - vu.x));
  div_u = f32_rn(f64_of(div_u) + f64_of(yij) * (T.vty - vu.y));
  const float sq = sqrtf(xij * xij + yij * yij);
  const float theta = (h * div_u) / (sq * sq + 0.01f * (h * h));
  float visc = 0.0f;
  if (div_u < 0) {
    if (rho2 != T.yfor) {
      T.yfor = rho2;
      T.yrho = 1.0 / f64_of(rho2);
    }
    const double num = -(T.a600 * f64_of(theta)) + T.beta * f64_of(theta * theta);
    visc = div_rcp_f32(num, f64_of(rho2), T.yrho);
  }
  return make_float2(visc * __int_as_float(e.z), visc * __int_as_float(e.w));
}

// sigma / rho_d^2 of a node's dummy partner (out of line as wall_du64)
static __device__ __noinline__ double wall_A(double s, double r2, double y) { return div_pre(s, r2, y); }

// One stage of a node; LN = 4: lane q of the group sums stress component q, then the
// derivative sums of component q (q < 3)
template <int LN>
__device__ __forceinline__ void node_stage(const Dev& D, int stage, int k, bool act, int q) {
  constexpr int kP = LN == 1 ? 1 : 4;
  const int cur = stage & 1, nxt = cur ^ 1;
  const int t = D.colid[k];
  const double* __restrict__ ps = D.ps[cur];
  const double* __restrict__ pa = D.pa[cur];
  const int deg = act ? D.degC[k] : 0;
  const double norm = D.norm[k], rn = D.rnorm[k];
  const Real* Mp;
  const StepScalars* scp;
  load_real(D, t, Mp, scp);
  const Real& M = *Mp;
  const int b0 = LN == 4 ? (threadIdx.x & 31 & ~3) : 0;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (int j = 0; j < deg; j += kP) {
    int4 e[kP];
    double h[kP];
    d4 v[kP];
    double vq[kP];
#pragma unroll
    for (int i = 0; i < kP; i++) {
      e[i] = j + i < deg ? D.cross[ell(j + i, k, D.N2)] : make_int4(0, -1, 0, 0);
      h[i] = e[i].y >= 0 ? D.hW[(size_t)(j + i) * D.NT + k] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < kP; i++)
      if (e[i].y >= 0) {
        const double* p = ps + 4 * (size_t)(e[i].x - D.NN);
        if (LN == 1) v[i] = ld4(p);
        else vq[i] = p[q];
      }
#pragma unroll
    for (int i = 0; i < kP; i++)
      if (e[i].y >= 0) {
        if (LN == 1) {
          s[0] = s[0] + mul_int(v[i].a, h[i]);
          s[1] = s[1] + mul_int(v[i].b, h[i]);
          s[2] = s[2] + mul_int(v[i].c, h[i]);
          s[3] = s[3] + mul_int(v[i].d, h[i]);
        } else {
          s[0] = s[0] + vq[i] * h[i];
        }
      }
  }
  if (norm != 0.0) {
    if (LN == 1) {
      for (int i = 0; i < 4; i++) s[i] = div_pre(s[i], norm, rn);
    } else {
      s[0] = div_pre(s[0], norm, rn);
    }
  }
  if (LN == 4) {
    const double o = s[0];
    for (int i = 0; i < 4; i++) s[i] = __shfl_sync(0xffffffffu, o, b0 + i);
  }
  double2 v = reinterpret_cast<const double2*>(D.pv[cur])[t];
  if (norm == 0.0) {  // the stress of the last return, returned again at the stage's start
    s[0] = D.s0[t];
    s[1] = D.s1[t];
    s[2] = D.s2[t];
    s[3] = D.s3[t];
    if (stage > 0) {
      ret(M, s[0], s[1], s[2], s[3]);
      apply_bcs(D, *scp, t, v.x, v.y, s[0], s[1], s[2], s[3]);
    }
  }
  ret(M, s[0], s[1], s[2], s[3]);
  apply_bcs(D, *scp, t, v.x, v.y, s[0], s[1], s[2], s[3]);
  const double r2 = D.rho2[t], y2 = D.rinv2[t];
  double at[3];
  if (LN == 1) {
    for (int i = 0; i < 3; i++) at[i] = div_pre(s[i], r2, y2);
  } else {
    at[0] = div_pre(q == 0 ? s[0] : q == 1 ? s[1] : s[2], r2, y2);
  }
  double g2[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};  // grad2(s,b) at s + 3b
  const double sq = q == 0 ? s[0] : q == 1 ? s[1] : s[2];
  const int qa = LN == 4 ? (q < 3 ? q : 2) : 0;
  for (int j = 0; j < deg; j += kP) {
    int4 e[kP];
    d4 v4[kP];
    double aq[kP], mu[kP];
#pragma unroll
    for (int i = 0; i < kP; i++)
      e[i] = j + i < deg ? D.cross[ell(j + i, k, D.N2)] : make_int4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < kP; i++)
      if (j + i < deg && e[i].y >= 0) {
        const double* p = pa + 4 * (size_t)(e[i].x - D.NN);
        if (LN == 1) {
          v4[i] = ld4(p);
          mu[i] = v4[i].d;
        } else {
          aq[i] = p[qa];
          mu[i] = p[3];
        }
      }
#pragma unroll
    for (int i = 0; i < kP; i++)
      if (j + i < deg) {
        const double dwx = -f64_of(__int_as_float(e[i].z)), dwy = -f64_of(__int_as_float(e[i].w));
        if (e[i].y < 0) {  // a dummy carries the node's stress
          const int u = e[i].x;
          const double ru2 = D.rho2[u], yu2 = D.rinv2[u];
          mu[i] = D.mass[u];
          if (LN == 1) {
            v4[i].a = wall_A(s[0], ru2, yu2);
            v4[i].b = wall_A(s[1], ru2, yu2);
            v4[i].c = wall_A(s[2], ru2, yu2);
          } else {
            aq[i] = wall_A(sq, ru2, yu2);
          }
        }
        if (LN == 1) {
          const double au[3] = {v4[i].a, v4[i].b, v4[i].c};
#pragma unroll
          for (int p = 0; p < 3; p++) {
            const double sum = at[p] + au[p];
            g2[p] = g2[p] - mul_int(mu[i], mul_int(dwx, sum));
            g2[p + 3] = g2[p + 3] - mul_int(mu[i], mul_int(dwy, sum));
          }
        } else {
          const double sum = at[0] + aq[i];
          g2[0] = g2[0] - mu[i] * (dwx * sum);
          g2[3] = g2[3] - mu[i] * (dwy * sum);
        }
      }
  }
  if (LN == 4) {
    const double a = g2[0], b = g2[3];
    for (int i = 0; i < 3; i++) {
      g2[i] = __shfl_sync(0xffffffffu, a, b0 + i);
      g2[i + 3] = __shfl_sync(0xffffffffu, b, b0 + i);
    }
  }
  double avx = 0.0, avy = 0.0;
  if (M.alpha > 0 || M.beta > 0) {
    // artificial_viscosity (2_SPH_main_2018.f90:826-904): FP32 accumulators.  LN = 4: the
    // group's lanes evaluate four pairs together, then add them in list order
    float ax = 0.0f, ay = 0.0f;
    const int degs = act ? D.degS[k] : 0;
    const double2* __restrict__ pv = reinterpret_cast<const double2*>(D.pv[cur]);
    ViscT T;
    T.xt = D.px[t];
    T.yt = D.py[t];
    T.vtx = v.x;
    T.vty = v.y;
    T.ht = D.hsml[t];
    T.rt = D.rho[t];
    T.hf = f32_rn(T.ht);
    T.rf = f32_rn(T.rt);
    T.a600 = M.alpha * 600.0;
    T.beta = M.beta;
    T.yfor = 0.0f;
    T.yrho = 0.0;
    int nmax = degs;
    if (LN == 4) nmax = __reduce_max_sync(0xffffffffu, degs);  // every lane meets the shuffles
    for (int j = 0; j < nmax; j += LN) {
      double px = 0.0, py = 0.0;
      const int jj = j + (LN == 4 ? q : 0);
      if (jj < degs) {
        const int4 e = D.same[ell(jj, k, D.N2)];
        const float2 p = visc_pair(D, T, e, pv[e.x]);
        const double mu = D.mass[e.x];
        px = f64_of(p.x) * mu;
        py = f64_of(p.y) * mu;
      }
      if (LN == 1) {
        ax = f32_rn(f64_of(ax) + px);
        ay = f32_rn(f64_of(ay) + py);
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const double qx = __shfl_sync(0xffffffffu, px, b0 + i);
          const double qy = __shfl_sync(0xffffffffu, py, b0 + i);
          if (j + i < degs) {
            ax = f32_rn(f64_of(ax) + qx);
            ay = f32_rn(f64_of(ay) + qy);
          }
        }
      }
    }
    avx = -f64_of(ax);
    avy = -f64_of(ay);
  }
  if (LN == 4 && q) return;
  if (!act) return;
  if (D.cspm) {
    double A[5];
    for (int i = 0; i < 5; i++) A[i] = D.AE[(size_t)i * D.NT + k];
    cspm_correct<3, false>(A, g2);
  }
  double rx, ry;
  node_rhs_f64(D, M, *scp, t, g2, v.x, v.y, avx, avy, 0.0, 0.0, rx, ry);
  const double f2 = (stage == 1 || stage == 2) ? 2.0 : 1.0;
  double kx = 0.0, ky = 0.0;
  if (stage > 0) {
    kx = D.RKv[0][t];
    ky = D.RKv[1][t];
  }
  kx = kx + f2 * rx;
  ky = ky + f2 * ry;
  const double v0x = D.vx0[t], v0y = D.vy0[t];
  double nx, ny, a = 0.0, b = 0.0, c = 0.0, d = 0.0;
  if (stage < 3) {
    D.RKv[0][t] = kx;
    D.RKv[1][t] = ky;
    const double f1dt = (stage == 2 ? 1.0 : 0.5) * M.dt;
    nx = v0x + f1dt * rx;
    ny = v0y + f1dt * ry;
  } else {
    nx = v0x + M.dt6 * kx;
    ny = v0y + M.dt6 * ky;
  }
  if (norm == 0.0) {
    D.s0[t] = s[0];
    D.s1[t] = s[1];
    D.s2[t] = s[2];
    D.s3[t] = s[3];
    nx = 0.0;
    ny = 0.0;
  }
  apply_bcs(D, *scp, t, nx, ny, a, b, c, d);
  reinterpret_cast<double2*>(D.pv[nxt])[t] = make_double2(nx, ny);
}

// RK4 stage (2_SPH_main_2018.f90:700-777): blocks [0, nbs) the stress-points, the rest the
// nodes
// One lane a target: 64 registers, eight blocks a multiprocessor, one entry in flight a lane; the
// FP64 pipe and the integer pipes work for different warps at the same time, so many of them are
// needed (2 million particles, us a step: four entries and 124 registers 6253, two and 5485,
// one and 80 registers 5037, one and 64 registers 4903, spills included; 4234 since the stress
// return and the flow rule repeat no FP64 work).
template <int LS, int LN>
__global__ void __launch_bounds__(128, LS == 1 ? 8 : 1) k_pstage(Dev D, int stage, int nbs) {
  const int ns = D.NT - D.NN;
  if ((int)blockIdx.x < nbs) {
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) / LS;
    const bool act = g < ns;
    if (LS == 1 && !act) return;
    sp_stage<LS>(D, stage, act ? g : 0, act, threadIdx.x & (LS - 1));
  } else {
    const int g = ((blockIdx.x - nbs) * blockDim.x + threadIdx.x) / LN;
    const bool act = g < D.NN;
    if (LN == 1 && !act) return;
    node_stage<LN>(D, stage, ns + (act ? g : 0), act, threadIdx.x & (LN - 1));
  }
}

// the final interpolation, return and BCs (2_SPH_main_2018.f90:130-135), then the position
// update (:140-146, without XSPH) and the displacements (:166-180)
// INT: the products on the integer pipes (large problems; below, where the chain of one warp's
// latencies counts and not the FP64 pipe, the FP64 multiplication is shorter: 600 particles 24
// us against 29; 2 million 581 against 396)
template <bool INT>
__global__ void __launch_bounds__(128) k_pfinish(Dev D) {
  constexpr int kP = INT ? 2 : 4;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= D.N2) return;
  if (k >= D.NT) {  // dummies: their place in the step's pair build
    D.x0x[k] = D.px[k];
    D.x0y[k] = D.py[k];
    return;
  }
  const int ns = D.NT - D.NN;
  const int t = D.colid[k];
  const int deg = D.degC[k];
  const double norm = D.norm[k], rn = D.rnorm[k];
  const Real* Mp;
  const StepScalars* scp;
  load_real(D, t, Mp, scp);
  const Real& M = *Mp;
  double vx, vy, vx0, vy0;
  if (k < ns) {
    const double2* __restrict__ pv = reinterpret_cast<const double2*>(D.pv[0]);
    double v0 = 0.0, v1 = 0.0;
    for (int j = 0; j < deg; j += kP) {
      int4 e[kP];
      double h[kP];
      double2 v[kP];
#pragma unroll
      for (int i = 0; i < kP; i++) {
        e[i] = j + i < deg ? D.cross[ell(j + i, k, D.N2)] : make_int4(0, -1, 0, 0);
        h[i] = e[i].y >= 0 ? D.hW[(size_t)(j + i) * D.NT + k] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < kP; i++) v[i] = e[i].y >= 0 ? pv[e[i].x] : make_double2(0.0, 0.0);
#pragma unroll
      for (int i = 0; i < kP; i++)
        if (e[i].y >= 0) {
          v0 = v0 + (INT ? mul_int(v[i].x, h[i]) : v[i].x * h[i]);
          v1 = v1 + (INT ? mul_int(v[i].y, h[i]) : v[i].y * h[i]);
        }
    }
    vx0 = D.vx[t];
    vy0 = D.vy[t];
    vx = vy = 0.0;
    if (norm != 0.0) {
      vx = div_pre(v0, norm, rn);
      vy = div_pre(v1, norm, rn);
    }
    double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
    apply_bcs(D, *scp, t, vx, vy, a, b, c, d);
    D.vx0[t] = vx0;
    D.vy0[t] = vy0;
  } else {
    const double* __restrict__ ps = D.ps[0];
    double s[4] = {0.0, 0.0, 0.0, 0.0}, iv = 0.0;
    for (int j = 0; j < deg; j += kP) {
      int4 e[kP];
      double h[kP], w[kP];
      d4 v[kP];
#pragma unroll
      for (int i = 0; i < kP; i++) {
        e[i] = j + i < deg ? D.cross[ell(j + i, k, D.N2)] : make_int4(0, -1, 0, 0);
        h[i] = e[i].y >= 0 ? D.hW[(size_t)(j + i) * D.NT + k] : 0.0;
      }
#pragma unroll
      for (int i = 0; i < kP; i++)
        if (e[i].y >= 0) {
          v[i] = ld4(ps + 4 * (size_t)(e[i].x - D.NN));
          w[i] = D.iv1[e[i].x];
        }
#pragma unroll
      for (int i = 0; i < kP; i++)
        if (e[i].y >= 0) {
          s[0] = s[0] + (INT ? mul_int(v[i].a, h[i]) : v[i].a * h[i]);
          s[1] = s[1] + (INT ? mul_int(v[i].b, h[i]) : v[i].b * h[i]);
          s[2] = s[2] + (INT ? mul_int(v[i].c, h[i]) : v[i].c * h[i]);
          s[3] = s[3] + (INT ? mul_int(v[i].d, h[i]) : v[i].d * h[i]);
          iv = iv + w[i] * h[i];
        }
    }
    const double2 v = reinterpret_cast<const double2*>(D.pv[0])[t];
    vx = v.x;
    vy = v.y;
    if (norm != 0.0) {
      for (int i = 0; i < 4; i++) s[i] = div_pre(s[i], norm, rn);
      D.iv1[t] = div_pre(iv, norm, rn);
    } else {  // RK4's last return and BCs, then no interpolated stress
      s[0] = D.s0[t];
      s[1] = D.s1[t];
      s[2] = D.s2[t];
      s[3] = D.s3[t];
      ret(M, s[0], s[1], s[2], s[3]);
      apply_bcs(D, *scp, t, vx, vy, s[0], s[1], s[2], s[3]);
      vx = 0.0;
      vy = 0.0;
    }
    ret(M, s[0], s[1], s[2], s[3]);
    apply_bcs(D, *scp, t, vx, vy, s[0], s[1], s[2], s[3]);
    D.s0[t] = s[0];
    D.s1[t] = s[1];
    D.s2[t] = s[2];
    D.s3[t] = s[3];
    vx0 = D.vx0[t];
    vy0 = D.vy0[t];
  }
  D.vx[t] = vx;
  D.vy[t] = vy;
  move_particle(D, M, t, k >= ns, vx0, vy0, vx, vy);
}

}  // namespace

void launch_pprep(Ctx& c) {
  Dev D = c.d;
  if (c.reinterpolates()) D.walk_order = 0;  // done
  D.same_entries = c.same_now();  // the lists to put in walk order
  const bool group = D.NT <= c.group_max;
  const int n = group ? 8 * D.NT : D.NT, b = c.block_for(n, 128), nb = (n + b - 1) / b;
  auto k = D.cspm ? (group ? k_pprep<8, true> : k_pprep<1, true>)
                  : (group ? k_pprep<8, false> : k_pprep<1, false>);
  k<<<nb, b, 0, c.stream>>>(D);
}

// Lanes a target: split by component while one lane a target leaves most of the chip's 608
// FP64 pipes with a warp or less
void launch_pstage(Ctx& c, int stage) {
  const Dev& D = c.d;
  const int ns = D.NT - D.NN;
  const bool split = D.NT <= c.split_max;
  const int ls = split ? 2 : 1, ln = split ? 4 : 1;
  const int b = c.block_for(ns * ls + D.NN * ln, std::min(c.blk[TK_DERIVS], 128));
  const int nbs = (ns * ls + b - 1) / b, nbn = (D.NN * ln + b - 1) / b;
  if (split) k_pstage<2, 4><<<nbs + nbn, b, 0, c.stream>>>(D, stage, nbs);
  else k_pstage<1, 1><<<nbs + nbn, b, 0, c.stream>>>(D, stage, nbs);
}

void launch_pfinish(Ctx& c) {
  const int b = c.block_for(c.d.N2, 128);
  if (c.d.NT > c.split_max) k_pfinish<true><<<(c.d.N2 + b - 1) / b, b, 0, c.stream>>>(c.d);
  else k_pfinish<false><<<(c.d.N2 + b - 1) / b, b, 0, c.stream>>>(c.d);
}

}  // namespace sps
