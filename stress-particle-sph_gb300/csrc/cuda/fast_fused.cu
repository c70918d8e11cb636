// fast_fused.cu -- the RK4 stages of the FP32 form as one launch per stage.
//
// As in plain_fused.cu, positions, neighbour lists and densities are constant within a step, so
// k_fprep forms once what the pair sums take from them alone:
//   crossW  {partner, (m/rho) W} of every entry (the wall entries keep their sign bit)
//   hGf     {Gx m/rho, Gy m/rho} of a stress-point's entries, {-m Gx, -m Gy} of a node's
//   hB      1 - beta of the wall velocity of a stress-point's wall entries
//   normf   a target's interpolation norm and its reciprocal
//   msum    a node's sum of m dW (error-free products)
//   AE      the CSPM moments
// A stage then reads 16 bytes an entry (24 before) and one record a neighbour and sum (two
// before: m/rho came from a record of its own).
//
// k_fstage runs a whole stage of both kinds: stress_point_update, the stress return and BCs,
// get_derivatives, the rates, the RK accumulation and the next stage's state with its records.
// The records are double buffered, so the kinds need no order between them; the passes over
// the state between the separate kernels (stage begin, return, record writes, stress-point
// tail) are gone.  The sums are the separate kernels', term by term and in the same order:
// bit-identical results.
//
// With the learned surrogate, a step whose gate is open stores the gradients here instead
// and the rates follow in k_fstail after the network has run.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <string>

#include "ctx.cuh"
#include "fast_sums.cuh"

namespace sps {

namespace {

// adapt_stress2 (the FP32 form's stress_return of plain_step.cu)
__device__ __forceinline__ void retf(const Real& M, double& a, double& b, double& c, double& d) {
  if (M.ncrit != 12) return;
  if (inside_cone_f32(M.alpha2f, M.kcf, a, b, c, d)) return;
  adapt_stress_fast(M.alpha2, M.kc, M.kc_shift, a, b, c, d);
}

__device__ __forceinline__ float4 split2f(double x, double y) {
  float xh, xl, yh, yl;
  f32_split(x, xh, xl);
  f32_split(y, yh, yl);
  return make_float4(xh, yh, xl, yl);
}

// a + b c with both roundings (the step's updates are not contracted)
__device__ __forceinline__ double mad2(double a, double b, double c) {
  return __dadd_rn(a, __dmul_rn(b, c));
}

// sigma / rho^2 as hi + lo (k_adapt_bc's form)
__device__ __forceinline__ void split_A(const Dev& D, int t, double a, double b, double c,
                                        float4& h, float4& l) {
  const double ri = D.rinv[t];
  const double ri2 = ri * ri;
  f32_split(a * ri2, h.x, l.x);
  f32_split(b * ri2, h.y, l.y);
  f32_split(c * ri2, h.z, l.z);
  h.w = 0.0f;
  l.w = 0.0f;
}

// the state of a stress-point at the start of a stage (column k): return, BCs, and the
// records its nodes read
__device__ __forceinline__ void spf_publish(const Dev& D, const Real& M, const StepScalars& sc,
                                            int k, int t, int buf, double& a, double& b, double& c,
                                            double& d, bool last) {
  double vx = 0.0, vy = 0.0;
  retf(M, a, b, c, d);
  apply_bcs(D, sc, t, vx, vy, a, b, c, d);
  float4* rs = buf ? D.recS1 : D.recS;
  rs[t] = make_float4(f32_rn(a), f32_rn(b), f32_rn(c), f32_rn(d));
  if (last) return;
  st4(D.stc + 4 * (size_t)k, a, b, c, d);
  float4 h, l;
  split_A(D, t, a, b, c, h, l);
  (buf ? D.recA1 : D.recA)[t] = h;
  (buf ? D.recAl1 : D.recAl)[t] = l;
}

// one entry of a target: its constants, and what its sums take of it
struct TermF {
  bool wall, push;
  int u;
  float h;         // (m/rho) W
  float m, gx, gy; // node: mass and gradient -dW (m dW summed without error)
  float xu, yu, hx, hy;  // CSPM: separation and gradient factors
  float fx, fy;    // a wall's force on a node
};
template <bool CSPM>
__device__ __forceinline__ void spf_entry(const Dev& D, int k, int j, double xt, double yt,
                                          TermF& T) {
  const int ns = D.NT - D.NN;
  const int4 e = D.cross[ell(j, k, D.N2)];
  const int u = e.x;
  const float Gx = __int_as_float(e.z), Gy = __int_as_float(e.w);
  const float vol = D.recI[u].y;
  T.wall = e.y < 0;
  if (!T.wall) {
    T.h = vol * __int_as_float(e.y);
    D.crossW[(size_t)j * D.N2 + k] = make_int2(u, __float_as_int(T.h));
    T.hx = Gx * vol;
    T.hy = Gy * vol;
    D.hGf[(size_t)j * D.NT + k] = make_float2(T.hx, T.hy);
    if (CSPM) {
      T.xu = (float)(D.px[u] - xt);
      T.yu = (float)(D.py[u] - yt);
    }
    return;
  }
  const double wall = (double)D.wallpos[u];
  double da, db;
  if (D.horiz[u] == 1.0f) {
    da = fabs(yt - wall);
    db = fabs(D.py[u] - wall);
  } else {
    da = fabs(xt - wall);
    db = fabs(D.px[u] - wall);
  }
  const double bq = 1.0 + db / da;
  const double beta = 1.5 < bq ? 1.5 : bq;
  D.hB[(size_t)j * ns + k] = 1.0 - beta;
  D.crossW[(size_t)j * D.N2 + k] = make_int2(u, (int)0x80000000u);
  D.hGf[(size_t)j * D.NT + k] = make_float2(-Gx * vol, -Gy * vol);
}
template <bool CSPM>
__device__ __forceinline__ void nodef_entry(const Dev& D, const Real& M, int t, int k, int j,
                                            double xt, double yt, TermF& T) {
  const int4 e = D.cross[ell(j, k, D.N2)];
  const int u = e.x;
  const float dwx = -__int_as_float(e.z), dwy = -__int_as_float(e.w);
  T.u = u;
  T.gx = dwx;
  T.gy = dwy;
  T.wall = e.y < 0;
  if (!T.wall) {
    const float4 ri = D.recI[u];
    T.m = ri.w;
    T.h = ri.y * __int_as_float(e.y);
    D.crossW[(size_t)j * D.N2 + k] = make_int2(u, __float_as_int(T.h));
    if (CSPM) {
      const float vol = ri.y;
      T.hx = -(dwx * vol);
      T.hy = -(dwy * vol);
      T.xu = (float)(D.px[u] - xt);
      T.yu = (float)(D.py[u] - yt);
    }
  } else {
    T.m = (float)D.mass[u];
    D.crossW[(size_t)j * D.N2 + k] = make_int2(u, (int)0x80000000u);
    T.push = D.inside && D.bound_from_lists && u >= M.dum0 && u < M.dum0 + M.ndum2 &&
             bound_term(D, M, t, u, T.fx, T.fy);
  }
  D.hGf[(size_t)j * D.NT + k] = make_float2(T.m * dwx, T.m * dwy);
}

// Once per step, per target: the list constants (file comment), a node's wall force and wall
// flag, the state of stage 0.  L = 8 as k_pprep: eight lanes form the entries' constants, each
// adds their terms in list order (37 -> 20 us at 10,000 particles).
template <int L, bool CSPM>
__global__ void __launch_bounds__(128) k_fprep(Dev D) {
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
  Kahan nm;
  Kahan e0, e1, e2, e3;
  ProdSum sx, sy;
  WallForce F;
  const double xt = D.px[t], yt = D.py[t];
  auto take = [&](const TermF& x, bool node) {
    if (!x.wall) {
      nm.add(x.h);
      if (CSPM) {
        e0.add(x.xu * x.hx);
        e1.add(x.yu * x.hx);
        e2.add(x.xu * x.hy);
        e3.add(x.yu * x.hy);
      }
    } else if (node) {
      F.met(D, x.push, x.u, x.fx, x.fy);
    }
    if (node) {
      sx.add(x.m, x.gx);
      sy.add(x.m, x.gy);
    }
  };
  if (L == 1) {
    if (sp) {
      for (int j = 0; j < deg; j++) {
        TermF T;
        spf_entry<CSPM>(D, k, j, xt, yt, T);
        take(T, false);
      }
    } else {
      for (int j = 0; j < deg; j++) {
        TermF T;
        nodef_entry<CSPM>(D, M, t, k, j, xt, yt, T);
        take(T, true);
      }
    }
  } else {
    const int nmax = __reduce_max_sync(all, deg);
    for (int j = 0; j < nmax; j += L) {
      TermF T = {};
      if (j + q < deg) {
        if (sp) spf_entry<CSPM>(D, k, j + q, xt, yt, T);
        else nodef_entry<CSPM>(D, M, t, k, j + q, xt, yt, T);
      }
      const bool walls = __any_sync(all, T.wall);
#pragma unroll
      for (int o = 0; o < L; o++) {
        TermF x = {};
        x.wall = __shfl_sync(all, (int)T.wall, o, L);
        x.h = __shfl_sync(all, T.h, o, L);
        x.m = __shfl_sync(all, T.m, o, L);
        x.gx = __shfl_sync(all, T.gx, o, L);
        x.gy = __shfl_sync(all, T.gy, o, L);
        if (CSPM) {
          x.xu = __shfl_sync(all, T.xu, o, L);
          x.yu = __shfl_sync(all, T.yu, o, L);
          x.hx = __shfl_sync(all, T.hx, o, L);
          x.hy = __shfl_sync(all, T.hy, o, L);
        }
        if (walls) {
          x.push = __shfl_sync(all, (int)T.push, o, L);
          x.u = __shfl_sync(all, T.u, o, L);
          x.fx = __shfl_sync(all, T.fx, o, L);
          x.fy = __shfl_sync(all, T.fy, o, L);
        }
        if (j + o < deg) take(x, !sp);
      }
    }
  }
  if (q || !act) return;
  if (!sp) {
    F.store(D, M, t);
    D.bc_int[t] = F.bc_int;
    D.msum[k - ns] = make_float4(sx.hi.s, sx.lo - sx.hi.c, sy.hi.s, sy.lo - sy.hi.c);
  }
  const float norm = nm.fval();
  D.normf[k] = make_float2(norm, norm != 0.0f ? __frcp_rn(norm) : 0.0f);
  if (CSPM) {
    const double AE[4] = {e0.val(), e1.val(), e2.val(), e3.val()};
    double A[5];
    cspm_moments<true>(D, AE, A);
    for (int q = 0; q < 5; q++) D.AE[(size_t)q * D.NT + k] = A[q];
  }
  if (sp) {
    double a = D.s0[t], b = D.s1[t], c = D.s2[t], d = D.s3[t];
    st4(D.st0c + 4 * (size_t)k, a, b, c, d);
    a = a + 0.0;  // RK4 starts from zero rates
    b = b + 0.0;
    c = c + 0.0;
    d = d + 0.0;
    spf_publish(D, M, *scp, k, t, 0, a, b, c, d, false);
  } else {
    const double v0x = D.vx[t], v0y = D.vy[t];
    D.vx0[t] = v0x;
    D.vy0[t] = v0y;
    double vx = v0x + 0.0, vy = v0y + 0.0, a = 0.0, b = 0.0, c = 0.0, d = 0.0;
    if (norm == 0.0f) {  // no stress-point in reach: RK4 clears the stress, nothing sets it
      apply_bcs(D, *scp, t, vx, vy, a, b, c, d);
      D.s0[t] = a;
      D.s1[t] = b;
      D.s2[t] = c;
      D.s3[t] = d;
      vx = 0.0;
      vy = 0.0;
    }
    apply_bcs(D, *scp, t, vx, vy, a, b, c, d);
    D.recV[t] = split2f(vx, vy);
    // the correction's right-hand side takes the stage velocity in FP64 (its own node's only)
    if (CSPM) reinterpret_cast<double2*>(D.pv[0])[t] = make_double2(vx, vy);
  }
}

// The interpolated velocity of a stress-point (k_finterp): the first node's velocity plus the
// weighted mean of the deviations
template <int KP>
__device__ __forceinline__ void sp_velocity(const Dev& D, int k, int deg,
                                            const float4* __restrict__ rv, double& vx,
                                            double& vy) {
  Kahan v0, v1;
  bool have = false;
  float4 ref = make_float4(0.f, 0.f, 0.f, 0.f);
  walk_compact<KP, float4>(
      D.crossW, k, D.N2, deg,
      [&](const int2& e) { return e.y >= 0 ? rv[e.x] : make_float4(0.f, 0.f, 0.f, 0.f); },
      [&](const int2& e, const float4& r) {
        if (e.y < 0) return;
        if (!have) {
          ref = r;
          have = true;
        }
        const float h2 = __int_as_float(e.y);
        v0.add(dfdiff(r.x, r.z, ref.x, ref.z) * h2);
        v1.add(dfdiff(r.y, r.w, ref.y, ref.w) * h2);
      });
  vx = 0.0;
  vy = 0.0;
  const float2 nf = D.normf[k];
  if (nf.x != 0.0f) {
    vx = (f64_of(ref.x) + f64_of(ref.z)) + f64_of(v0.fval() * nf.y);
    vy = (f64_of(ref.y) + f64_of(ref.w)) + f64_of(v1.fval() * nf.y);
  }
}

// entry j of column k of the compact list and its gradient constants
struct EntG {
  int2 w;
  float2 g;
};
__device__ __forceinline__ EntG ent_g(const Dev& D, int j, int k) {
  EntG e;
  e.w = D.crossW[(size_t)j * D.N2 + k];
  e.g = D.hGf[(size_t)j * D.NT + k];
  return e;
}
// the derivative sums' walk (walk_list over the compact entries and their gradients)
template <int KP, typename Rec, typename Load, typename Sum>
__device__ __forceinline__ void walk_g(const Dev& D, int k, int deg, Load&& load, Sum&& sum) {
  EntG nxt[KP];
  const EntG none = {make_int2(0, 0), make_float2(0.f, 0.f)};
#pragma unroll
  for (int q = 0; q < KP; q++) nxt[q] = q < deg ? ent_g(D, q, k) : none;
  for (int j = 0; j < deg; j += KP) {
    EntG cur[KP];
    Rec rec[KP] = {};
#pragma unroll
    for (int q = 0; q < KP; q++) {
      cur[q] = nxt[q];
      if (j + q < deg) rec[q] = load(cur[q].w);
    }
#pragma unroll
    for (int q = 0; q < KP; q++) nxt[q] = j + KP + q < deg ? ent_g(D, j + KP + q, k) : none;
#pragma unroll
    for (int q = 0; q < KP; q++)
      if (j + q < deg) sum(cur[q], rec[q], j + q);
  }
}

// from a stage's rates: the RK sum and the next stage's stress, or after the last stage the
// end of RK4 (2_SPH_main_2018.f90:784-799) and update_strain
__device__ __forceinline__ void spf_advance(const Dev& D, const Real& M, const StepScalars& sc,
                                            int stage, int k, int t, const double* rhs,
                                            double der) {
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
#pragma unroll
  for (int i = 0; i < 4; i++) rk[i] = fma(f2, rhs[i], rk[i]);
  rd = rd + der * f2;
  const d4 s0 = ld4(D.st0c + 4 * (size_t)k);
  const int nxt = (stage & 1) ^ 1;
  if (stage < 3) {
    st4(rks, rk[0], rk[1], rk[2], rk[3]);
    D.RKd[k] = rd;
    const double f1dt = (stage == 2 ? 1.0 : 0.5) * M.dt;  // RK4 nodes 1/2, 1/2, 1
    double a = mad2(s0.a, f1dt, rhs[0]), b = mad2(s0.b, f1dt, rhs[1]),
           c = mad2(s0.c, f1dt, rhs[2]), d = mad2(s0.d, f1dt, rhs[3]);
    spf_publish(D, M, sc, k, t, nxt, a, b, c, d, false);
  } else {
    const double dt6 = M.dt6;
    double a = mad2(s0.a, dt6, rk[0]), b = mad2(s0.b, dt6, rk[1]), c = mad2(s0.c, dt6, rk[2]),
           d = mad2(s0.d, dt6, rk[3]);
    spf_publish(D, M, sc, k, t, nxt, a, b, c, d, true);
    D.s0[t] = a;
    D.s1[t] = b;
    D.s2[t] = c;
    D.s3[t] = d;
    const int ex = (int)((__double_as_longlong(rd) >> 52) & 0x7FF);
    const double dd = (ex > 64 && ex < 1980) ? div_rcp(rd, 6.0, 1.0 / 6.0)
                      : (__double_as_longlong(rd) << 1) == 0 ? rd : rd / 6.0;
    D.Ddev[t] = dd;
    const double iv = mad2(D.iv1[t], M.dt, dd);
    D.iv1[t] = iv;
    D.recI[t] = make_float4(f32_rn(iv), f32_rn(D.vol[t]), f32_rn(D.rho[t]), f32_rn(D.mass[t]));
  }
}

// The wall terms are rare and FP64: out of line, because the compiler turns so short a branch
// into predicated instructions, which occupy the FP64 pipe for every entry (58% of its cycles,
// 0.11 ms against 0.05 a stage at 322k particles).
// v - v (1 - beta) of a stress-point next to a wall
static __device__ __noinline__ float2 wall_du(double vx, double vy, double ob) {
  return make_float2((float)(vx - vx * ob), (float)(vy - vy * ob));
}
// a node's dummy partner carries the node's stress: A_u - A_t = sigma_t / rho_d^2 - sigma_t /
// rho_t^2
static __device__ __noinline__ float3 wall_dA(double s0, double s1, double s2, double rd, double rt) {
  const double ri2 = rd * rd, rt2 = rt * rt;
  return make_float3((float)fma(s0, ri2, -(s0 * rt2)), (float)fma(s1, ri2, -(s1 * rt2)),
                     (float)fma(s2, ri2, -(s2 * rt2)));
}

template <int KP, bool LEAN>
__device__ __forceinline__ void spf_stage(const Dev& D, int stage, int k) {
  const int ns = D.NT - D.NN;
  const int t = D.colid[k];
  const float4* __restrict__ rv = (stage & 1) ? D.recV1 : D.recV;
  const int deg = D.degC[k];
  const Real* Mp;
  const StepScalars* scp;
  load_real(D, t, Mp, scp);
  const Real& M = *Mp;
  double vtx, vty;
  sp_velocity<KP>(D, k, deg, rv, vtx, vty);
  if (D.no_bcs > 0) {
    double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
    apply_bcs(D, *scp, t, vtx, vty, a, b, c, d);
  }
  Kahan g0, g1, g2, g3;
  float vh0, vh1, vl0, vl1;
  f32_split(vtx, vh0, vl0);
  f32_split(vty, vh1, vl1);
  walk_g<(KP > 2 ? 2 : 1), float4>(
      D, k, deg,
      [&](const int2& e) { return e.y >= 0 ? rv[e.x] : make_float4(0.f, 0.f, 0.f, 0.f); },
      [&](const EntG& e, const float4& r, int j) {
        const float h1 = e.g.x, h2 = e.g.y;
        float du0, du1;
        if (e.w.y >= 0) {
          du0 = dfdiff(r.x, r.z, vh0, vl0);
          du1 = dfdiff(r.y, r.w, vh1, vl1);
        } else {  // a dummy partner: v - v (1 - beta)
          const float2 du = wall_du(vtx, vty, D.hB[(size_t)j * ns + k]);
          du0 = du.x;
          du1 = du.y;
        }
        g0.add(du0 * h1);
        g2.add(du0 * h2);
        g1.add(du1 * h1);
        g3.add(du1 * h2);
      });
  const d4 own = ld4(D.stc + 4 * (size_t)k);
  const double st[4] = {own.a, own.b, own.c, own.d};
  double g[4];
  float h11 = g0.fval(), h21 = g1.fval(), h12 = g2.fval(), h22 = g3.fval();
  if (D.cspm) {
    g[0] = g0.val();
    g[1] = g1.val();
    g[2] = g2.val();
    g[3] = g3.val();
    double A[5];
    for (int i = 0; i < 5; i++) A[i] = D.AE[(size_t)i * D.NT + k];
    cspm_correct<2, true>(A, g);
    h11 = f32_rn(g[0]);
    h21 = f32_rn(g[1]);
    h12 = f32_rn(g[2]);
    h22 = f32_rn(g[3]);
  } else if (!LEAN || D.surr) {
    g[0] = f64_of(h11);
    g[1] = f64_of(h21);
    g[2] = f64_of(h12);
    g[3] = f64_of(h22);
  }
  if (D.surr && D.surr_gate->on) {  // the network runs in this step: k_fstail finishes
    for (int i = 0; i < 4; i++) D.grad_u[4 * (size_t)t + i] = g[i];
    return;
  }
  double rhs[4], der = 0.0;
  if (LEAN) sp_rates_lean(D, M, *scp, t, h11, h21, h12, h22, st, rhs, der);
  else sp_rates_fast(D, M, *scp, t, g, st, nullptr, 0.0, nullptr, rhs, der);
  spf_advance(D, M, *scp, stage, k, t, rhs, der);
}

// the interpolated stress of a node (k_finterp); iv: the internal variable too (only the
// step's last interpolation leaves it behind)
template <int KP, bool IV>
__device__ __forceinline__ void node_stress(const Dev& D, int k, int deg,
                                            const float4* __restrict__ rs, float* s, float* ivm) {
  struct Rec {
    float4 s;
    float iv;
  };
  Kahan a, b, c, d, iv;
  walk_compact<KP, Rec>(
      D.crossW, k, D.N2, deg,
      [&](const int2& e) {
        Rec r = {make_float4(0.f, 0.f, 0.f, 0.f), 0.f};
        if (e.y >= 0) {
          r.s = rs[e.x];
          if (IV) r.iv = D.recI[e.x].x;
        }
        return r;
      },
      [&](const int2& e, const Rec& r) {
        if (e.y < 0) return;
        const float h1 = __int_as_float(e.y);
        a.add(r.s.x * h1);
        b.add(r.s.y * h1);
        c.add(r.s.z * h1);
        d.add(r.s.w * h1);
        if (IV) iv.add(r.iv * h1);
      });
  const float rn = D.normf[k].y;
  s[0] = a.fval() * rn;
  s[1] = b.fval() * rn;
  s[2] = c.fval() * rn;
  s[3] = d.fval() * rn;
  if (IV) *ivm = iv.fval() * rn;
}

template <int KP, int KD>
__device__ __forceinline__ void nodef_stage(const Dev& D, int stage, int k) {
  const int ns = D.NT - D.NN, cur = stage & 1;
  const int t = D.colid[k];
  const int deg = D.degC[k];
  const float4* __restrict__ rA = cur ? D.recA1 : D.recA;
  const float4* __restrict__ rL = cur ? D.recAl1 : D.recAl;
  const Real* Mp;
  const StepScalars* scp;
  load_real(D, t, Mp, scp);
  const Real& M = *Mp;
  const float norm = D.normf[k].x;
  double s[4];
  {
    float sf[4];
    node_stress<KP, false>(D, k, deg, cur ? D.recS1 : D.recS, sf, nullptr);
    for (int i = 0; i < 4; i++) s[i] = f64_of(sf[i]);
  }
  const float4 vr = (cur ? D.recV1 : D.recV)[t];  // the stage velocity, hi and lo
  double vdx = 0.0, vdy = 0.0;
  if (norm == 0.0f) {  // the stress of the last return, its BCs applied at the stage's start
    s[0] = D.s0[t];
    s[1] = D.s1[t];
    s[2] = D.s2[t];
    s[3] = D.s3[t];
    if (stage > 0) apply_bcs(D, *scp, t, vdx, vdy, s[0], s[1], s[2], s[3]);
  }
  retf(M, s[0], s[1], s[2], s[3]);
  apply_bcs(D, *scp, t, vdx, vdy, s[0], s[1], s[2], s[3]);
  if (norm == 0.0f) {
    D.s0[t] = s[0];
    D.s1[t] = s[1];
    D.s2[t] = s[2];
    D.s3[t] = s[3];
  }
  float4 ah, al;
  split_A(D, t, s[0], s[1], s[2], ah, al);
  Kahan q0, q1, q2, q3, q4, q5;
  walk_g<KD, RecA>(
      D, k, deg,
      [&](const int2& e) {
        RecA r = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        if (e.y >= 0) {
          r.a = rA[e.x];
          r.l = rL[e.x];
        }
        return r;
      },
      [&](const EntG& e, const RecA& r, int) {
        float d0, d1, d2;
        if (e.w.y >= 0) {
          d0 = dfdiff(r.a.x, r.l.x, ah.x, al.x);
          d1 = dfdiff(r.a.y, r.l.y, ah.y, al.y);
          d2 = dfdiff(r.a.z, r.l.z, ah.z, al.z);
        } else {
          const float3 dA = wall_dA(s[0], s[1], s[2], D.rinv[e.w.x], D.rinv[t]);
          d0 = dA.x;
          d1 = dA.y;
          d2 = dA.z;
        }
        const float mx = e.g.x, my = e.g.y;
        q0.add(mx * d0);
        q1.add(mx * d1);
        q2.add(mx * d2);
        q3.add(my * d0);
        q4.add(my * d1);
        q5.add(my * d2);
      });
  float avx = 0.0f, avy = 0.0f;
  // alpha > 0 or beta > 0 (non-negative doubles: a positive one has a positive bit pattern)
  if (__double_as_longlong(M.alpha) > 0 || __double_as_longlong(M.beta) > 0) {
    // artificial_viscosity (2_SPH_main_2018.f90:826-904) in FP32
    Kahan ax, ay;
    const int degs = D.degS[k];
    const float4* __restrict__ rv = cur ? D.recV1 : D.recV;
    const double xt = D.px[t], yt = D.py[t];
    const float ht = f32_rn(D.hsml[t]), rt = f32_rn(D.rho[t]);
    for (int j = 0; j < degs; j++) {
      const int4 e = D.same[ell(j, k, D.N2)];
      const int u = e.x;
      const float4 r = rv[u];
      const float4 ri = D.recI[u];
      const float xij = f32_rn(xt - D.px[u]);
      const float yij = f32_rn(yt - D.py[u]);
      const float h = 0.5f * (ht + f32_rn(D.hsml[u]));
      const float rho2 = 0.5f * (rt + ri.z);
      const float div_u = xij * dfdiff(vr.x, vr.z, r.x, r.z) + yij * dfdiff(vr.y, vr.w, r.y, r.w);
      const float sq2 = xij * xij + yij * yij;
      const float theta = (h * div_u) / (sq2 + 0.01f * (h * h));
      float visc = 0.0f;
      if (div_u < 0)
        visc = (-((float)M.alpha * 600.0f) * theta + (float)M.beta * (theta * theta)) / rho2;
      ax.add(visc * __int_as_float(e.z) * ri.w);
      ay.add(visc * __int_as_float(e.w) * ri.w);
    }
    avx = -ax.fval();
    avy = -ay.fval();
  }
  // g2 = -(q + 2 A_t S) in FP32: A_t (hi + lo) times S (hi + lo) as a double-float product, so
  // that the large, nearly cancelling part 2 A_t S keeps FP32 accuracy relative to the result
  const float4 S = D.msum[k - ns];
  auto g2of = [](float q, float ah_, float al_, float sh, float sl) {
    const float p = ah_ * sh;
    const float e = fmaf(ah_, sl, fmaf(al_, sh, fmaf(ah_, sh, -p)));
    return -(fmaf(2.0f, p, q) + 2.0f * e);
  };
  float g2v[6];
  g2v[0] = g2of(q0.fval(), ah.x, al.x, S.x, S.y);
  g2v[1] = g2of(q1.fval(), ah.y, al.y, S.x, S.y);
  g2v[2] = g2of(q2.fval(), ah.z, al.z, S.x, S.y);
  g2v[3] = g2of(q3.fval(), ah.x, al.x, S.z, S.w);
  g2v[4] = g2of(q4.fval(), ah.y, al.y, S.z, S.w);
  g2v[5] = g2of(q5.fval(), ah.z, al.z, S.z, S.w);
  double rx, ry;
  if (D.cspm) {  // the CSPM correction in FP64 (the reference's form)
    double g2d[6];
    for (int q = 0; q < 6; q++) g2d[q] = f64_of(g2v[q]);
    double A[5];
    for (int i = 0; i < 5; i++) A[i] = D.AE[(size_t)i * D.NT + k];
    cspm_correct<3, true>(A, g2d);
    const double2 vt = reinterpret_cast<const double2*>(D.pv[0])[t];
    node_rhs_f64(D, M, *scp, t, g2d, vt.x, vt.y, f64_of(avx), f64_of(avy), 0.0, 0.0, rx, ry);
  } else {
    // tail_node in FP32: the divergence, gravity with damping and the right-hand side carry
    // the FP32 accuracy of the sums they come from
    const float div2x = -(g2v[0] + g2v[5]);
    const float div2y = -(g2v[2] + g2v[4]);
    float gx = 0.0f, gy = 0.0f;
    if (M.ic_grav == 1) {
      const float fg = f32_rn(scp->factg);
      gx = fg * f32_rn(M.cgrav[0]);
      gy = fg * f32_rn(M.cgrav[1]);
    }
    if ((__double_as_longlong(M.damping) << 1) != 0) {  // non-zero, on the integer pipe
      const float dmp = f32_rn(M.damping);
      gx = fmaf(-dmp, vr.x, gx);
      gy = fmaf(-dmp, vr.y, gy);
    }
    rx = f64_of(((-div2x + gx) + avx) + f32_rn(D.fbx[t]));
    ry = f64_of(((-div2y + gy) + avy) + f32_rn(D.fby[t]));
  }
  const double f2 = (stage == 1 || stage == 2) ? 2.0 : 1.0;
  double kx = 0.0, ky = 0.0;
  if (stage > 0) {
    kx = D.RKv[0][t];
    ky = D.RKv[1][t];
  }
  kx = fma(f2, rx, kx);
  ky = fma(f2, ry, ky);
  const double v0x = D.vx0[t], v0y = D.vy0[t];
  double nx, ny;
  if (stage < 3) {
    D.RKv[0][t] = kx;
    D.RKv[1][t] = ky;
    const double f1dt = (stage == 2 ? 1.0 : 0.5) * M.dt;
    nx = mad2(v0x, f1dt, rx);
    ny = mad2(v0y, f1dt, ry);
  } else {
    nx = mad2(v0x, M.dt6, kx);
    ny = mad2(v0y, M.dt6, ky);
  }
  if (norm == 0.0f) {
    nx = 0.0;
    ny = 0.0;
  }
  double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
  apply_bcs(D, *scp, t, nx, ny, a, b, c, d);
  (cur ? D.recV : D.recV1)[t] = split2f(nx, ny);
  if (D.cspm) reinterpret_cast<double2*>(D.pv[0])[t] = make_double2(nx, ny);
  if (stage == 3) {
    D.vx[t] = nx;
    D.vy[t] = ny;
  }
}

// RK4 stage (2_SPH_main_2018.f90:700-777): blocks [0, nbs) the stress-points, the rest the
// nodes
// MINB: blocks of 128 an SM must hold.  Large problems wait on the record gathers (18 resident
// warps of 64 issue a quarter of the cycles), so 64 registers and some spills pay: a stage at
// 2.0M particles takes 0.409 ms at 96 registers, 0.364 at 80, 0.340 at 72, 0.327 at 64 and
// 0.340 at 56.  Small ones cannot fill the SMs anyway and keep their registers (10k particles:
// 25 us against 27).
template <int KP, int KD, bool LEAN, int MINB>
__global__ void __launch_bounds__(128, MINB) k_fstage(Dev D, int stage, int nbs) {
  const int ns = D.NT - D.NN;
  if ((int)blockIdx.x < nbs) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < ns) spf_stage<KP, LEAN>(D, stage, k);
  } else {
    const int k = (blockIdx.x - nbs) * blockDim.x + threadIdx.x;
    if (k < D.NN) nodef_stage<KP, KD>(D, stage, ns + k);
  }
}

// the stress-points' rates of a stage after the network has run (surr_answer), in a step
// whose gate is open
__global__ void __launch_bounds__(128) k_fstail(Dev D, int stage) {
  if (!D.surr_gate->on) return;
  const int ns = D.NT - D.NN;
  for (int base = blockIdx.x * blockDim.x; base < ns; base += gridDim.x * blockDim.x) {
    const int k = base + threadIdx.x;
    const bool act = k < ns;
    const int kk = act ? k : 0;
    const int t = D.colid[kk];
    const Real* Mp;
    const StepScalars* scp;
    load_real(D, t, Mp, scp);
    const d4 own = ld4(D.stc + 4 * (size_t)kk);
    const double st[4] = {own.a, own.b, own.c, own.d};
    double g[4] = {0.0, 0.0, 0.0, 0.0}, Gnet[4], dp[9], dn = 0.0;
    bool have_dp = false;
    const bool accept = surr_answer(D, *Mp, *scp, act, kk, t, st, g, Gnet, dn, dp, have_dp);
    if (!act) continue;
    double rhs[4], der = 0.0;
    sp_rates_fast(D, *Mp, *scp, t, D.grad_u + 4 * (size_t)t, st, accept ? Gnet : nullptr, dn,
                  have_dp ? dp : nullptr, rhs, der);
    spf_advance(D, *Mp, *scp, stage, k, t, rhs, der);
  }
}

// the final interpolation, return and BCs (2_SPH_main_2018.f90:130-135), then the position
// update (:140-146, without XSPH) and the displacements (:166-180)
template <int KP>
__global__ void __launch_bounds__(128) k_ffinish(Dev D) {
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
  const Real* Mp;
  const StepScalars* scp;
  load_real(D, t, Mp, scp);
  const Real& M = *Mp;
  double vx, vy, vx0, vy0;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  if (k < ns) {
    sp_velocity<KP>(D, k, deg, D.recV, vx, vy);
    apply_bcs(D, *scp, t, vx, vy, s[0], s[1], s[2], s[3]);
    vx0 = D.vx[t];
    vy0 = D.vy[t];
    D.vx0[t] = vx0;
    D.vy0[t] = vy0;
    D.vx[t] = vx;
    D.vy[t] = vy;
    if (D.xsph) D.recV[t] = split2f(vx, vy);
  } else {
    float sf[4], iv;
    node_stress<KP, true>(D, k, deg, D.recS, sf, &iv);
    const float norm = D.normf[k].x;
    vx = D.vx[t];
    vy = D.vy[t];
    if (norm != 0.0f) {
      for (int i = 0; i < 4; i++) s[i] = f64_of(sf[i]);
      D.iv1[t] = f64_of(iv);
    } else {  // RK4's last BCs, then no interpolated stress
      s[0] = D.s0[t];
      s[1] = D.s1[t];
      s[2] = D.s2[t];
      s[3] = D.s3[t];
      apply_bcs(D, *scp, t, vx, vy, s[0], s[1], s[2], s[3]);
      vx = 0.0;
      vy = 0.0;
    }
    retf(M, s[0], s[1], s[2], s[3]);
    apply_bcs(D, *scp, t, vx, vy, s[0], s[1], s[2], s[3]);
    D.s0[t] = s[0];
    D.s1[t] = s[1];
    D.s2[t] = s[2];
    D.s3[t] = s[3];
    D.vx[t] = vx;
    D.vy[t] = vy;
    vx0 = D.vx0[t];
    vy0 = D.vy0[t];
  }
  move_particle(D, M, t, k >= ns, vx0, vy0, vx, vy);
}

template <int KP, int KD>
void launch_fstage_kp(Ctx& c, int stage) {
  const Dev& D = c.d;
  const int ns = D.NT - D.NN;
  const int b = c.block_for(D.NT, std::min(c.blk[TK_DERIVS], 128));
  const int nbs = (ns + b - 1) / b, nbn = (D.NN + b - 1) / b;
  const int nb = nbs + nbn;
  // up to eight blocks an SM in all, a tighter bound on the registers adds no resident block
  const bool small = D.NT <= 152 * 8 * 128;
  if (c.lean_tail && !D.cap_buf) {
    if (small) k_fstage<KP, KD, true, 1><<<nb, b, 0, c.stream>>>(D, stage, nbs);
    else k_fstage<KP, KD, true, 8><<<nb, b, 0, c.stream>>>(D, stage, nbs);
  } else {
    if (small) k_fstage<KP, KD, false, 1><<<nb, b, 0, c.stream>>>(D, stage, nbs);
    else k_fstage<KP, KD, false, 8><<<nb, b, 0, c.stream>>>(D, stage, nbs);
  }
}

}  // namespace

void launch_fprep(Ctx& c) {
  Dev D = c.d;
  if (c.reinterpolates()) D.walk_order = 0;  // done
  D.same_entries = c.same_now();  // the lists to put in walk order
  const bool group = D.NT <= c.group_max;
  const int n = group ? 8 * D.NT : D.NT, b = c.block_for(n, 128), nb = (n + b - 1) / b;
  auto k = D.cspm ? (group ? k_fprep<8, true> : k_fprep<1, true>)
                  : (group ? k_fprep<8, false> : k_fprep<1, false>);
  k<<<nb, b, 0, c.stream>>>(D);
}

// The look-ahead of the interpolation (ahead[0]) sets the pair; the node derivative sums'
// (ahead[1]) follows it where a kernel of that pair exists (results do not depend on either)
void launch_fstage(Ctx& c, int stage) {
  if (c.ahead[0] == 8) launch_fstage_kp<8, 4>(c, stage);
  else if (c.ahead[0] == 4) launch_fstage_kp<4, 2>(c, stage);
  else if (c.ahead[1] == 1) launch_fstage_kp<2, 1>(c, stage);
  else launch_fstage_kp<2, 2>(c, stage);
  const int ns = c.d.NT - c.d.NN;
  if (c.d.surr && ns > 0) {
    launch_fsp_cand(c, stage, true);
    c.kernels_launched += 1;
    k_fstail<<<std::min((ns + 127) / 128, 152 * 8), 128, 0, c.stream>>>(c.d, stage);
  }
}

void launch_ffinish(Ctx& c) {
  const int b = c.block_for(c.d.N2, 128);
  const int nb = (c.d.N2 + b - 1) / b;
  if (c.ahead[0] == 8) k_ffinish<8><<<nb, b, 0, c.stream>>>(c.d);
  else if (c.ahead[0] == 4) k_ffinish<4><<<nb, b, 0, c.stream>>>(c.d);
  else k_ffinish<2><<<nb, b, 0, c.stream>>>(c.d);
}

}  // namespace sps
