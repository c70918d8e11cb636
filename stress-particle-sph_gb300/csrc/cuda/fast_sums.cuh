// fast_sums.cuh -- the FP32 form's neighbour sums: compensated FP32 sums, double-float
// differences, the software-pipelined list walks and the stress-point rates with and without
// the learned surrogate, shared by the separate kernels (fast_step.cu) and the one-launch
// stages (fast_fused.cu).
#pragma once
#include "stage_tail.cuh"

namespace sps {

struct Kahan {
  float s = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(float x) {
    float y = x - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double val() const { return (double)s - (double)c; }
  // the compensated sum rounded to FP32
  __device__ __forceinline__ float fval() const { return s - c; }
};

// sum of exact FP32 products: p = RN(a b) and e = a b - p (exact, by one FMA: the
// error-free product transformation of Ogita, Rump and Oishi, "Accurate sum and dot
// product", SIAM J. Sci. Comput. 26(6), 2005); p is Kahan-summed, e summed plainly
struct ProdSum {
  Kahan hi;
  float lo = 0.0f;
  __device__ __forceinline__ void add(float a, float b) {
    float p = a * b;
    float e = fmaf(a, b, -p);
    hi.add(p);
    lo += e;
  }
};

// difference of two double-float values (hi + lo) in FP32
__device__ __forceinline__ float dfdiff(float ah, float al, float bh, float bl) {
  return (ah - bh) + (al - bl);
}

// Walks entries 0 .. deg of list column col, KP entries a pass, software-pipelined: the
// next pass's entries are loaded while the current pass's records are gathered and summed,
// so that the entry loads (streamed from DRAM) overlap the record gathers (mostly L2 hits)
// instead of adding their latency to them.  load(e) returns the records of entry e (called
// only for entries below deg), sum(e, rec) adds one term; terms are added in list order,
// so the result does not depend on KP.
template <int KP, typename Rec, typename Load, typename Sum>
__device__ __forceinline__ void walk_list(const int4* __restrict__ list, int col, int N2,
                                          int deg, Load&& load, Sum&& sum) {
  int4 nxt[KP];
#pragma unroll
  for (int q = 0; q < KP; q++)
    nxt[q] = q < deg ? list[ell(q, col, N2)] : make_int4(0, 0, 0, 0);
  for (int k = 0; k < deg; k += KP) {
    int4 cur[KP];
    Rec rec[KP] = {};
#pragma unroll
    for (int q = 0; q < KP; q++) {
      cur[q] = nxt[q];
      if (k + q < deg) rec[q] = load(cur[q]);
    }
#pragma unroll
    for (int q = 0; q < KP; q++)
      nxt[q] = k + KP + q < deg ? list[ell(k + KP + q, col, N2)] : make_int4(0, 0, 0, 0);
#pragma unroll
    for (int q = 0; q < KP; q++)
      if (k + q < deg) sum(cur[q], rec[q]);
  }
}

// the same walk over the compact {id, W} entries (crossW: entry k of column col at
// k * N2 + col)
template <int KP, typename Rec, typename Load, typename Sum>
__device__ __forceinline__ void walk_compact(const int2* __restrict__ list, int col, int N2,
                                             int deg, Load&& load, Sum&& sum) {
  int2 nxt[KP];
#pragma unroll
  for (int q = 0; q < KP; q++) nxt[q] = q < deg ? list[(size_t)q * N2 + col] : make_int2(0, 0);
  for (int k = 0; k < deg; k += KP) {
    int2 cur[KP];
    Rec rec[KP] = {};
#pragma unroll
    for (int q = 0; q < KP; q++) {
      cur[q] = nxt[q];
      if (k + q < deg) rec[q] = load(cur[q]);
    }
#pragma unroll
    for (int q = 0; q < KP; q++)
      nxt[q] = k + KP + q < deg ? list[(size_t)(k + KP + q) * N2 + col] : make_int2(0, 0);
#pragma unroll
    for (int q = 0; q < KP; q++)
      if (k + q < deg) sum(cur[q], rec[q]);
  }
}

// records of one neighbour, as the four sums read them
struct RecVI {  // velocity (hi, lo) and m / rho
  float4 v;
  float vol;
};
struct RecSI {  // stress and {intvar1, m / rho, rho, m}
  float4 s, i;
};
struct RecA {  // sigma / rho^2 (hi with m, lo)
  float4 a, l;
};

// the stress-point rates without the network, for the Drucker-Prager plane strain case (every
// realisation: ntype_eco > 1, ncrit 12, ntype_solid != 1, no continuity density, no training
// capture; the host checks): the arithmetic of sp_rates_fast with the flow rule's outputs
// kept as the FP32 values they are (fewer registers, no FP64 copies); g: grad_u(a,b) in FP32
__device__ __forceinline__ void sp_rates_lean(const Dev& D, const Real& M, const StepScalars& sc,
                                              int t, float h11, float h21, float h12, float h22,
                                              const double* st, double* rhs, double& der) {
  double f = D.fdp[t];
  float G[4], vv[4];
  drucker_prager_f32g(M, sc.time_sph, st, h11, h21, h12, h22, &f, G, vv);
  D.fdp[t] = f;
  // explicit fmaf: the same rounding as sp_rates_fast
  const float q = fmaf(2.0f, fmaf(vv[0], vv[0], fmaf(vv[1], vv[1], __fmul_rn(vv[3], vv[3]))),
                       __fmul_rn(vv[2], vv[2]));
  der = f64_of(sqrtf(__fmul_rn(q, 1.0f / 3.0f)));
  float r[4];
  r[0] = fmaf(M.D11f, h11, M.D12f * h22);
  r[1] = fmaf(M.D12f, h11, M.D22f * h22);
  r[2] = M.D33f * (h21 + h12);
  r[3] = fmaf(M.D41f, h11, M.D42f * h22);
  if (D.update_x) {
    const float om1 = 0.5f * (h12 - h21);
    const float t0 = f32_rn(st[0]), t1 = f32_rn(st[1]), t2 = f32_rn(st[2]);
    r[0] = fmaf(2.0f * om1, t2, r[0]);
    r[1] = fmaf(-2.0f * om1, t2, r[1]);
    r[2] = fmaf(om1, t1 - t0, r[2]);
  }
#pragma unroll
  for (int k = 0; k < 4; k++) rhs[k] = f64_of(r[k] + -G[k]);
}

// The surrogate's view of stress-point t: the exact rule (drucker_prager, whose results dp
// = {G, vivel, f} the tail reuses), whether it is loading, and for a loading point the
// network's inputs x, their output scale and whether they lie in the training envelope.
// Deterministic, so k_fsp_cand and k_fsp_tail<true> reach the same decisions.
__device__ __forceinline__ void surr_front(const Dev& D, const Real& M, const StepScalars& sc,
                                           int t, const double* st, double* g, double* s2v,
                                           float* x, double& scale, bool& loading, bool& cand,
                                           double* dp) {
  const double* gu = D.grad_u + 4 * (size_t)t;
  for (int k = 0; k < 4; k++) g[k] = gu[k];
  for (int k = 0; k < 4; k++) s2v[k] = st[k];
  if (M.ntype_solid == 1) s2v[3] = M.poiss * (s2v[0] + s2v[1]);
  double f = D.fdp[t], G2[4], vivel[4];
  drucker_prager_f32(M, sc.time_sph, s2v, g, &f, G2, vivel);  // the exact rule
  loading = G2[0] != 0.0 || G2[1] != 0.0 || G2[2] != 0.0 || G2[3] != 0.0;
  for (int k = 0; k < 4; k++) {
    dp[k] = G2[k];
    dp[4 + k] = vivel[k];
  }
  dp[8] = f;
  scale = 0.0;
  cand = false;
  if (loading) {
    scale = mlp_features(s2v, g, M.tanfi, M.coh, M.young, M.poiss, D.rho[t], x);
    cand = scale > 0.0;
    for (int k = 0; k < MLP_NIN && cand; k++) cand = x[k] >= D.env_lo[k] && x[k] <= D.env_hi[k];
  }
}

// The network's answer for one stress-point, row i of the candidates (the warp's 32 lanes call
// it together): surr_front again (its results in g, s2v, dp), the candidate's prediction
// (computed by the tensor-core kernel from the row that k_fsp_cand appended this stage), the
// drift test and the counters.  Returns whether the prediction Gnet (with its plastic strain
// rate der) is kept.
__device__ __forceinline__ bool surr_answer(const Dev& D, const Real& M, const StepScalars& sc,
                                            bool act, int i, int t, const double* st, double* g,
                                            double* Gnet, double& der, double* dp,
                                            bool& have_dp) {
  double s2v[4] = {0.0, 0.0, 0.0, 0.0};
  float x[16];
  double scale = 0.0;
  bool loading = false, cand = false;
  have_dp = false;
  if (act && M.ntype_eco > 1 && M.ncrit == 12) {
    surr_front(D, M, sc, t, st, g, s2v, x, scale, loading, cand, dp);
    have_dp = true;
  }
  bool accept = false;
  if (cand) {
    const float* y = D.ycand + 4 * (size_t)D.cand_row[i];
    bool inside = true;
    for (int k = 0; k < MLP_NOUT; k++) {
      const float yk = y[k];
      inside = inside && fabsf(yk) <= 1.5f * D.out_max;
      Gnet[k] = (double)yk * scale;
    }
    if (inside) {
      // drift test in FP64
      double sm = ((s2v[0] + s2v[1]) + s2v[3]) / 3.0;
      double d0 = s2v[0] - sm, d1 = s2v[1] - sm, d2 = s2v[2], d3 = s2v[3] - sm;
      double sj = sqrt(d2 * d2 + 0.5 * ((d0 * d0 + d1 * d1) + d3 * d3));
      double e0 = M.D11 * g[0] + M.D12 * g[3] + Gnet[0];
      double e1 = M.D12 * g[0] + M.D22 * g[3] + Gnet[1];
      double e2 = M.D33 * g[1] + M.D33 * g[2] + Gnet[2];
      double e3 = M.D41 * g[0] + M.D42 * g[3] + Gnet[3];
      double df = (d0 * e0 + d1 * e1 + d3 * e3 + 2.0 * d2 * e2) / (2.0 * sj) +
                  M.alpha2 * (e0 + e1 + e3);
      accept = sj > 0.0 && M.dt * fabs(df) <= D.surr_tol * sj;
    } else {
      cand = false;  // counted as outside the envelope
    }
  }
  // counters: loading, answered, outside the envelope, drift-rejected
  unsigned ml = __ballot_sync(0xffffffffu, loading), ma = __ballot_sync(0xffffffffu, accept),
           mc = __ballot_sync(0xffffffffu, cand);
  if ((threadIdx.x & 31) == 0 && ml) {
    atomicAdd(&D.surr_cnt[0], (unsigned long long)__popc(ml));
    atomicAdd(&D.surr_cnt[1], (unsigned long long)__popc(ma));
    atomicAdd(&D.surr_cnt[2], (unsigned long long)(__popc(ml) - __popc(mc)));
    atomicAdd(&D.surr_cnt[3], (unsigned long long)(__popc(mc) - __popc(ma)));
  }
  if (accept) {
    // plastic strain rate of the predicted source: e_p = G / (2 G_mod), shear G / G_mod
    const double gm = M.young / (2.0 * (1.0 + M.poiss));
    double v0 = -Gnet[0] / (2.0 * gm), v1 = -Gnet[1] / (2.0 * gm), v2 = -Gnet[2] / gm,
           v3 = -Gnet[3] / (2.0 * gm);
    der = sqrt((2.0 * ((v0 * v0 + v1 * v1) + v3 * v3) + v2 * v2) / 3.0);
  }
  return accept;
}

}  // namespace sps
