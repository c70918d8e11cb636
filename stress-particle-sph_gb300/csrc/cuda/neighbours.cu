// neighbours.cu -- cell-linked neighbour search of the SPS step (compiled with -fmad=false).
//
// Restates grid_find_NEW (example_problems/soil_failure_bui_et_al_2008/
// 2_SPH_main_2018.f90:1199-1435), kernel (:1440) and Pint_Update
// (3_SPH_material_2018.f90:1574) as a GB300 pipeline:
//   k_bbox      Check_Out_Domain (:1170) + bounding box / max h over active particles; its last
//               block forms the grid parameters with the reference's arithmetic (:1245-1258)
//   k_cell_*    counting sort by cell and kind, then by particle id (the order list_picell
//               holds), with the list column of every particle
//   k_half      pairs created by each particle over the half stencil (self, +x, row
//               above), in the reference's creation order, with FP32-stored W and dW
//   k_lists     per-target neighbour lists in the reference's linked-list walk order
// The distance test r < scale_k*(h_i+h_j)/2 is decided on FP32 cell-frame coordinates
// with a guard band; candidates inside the band are re-tested with the exact FP64
// expression, so the pair set equals the reference's.
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>

#include "ctx.cuh"
#include "stage_tail.cuh"

namespace sps {

namespace {

constexpr int kBlock = 256;
// half-list entries: partner id in the low 28 bits, pair type (pint_type) in the top 4
constexpr int kHalfTypeShift = 28;
constexpr unsigned kHalfIdMask = (1u << kHalfTypeShift) - 1u;

// ---- double-float (unevaluated sum of two FP32 numbers) arithmetic: Dekker, "A floating-
// point technique for extending the available precision", Numer. Math. 18, 1971, with the
// FMA-based exact product.  Used by the FP32 form for the separations and r/h of its pairs
// (cubic_mixed).
__device__ __forceinline__ dfl df_fast2sum(float a, float b) {
  float s = a + b;
  return {s, b - (s - a)};
}
__device__ __forceinline__ dfl df_2sum(float a, float b) {
  float s = a + b;
  float bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ dfl df_mul(dfl x, dfl y) {
  float p = x.hi * y.hi;
  float e = fmaf(x.hi, y.hi, -p);
  e += x.hi * y.lo + x.lo * y.hi;
  return df_fast2sum(p, e);
}
__device__ __forceinline__ dfl df_sqrt(dfl x) {
  if (x.hi <= 0.0f) return {0.0f, 0.0f};
  float s = x.hi * rsqrtf(x.hi);  // approximate seed, corrected below
  float p = s * s;
  float e = fmaf(s, s, -p);
  float r = ((x.hi - p) - e) + x.lo;
  return df_fast2sum(s, r * (0.5f * __frcp_rn(s)));
}
// the same from the correctly rounded FP32 root: its error of 2^-25 leaves a correction that FP32
// carries to 2^-47 (the FP32 form keeps df_sqrt, and with it its kernel values' last bits)
__device__ __forceinline__ dfl df_sqrt_rn(dfl x) {
  const float s = __fsqrt_rn(x.hi);
  const float p = s * s;
  const float e = fmaf(s, s, -p);
  const float r = ((x.hi - p) - e) + x.lo;
  return df_fast2sum(s, r * (0.5f * __frcp_rn(s)));
}
// x^2 + y^2 of two double-float values, accurate to a few units of 2^-44: the exact
// squares of the high parts (FMA residuals) summed exactly, the cross terms and residuals
// added once; sign-symmetric in x and y
__device__ __forceinline__ dfl df_sumsq(dfl x, dfl y) {
  const float px = x.hi * x.hi, ex = fmaf(x.hi, x.hi, -px);
  const float py = y.hi * y.hi, ey = fmaf(y.hi, y.hi, -py);
  dfl s = df_2sum(px, py);
  s.lo += (ex + ey) + 2.0f * fmaf(x.hi, x.lo, y.hi * y.lo);
  return df_fast2sum(s.hi, s.lo);
}
// the separation (xa + xal) - (xb + xbl) - q (c.hi + c.lo), q in {-1, 0, 1}, as a
// double-float: the two exact sums of the high parts, the low parts added once (the cell
// shift q c.hi is exact); negating every input negates the result exactly
__device__ __forceinline__ dfl df_sep(float xa, float xal, float xb, float xbl, int q, dfl c) {
  const float ch = q < 0 ? -c.hi : (q > 0 ? c.hi : 0.0f);
  const float cl = q < 0 ? -c.lo : (q > 0 ? c.lo : 0.0f);
  const dfl a = df_2sum(xa, -xb);
  const dfl b = df_2sum(a.hi, -ch);
  return df_fast2sum(b.hi, ((a.lo + b.lo) + (xal - xbl)) - cl);
}
__device__ __forceinline__ dfl df_from(double v) {
  float h = (float)v;
  return {h, (float)(v - (double)h)};
}

// ordered key of a double: unsigned order of the keys = numeric order of the values, so
// that atomicMin on keys is an exact min over doubles
__device__ __forceinline__ unsigned long long okey(double x) {
  unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double unkey(unsigned long long k) {
  unsigned long long b = (k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)b);
}
constexpr unsigned long long kNoKey = ~0ull;  // no active particle

__device__ __forceinline__ unsigned long long warp_min(unsigned long long v) {
  const unsigned hi = __reduce_min_sync(0xffffffffu, (unsigned)(v >> 32));
  const unsigned lo =
      __reduce_min_sync(0xffffffffu, (unsigned)(v >> 32) == hi ? (unsigned)v : 0xffffffffu);
  return ((unsigned long long)hi << 32) | lo;
}

// true for every thread of the block that is the last of its grid to get here, once all
// blocks' earlier global writes are visible to it (read them past L1: __ldcg); the ticket is
// back at zero for the next launch
__device__ __forceinline__ bool last_block(unsigned* ticket) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (last) {
      *ticket = 0u;
      __threadfence();
    }
  }
  __syncthreads();
  return last;
}

// Check_Out_Domain (2_SPH_main_2018.f90:1170) + the bounding box of the active particles of
// every realisation: keys of (minx, miny, -maxx, -maxy, -maxh, minh).  A warp keeps the keys of
// its stretch of consecutive particles in registers while they belong to one realisation,
// and a block that holds one realisation combines its warps' before its atomicMin: one block's
// worth of atomics for each 256 particles, to six addresses, took longer than the 29 bytes a
// particle (2 million: 90 -> 37 us).
// The step's first kernel: it also loads the step's scalars, clears the cell counts, and its
// last block forms the grids (one launch instead of five: each of the small ones took about
// 5 us of a step that lasts 300 at 10,000 particles).
__device__ void grid_block(const Dev& D);
__global__ void __launch_bounds__(kBlock) k_bbox(Dev D, int per) {
  __shared__ unsigned long long sh[kBlock / 32][6];
  __shared__ int shr[kBlock / 32];
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (blockIdx.x == 0) {
    const int k = *D.step_idx;
    if (D.surr && threadIdx.x < 4) D.cand_count[threadIdx.x] = 0;  // the network's rows
    for (int r = threadIdx.x; r < D.R; r += blockDim.x)
      D.cur[r] = D.scal_table[(size_t)k * D.R + r];
    __syncthreads();
    if (threadIdx.x == 0) *D.step_idx = k + 1;
  }
  for (int c = gid; c < D.cell_cap + 2; c += gridDim.x * blockDim.x) {
    D.cntK[c] = 0ull;
    D.cntD[c] = 0;
  }
  unsigned long long m[6] = {kNoKey, kNoKey, kNoKey, kNoKey, kNoKey, kNoKey};
  int run = -1;  // the realisation that m is of
  auto reduce = [&] {
    for (int k = 0; k < 6; k++) m[k] = warp_min(m[k]);
  };
  // (x - xmin)(x - xmax) > 0 of the reference: both differences non-zero and of one sign, i.e.
  // x outside [xmin, xmax] (the product of two such differences cannot underflow to zero for a
  // domain of non-zero width; a NaN coordinate gives false), decided on the integer pipe
  // with ordered keys
  long long dom[4] = {0, 0, 0, 0};  // the realisation's domain: lowest and highest key by axis
  auto domain = [&](int r) {
    const Real& M = D.real[r];
    for (int d = 0; d < 2; d++) {
      const long long a = f64_key(M.xmin_dom[d]), b = f64_key(M.xmax_dom[d]);
      dom[2 * d] = min(a, b);
      dom[2 * d + 1] = max(a, b);
    }
  };
  auto outside = [](double v, long long lo, long long hi) {
    const long long k = f64_key(v);
    return !f64_isnan(v) && (k < lo || k > hi);
  };
  constexpr int U = 4;  // particles a lane whose loads are in flight together
  const int i0 = (gid >> 5) * 32 * per + lane;
  for (int q0 = 0; q0 < per; q0 += U) {
    double X[U], Y[U], H[U];
    int R[U];
    uint8_t O[U];
#pragma unroll
    for (int q = 0; q < U; q++) {
      const int i = i0 + 32 * (q0 + q);
      const bool in = q0 + q < per && i < D.N2;
      R[q] = in ? D.rid[i] : -1;
      X[q] = in ? D.px[i] : 0.0;
      Y[q] = in ? D.py[i] : 0.0;
      H[q] = in ? D.hsml[i] : 0.0;
      O[q] = in ? D.out[i] : 1;
    }
#pragma unroll
    for (int q = 0; q < U; q++) {
      const int r = R[q];
      const int r0 = __reduce_max_sync(0xffffffffu, r);
      if (r0 < 0) continue;  // past the end
      // the 32 particles are of one realisation, or of several
      const bool one = __all_sync(0xffffffffu, r < 0 || r == r0);
      if (one && r0 != run) {
        if (run >= 0) {
          reduce();
          if (lane == 0 && m[0] != kNoKey)
            for (int k = 0; k < 6; k++) atomicMin(&D.bbox[6 * (size_t)run + k], m[k]);
        }
        for (int k = 0; k < 6; k++) m[k] = kNoKey;
        run = r0;
        domain(r0);
      }
      bool o = O[q];
      if (r >= 0 && !o) {
        if (!one) domain(r);
        if (outside(X[q], dom[0], dom[1]) || outside(Y[q], dom[2], dom[3])) {
          o = true;
          D.out[i0 + 32 * (q0 + q)] = 1;
        }
      }
      if (r >= 0 && !o) {
        // the key of -x is the complement of x's
        const unsigned long long kx = okey(X[q]), ky = okey(Y[q]), kh = okey(H[q]);
        const unsigned long long v[6] = {kx, ky, ~kx, ~ky, ~kh, kh};
        if (one) {
          for (int k = 0; k < 6; k++) m[k] = v[k] < m[k] ? v[k] : m[k];
        } else if (kx != kNoKey) {
          for (int k = 0; k < 6; k++) atomicMin(&D.bbox[6 * (size_t)r + k], v[k]);
        }
      }
      if (!one && run >= 0) domain(run);
    }
  }
  reduce();
  if (lane == 0) {
    shr[wid] = run;
    for (int k = 0; k < 6; k++) sh[wid][k] = m[k];
  }
  __syncthreads();
  int rb = -1;
  bool one = true;  // the block's warps hold one realisation
  for (int w = 0; w < kBlock / 32; w++) rb = max(rb, shr[w]);
  for (int w = 0; w < kBlock / 32; w++) one = one && (shr[w] < 0 || shr[w] == rb);
  const int t = threadIdx.x;
  if (one) {
    if (rb >= 0 && t < 6) {
      unsigned long long u = sh[0][t];
      for (int w = 1; w < kBlock / 32; w++) u = sh[w][t] < u ? sh[w][t] : u;
      if (u != kNoKey) atomicMin(&D.bbox[6 * (size_t)rb + t], u);
    }
  } else if (t < 6 * (kBlock / 32)) {
    const int w = t / 6, k = t % 6;
    if (shr[w] >= 0 && sh[w][k] != kNoKey)
      atomicMin(&D.bbox[6 * (size_t)shr[w] + k], sh[w][k]);
  }
  if (last_block(D.tick)) grid_block(D);
}

// grid parameters of every realisation (2_SPH_main_2018.f90:1230-1260) and the numbering
// of their cells (one block of kBlock threads; the bounding-box keys are reset for the next
// step)
__device__ void grid_block(const Dev& D) {
  __shared__ int sc[kBlock];
  __shared__ int carry, bad;
  const int tid = threadIdx.x;
  if (tid == 0) {
    carry = 0;
    bad = 0;
  }
  __syncthreads();
  for (int base = 0; base < D.R; base += kBlock) {
    const int r = base + tid;
    int nc = 0;
    Grid g;
    if (r < D.R) {
      double red[6];
      for (int k = 0; k < 6; k++) {
        unsigned long long key = __ldcg(&D.bbox[6 * (size_t)r + k]);
        D.bbox[6 * (size_t)r + k] = kNoKey;
        red[k] = key == kNoKey ? 1e300 : unkey(key);
      }
      double hmax = -red[4];
      if (red[0] > 1e299) hmax = 0.0;  // no active particle
      double cellsz = hmax * 2.0;
      double ncd = 1.0;
      for (int d = 0; d < 2; d++) {
        double xmin = red[d] > 1e299 ? (double)1.e10f : red[d];
        double xmax = red[d] > 1e299 ? -(double)1.e10f : -red[2 + d];
        double length = xmax - xmin;
        double qd = length / cellsz + 1.0;
        int ndiv = (qd >= 1.0 && qd < 1.0e9) ? (int)qd : 1;
        double length_new = (double)ndiv * cellsz;
        g.xmin[d] = (xmin - (length_new - length) / 2.0) - (double)0.001f * length;
        g.deltx[d] = cellsz;
        g.rdeltx[d] = 1.0 / cellsz;
        g.ndiv[d] = ndiv;
        ncd *= ndiv;
      }
      g.overflow = (ncd > (double)D.cell_cap || !(cellsz > 0.0)) ? 1 : 0;
      nc = g.overflow ? 0 : (int)ncd;
      if (g.overflow) bad = 1;
      // uniform smoothing length: (h + h) / 2 == h, so every pair's kernel shares these
      g.uniform_h = (D.skf == 1 && red[5] == hmax && hmax > 0.0) ? 1 : 0;
      double h = hmax;
      g.h = h;
      g.yh = 1.0 / h;
      g.hh = h * h;
      g.yhh = 1.0 / g.hh;
      g.factor = 15.0 / (7.0 * D.pi * h * h);
      g.factor6 = g.factor / 6.0;
      g.c3 = g.factor6 * 3.0;
      g.df_h = df_from(g.h);
      g.df_yh = df_from(g.yh);
      g.df_yhh = df_from(g.yhh);
      g.df_factor = df_from(g.factor);
      g.df_factor6 = df_from(g.factor6);
      g.df_c3 = df_from(g.c3);
      g.df_cell[0] = df_from(g.deltx[0]);
      g.df_cell[1] = df_from(g.deltx[1]);
      // FP32 prefilter band: cell-relative offsets and the cell-corner shift each carry
      // |err| <= 2^-24 * 2 cells; the band covers eight times that relative to the support
      double ext = 2.0 * fmax(g.deltx[0], g.deltx[1]);
      double smin = (double)D.scale_k * red[5];
      g.tau = (float)((smin > 0) ? 8.0 * ext * 1.1920929e-07 / smin + 4e-6 : 1.0);
    }
    sc[tid] = nc;
    __syncthreads();
    for (int off = 1; off < kBlock && off < D.R; off <<= 1) {
      int add = tid >= off ? sc[tid - off] : 0;
      __syncthreads();
      sc[tid] += add;
      __syncthreads();
    }
    if (r < D.R) {
      g.ncells = nc;
      g.cell0 = carry + sc[tid] - nc;
      D.grid[r] = g;
    }
    __syncthreads();
    if (tid == min(kBlock, D.R - base) - 1) carry += sc[tid];
    __syncthreads();
  }
  if (tid == 0) {
    GridTotal gt;
    gt.overflow = (bad || carry > D.cell_cap) ? 1 : 0;
    gt.ncells = gt.overflow ? 0 : carry;
    gt.nactive = 0;
    *D.gtot = gt;
    if (gt.overflow) atomicOr(D.err, ERR_CELLS);
  }
}

// (x - xmin) / deltx of the reference's cell index (2_SPH_main_2018.f90:1280), correctly
// rounded by div_rcp from the cell size's reciprocal (an IEEE division costs GB300's FP64
// pipe about ten times as much); non-finite offsets take the IEEE division
__device__ __forceinline__ double cell_quot(double a, double b, double y) {
  const bool finite = (__double_as_longlong(a) & 0x7FF0000000000000ll) != 0x7FF0000000000000ll;
  return finite ? div_rcp(a, b, y) : a / b;
}

// (int)q for 1 <= q < 2^31, truncating, on the integer pipe (the significand shifted by
// the exponent)
__device__ __forceinline__ int trunc_pos(double q) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(q);
  const int e = (int)((b >> 52) & 0x7FF) - 1023;  // 0 .. 30
  const unsigned long long m = (b & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull;
  return (int)(m >> (52 - e));
}

// (double)n for 0 <= n < 2^31, exact, on the integer pipe
__device__ __forceinline__ double i2d_pos(int n) {
  if (n == 0) return 0.0;
  const int e = 31 - __clz(n);  // the leading bit
  const unsigned long long m = ((unsigned long long)(unsigned)n << (52 - e)) & 0x000FFFFFFFFFFFFFull;
  return __longlong_as_double((long long)(((unsigned long long)(e + 1023) << 52) | m));
}

// local cell of a position in a realisation's grid: q = (x - xmin) / delta + 1 with the
// reference's rounding, then its integer part clamped to [1, ndiv]; the comparisons and
// conversions on the integer pipe (ordered keys; q >= 1 is positive, below 2^31)
__device__ __forceinline__ int cell_index(const Grid& g, double x, double y) {
  const double qx = cell_quot(x - g.xmin[0], g.deltx[0], g.rdeltx[0]) + 1.0;
  const double qy = cell_quot(y - g.xmin[1], g.deltx[1], g.rdeltx[1]) + 1.0;
  // particles inside the bounding box give 1 <= q < ndiv + 1; the clamps only guard
  // against non-finite coordinates (a NaN q takes cell 1, as the FP64 comparisons did)
  auto idx = [](double q, int nd) {
    if (f64_isnan(q)) return 1;
    const long long k = f64_key(q);
    if (!(k >= f64_key(1.0))) return 1;
    return k < f64_key(i2d_pos(nd)) ? trunc_pos(q) : nd;
  };
  const int ix = idx(qx, g.ndiv[0]), iy = idx(qy, g.ndiv[1]);
  return g.ndiv[0] * (iy - 1) + (ix - 1);
}

// Task 2 of grid_find_NEW (2_SPH_main_2018.f90:1275-1286): the cell of every particle
// inside the domain, and the cells' counts by kind: cntK (nodes in the high word, stress-points
// in the low one) and cntD (dummies).  A particle's place in the count is its slot among its
// cell's particles of its kind (spos, until k_cell_rank), so the fill needs no second atomic.
__global__ void k_cell_count(Dev D) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= D.N2) return;
  const GridTotal gt = *D.gtot;
  int c;
  const Grid& g = D.grid[D.rid[i]];
  if (D.out[i] || gt.overflow) {
    c = gt.ncells;  // out-of-domain bucket, after every real cell
  } else {
    double x = D.px[i], y = D.py[i];
    int cl = cell_index(g, x, y);
    // FP32 offsets from the particle's own cell corner (|offset| <= one cell)
    int ix = cl % g.ndiv[0], iy = cl / g.ndiv[0];
    double ox = x - (g.xmin[0] + i2d_pos(ix) * g.deltx[0]);
    double oy = y - (g.xmin[1] + i2d_pos(iy) * g.deltx[1]);
    // the conversions on the integer pipe (f32_split: hi = (float)ox and lo = (float)(ox -
    // hi), the same bits as the hardware conversions, which GB300 issues at its FP64 rate)
    float oxh, oxl, oyh, oyl;
    f32_split(ox, oxh, oxl);
    f32_split(oy, oyh, oyl);
    D.xr[i] = oxh;
    D.yr[i] = oyh;
    if (D.fast) {
      D.xrl[i] = oxl;
      D.yrl[i] = oyl;
    }
    D.hr[i] = f32_rn(D.hsml[i]);
    c = g.cell0 + cl;
  }
  D.cell_of[i] = c;
  if (i < D.NN) D.spos[i] = (int)(atomicAdd(&D.cntK[c], 1ull << 32) >> 32);
  else if (i < D.NT) D.spos[i] = (int)(unsigned)atomicAdd(&D.cntK[c], 1ull);
  else D.spos[i] = atomicAdd(&D.cntD[c], 1);
}

// Exclusive scans of the cells' counts (total and by kind), kScan cells a block: the scan
// within the block (cell_loc, cell_locK) and, by the last block, of the blocks' sums (cell_bs,
// cell_bsK); readers add the two.  Blocks past the last cell only take their ticket.  A chain of
// latencies: four elements a thread, loaded together (16, one after the other, took 20 us at 10,000
// particles where this takes 9, events included).
constexpr int kPer = kScan / kBlock;
template <typename T>
__device__ __forceinline__ T block_exclusive(T v, T* sh, T& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T u = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += u;
  }
  __syncthreads();
  if (lane == 31) sh[w] = s;
  __syncthreads();
  T before = 0;
  total = 0;
#pragma unroll
  for (int k = 0; k < kBlock / 32; k++) {
    if (k < w) before += sh[k];
    total += sh[k];
  }
  return before + s - v;
}
// in place, by one block: exclusive scan of the nb sums
template <typename T>
__device__ __forceinline__ T scan_sums(T* bs, int nb, T* sh) {
  T carry = 0;
  for (int base = 0; base < nb; base += kBlock) {
    const int i = base + threadIdx.x;
    const T v = i < nb ? __ldcg(&bs[i]) : (T)0;
    T total;
    const T e = block_exclusive(v, sh, total);
    if (i < nb) bs[i] = carry + e;
    carry += total;
  }
  return carry;
}
__global__ void __launch_bounds__(kBlock) k_scan_cells(Dev D) {
  __shared__ int shT[kBlock / 32];
  __shared__ unsigned long long shK[kBlock / 32];
  const int n = D.gtot->ncells + 1;  // the out-of-domain bucket is the last
  const int base = blockIdx.x * kScan;
  if (base < n) {
    const int i0 = base + threadIdx.x * kPer;
    int t[kPer], lt = 0;
    unsigned long long k[kPer], lk = 0;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      k[q] = i0 + q < n ? D.cntK[i0 + q] : 0ull;
      t[q] = i0 + q < n ? D.cntD[i0 + q] : 0;
    }
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      t[q] += (int)(k[q] >> 32) + (int)(unsigned)k[q];
      lt += t[q];
      lk += k[q];
    }
    int totT;
    unsigned long long totK;
    int rt = block_exclusive(lt, shT, totT);
    unsigned long long rk = block_exclusive(lk, shK, totK);
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      const int c = i0 + q;
      if (c < n) {
        D.cell_cnt[c] = t[q];
        D.cell_loc[c] = rt;
        D.cell_locK[c] = rk;
      }
      rt += t[q];
      rk += k[q];
    }
    if (threadIdx.x == 0) {
      D.cell_bs[blockIdx.x] = totT;
      D.cell_bsK[blockIdx.x] = totK;
    }
  }
  if (last_block(D.tick + 1)) {
    const int nb = (n + kScan - 1) / kScan;
    scan_sums(D.cell_bs, nb, shT);
    scan_sums(D.cell_bsK, nb, shK);
  }
}
__device__ __forceinline__ int cell_first(const Dev& D, int c) {
  return D.cell_loc[c] + D.cell_bs[c / kScan];
}

// the cells' particle lists (list_picell, 2_SPH_main_2018.f90:1288-1305): nodes, stress-points
// and dummies of a cell one after the other (ids ascend from kind to kind), each kind in any
// order (tflag, put in ascending id order by k_cell_rank); and the cells' starts
__global__ void k_cell_fill(Dev D) {
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
  const int nc = D.gtot->ncells;
  for (int c = i0; c <= nc; c += gridDim.x * blockDim.x) {
    const int st = cell_first(D, c);
    D.cell_start[c] = st;
    if (c == nc) D.gtot->nactive = st;
  }
  if (i0 >= D.N2) return;
  const int c = D.cell_of[i0];
  const unsigned long long k = D.cntK[c];
  const int nn = (int)(k >> 32), ns = (int)(unsigned)k;
  const int off = i0 < D.NN ? 0 : i0 < D.NT ? nn : nn + ns;
  D.tflag[cell_first(D, c) + off + D.spos[i0]] = i0;
}

// per sorted position: the particle's rank by id among its cell's particles of its kind
// (list_picell order, 2_SPH_main_2018.f90:1299-1305), hence its sorted position; its list
// column (stress-points, then nodes, then dummies, each in sorted order); and the pair
// search's per-particle values in sorted order (the candidates of a cell are then read
// contiguously).  A cell holds a handful of each kind, so a particle counts the smaller ids
// itself: 6 us at 10,000 particles where one thread a cell sorting by insertion, the sorted
// copy and the eight launches that compacted the kinds took 72.  The order of the
// out-of-domain particles, which have no pairs, is left as it is.
__global__ void k_cell_rank(Dev D) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= D.N2) return;
  const int t = D.tflag[p];
  const int c = D.cell_of[t];
  const unsigned long long k = D.cntK[c];
  const int nn = (int)(k >> 32), ns = (int)(unsigned)k;
  const int first = D.cell_start[c];
  const bool node = t < D.NN, sp = !node && t < D.NT;
  const int seg = first + (node ? 0 : sp ? nn : nn + ns);
  const int len = node ? nn : sp ? ns : D.cntD[c];
  int rank = 0;
  if (c == D.gtot->ncells) rank = p - seg;
  else
    for (int j = 0; j < len; j++) rank += D.tflag[seg + j] < t;
  const int s = seg + rank;
  D.sorted[s] = t;
  D.spos[t] = s;
  const unsigned long long before = D.cell_locK[c] + D.cell_bsK[c / kScan];
  const int bn = (int)(before >> 32), bsp = (int)(unsigned)before;
  int col;
  if (sp) {
    col = bsp + rank;
    D.tgtS[col] = s;
    D.colid[col] = t;
  } else if (node) {
    D.tgtN[bn + rank] = s;
    col = (D.NT - D.NN) + bn + rank;
    D.colid[col] = t;
  } else {
    col = D.NT + (first - bn - bsp) + rank;
  }
  D.lcol[s] = col;
  D.srec[s] = make_float4(D.xr[t], D.yr[t], D.hr[t], __int_as_float(D.itype[t]));
  if (D.fast) D.srecl[s] = make_float2(D.xrl[t], D.yrl[t]);
}

// exact distance test of the reference (2_SPH_main_2018.f90:1345-1353) on the pair
// (a = creator, b); returns true and r, dx, dy, mhsml when the pair is accepted
__device__ __forceinline__ bool exact_test(const Dev& D, int a, int b, double& r, double& dx,
                                           double& dy, double& mh) {
  dx = D.px[a] - D.px[b];
  double driac = dx * dx;
  dy = D.py[a] - D.py[b];
  driac = driac + dy * dy;
  mh = (D.hsml[a] + D.hsml[b]) * 0.5;  // / 2.0, exactly
  r = sqrt(driac);
  // r < scale_k mh with the conversion and the comparison on the integer pipe (r >= 0)
  return !f64_isnan(r) && f64_key(r) < f64_key(i2d_pos(D.scale_k) * mh);
}

// 0 = reject, 1 = accept, 2 = undecided (inside the guard band).  (cx, cy) is the corner
// of b's cell relative to a's in FP32 (multiples of the cell size); fx, fy return the
// FP32 separation x_a - x_b.
__device__ __forceinline__ int prefilter(const Dev& D, float xa, float ya, float ha, float4 rb,
                                         float cx, float cy, float tau, float& fx, float& fy) {
  fx = (xa - rb.x) - cx;
  fy = (ya - rb.y) - cy;
  float d2 = fx * fx + fy * fy;
  float s = (float)D.scale_k * ((ha + rb.z) * 0.5f);
  float s2 = s * s;
  if (d2 < s2 * (1.0f - tau)) return 1;
  if (d2 > s2 * (1.0f + tau)) return 0;
  return 2;
}

// FP32 cubic / Gaussian / quintic kernel of the FP32 form (same formulas as the reference's
// kernel routine, evaluated in single precision)
__device__ __forceinline__ void sph_kernel_f32(int skf, float pi, float r, float dx0, float dx1,
                                               float h, float* w, float* dw0, float* dw1) {
  float q = r / h;
  *w = 0.0f;
  *dw0 = 0.0f;
  *dw1 = 0.0f;
  if (skf == 1) {
    float factor = 15.0f / (7.0f * pi * h * h);
    if (q <= 1.0f) {
      *w = factor * ((2.0f / 3.0f - q * q) + (q * q * q) * 0.5f);
      float a = (factor * (-2.0f + 1.5f * q)) / (h * h);
      *dw0 = a * dx0;
      *dw1 = a * dx1;
    } else if (q <= 2.0f) {
      float t = 2.0f - q;
      *w = (factor / 6.0f) * (t * t * t);
      float a = -(factor * 0.5f) * (t * t) / (h * r);
      *dw0 = a * dx0;
      *dw1 = a * dx1;
    }
  } else if (skf == 2) {
    float factor = 1.0f / (h * h * pi);
    if (q <= 3.0f) {
      *w = factor * expf(-(q * q));
      *dw0 = *w * (-2.0f * dx0 / (h * h));
      *dw1 = *w * (-2.0f * dx1 / (h * h));
    }
  } else {
    float factor = 7.0f / (478.0f * pi * h * h);
    float a = 3.0f - q, b = 2.0f - q, c1 = 1.0f - q;
    float a2 = a * a, b2 = b * b, c2 = c1 * c1;
    float a4 = a2 * a2, b4 = b2 * b2;
    float a5 = a4 * a, b5 = b4 * b, c5 = c2 * c2 * c1;
    if (q <= 1.0f) {
      *w = factor * ((a5 - 6.0f * b5) + 15.0f * c5);
      float g = factor * ((-120.0f + 120.0f * q) - 50.0f * (q * q)) / (h * h);
      *dw0 = g * dx0;
      *dw1 = g * dx1;
    } else if (q <= 2.0f) {
      *w = factor * (a5 - 6.0f * b5);
      float g = factor * (-5.0f * a4 + 30.0f * b4) / (h * r);
      *dw0 = g * dx0;
      *dw1 = g * dx1;
    } else if (q <= 3.0f) {
      *w = factor * a5;
      float g = factor * (-5.0f * a4) / (h * r);
      *dw0 = g * dx0;
      *dw1 = g * dx1;
    }
  }
}

// the reference's cubic kernel for a uniform h (2_SPH_main_2018.f90:1468-1492) for the FP32
// form: the separation, r and q = r/h in double-float, which removes the cancellations (of
// the cell-relative offsets and of 2 - q near the edge of the support), then the
// polynomial and the gradient in FP32 from the accurate q: W and dW within a few FP32 ulps
// of the FP64 evaluation
__device__ __forceinline__ void cubic_mixed(const Grid& g, dfl dx, dfl dy, float* w, float* dw0,
                                            float* dw1) {
  const dfl r = df_sqrt(df_sumsq(dx, dy));
  const dfl q = df_mul(r, g.df_yh);
  *w = 0.0f;
  *dw0 = 0.0f;
  *dw1 = 0.0f;
  if (q.hi < 1.0f || (q.hi == 1.0f && q.lo <= 0.0f)) {
    const float qh = q.hi, q2 = qh * qh;
    *w = g.df_factor.hi * ((2.0f / 3.0f - q2) + 0.5f * (q2 * qh));
    const float a = (g.df_factor.hi * (-2.0f + 1.5f * qh)) * g.df_yhh.hi;
    *dw0 = a * dx.hi;
    *dw1 = a * dy.hi;
  } else if (q.hi < 2.0f || (q.hi == 2.0f && q.lo <= 0.0f)) {
    const float t = (2.0f - q.hi) - q.lo;  // 2 - q.hi is exact
    const float t2 = t * t;
    *w = g.df_factor6.hi * (t2 * t);
    const float ar = ((g.df_c3.hi * t2) * g.df_yh.hi) / r.hi;
    *dw0 = -(ar * dx.hi);
    *dw1 = -(ar * dy.hi);
  }
}

// RN32(v.hi + v.lo) is certainly the float nearest to every value within |v| rel of it: true
// when the rest of v and that error stay inside half an ulp of v.hi (a power of two, whose
// lower neighbour is closer, and values off the ordinary exponents are left undecided)
__device__ __forceinline__ bool rounds_to_hi(dfl v, float rel) {
  const unsigned b = __float_as_uint(v.hi), e = (b >> 23) & 0xFFu;
  if (e < 40u || e > 250u || (b & 0x7FFFFFu) == 0u) return false;
  return fabsf(v.lo) + fabsf(v.hi) * rel < __uint_as_float((e - 24u) << 23);
}

// The reference's cubic kernel for a uniform h as the plain form stores it -- the FP64 values of
// cubic_uniform rounded to FP32 -- from double-float arithmetic, without the FP64 pipe (the
// separation dx, dy apart): the values are formed to a relative E and kept when no float
// boundary lies within E of them, so that the FP64 evaluation, which lies within E of them too,
// rounds to the same floats.  Returns false when undecided (about one pair in ten thousand): the
// caller evaluates in FP64.
// Bounds: dx, dy split into hi + lo, the squared sum and its root to 2^-47, q = r / h to 2^-45.
// For q > 1, t = 2 - q carries 2^-44 / t, so t^2 and t^3 3 2^-44 / t; for q <= 1 the
// polynomials lose at most a factor 8 to cancellation.  The FP64 evaluation's own error is below
// 2^-49 (1 + 1 / t).  E = 2^-41 (1 + 1 / t), 2^-41 for q <= 1; the largest errors met in 2.4e7
// random pairs (h 3e-4 .. 3, all directions) were 2^-43.1 (1 + 1 / t) and 2^-44.  q within
// 2^-36 of 1 and t below 2^-9 stay undecided, and so does a separation component below 2^-74
// that is not zero (below about 2^-106 its low part is subnormal and no longer exact to 2^-47).
__device__ __forceinline__ bool cubic_certified(const Grid& g, double dxd, double dyd, float* w,
                                                float* dw0, float* dw1) {
  dfl dx, dy;
  const bool okx = f32_split_int(dxd, dx.hi, dx.lo), oky = f32_split_int(dyd, dy.hi, dy.lo);
  if (!(okx && oky)) return false;
  const dfl r2 = df_sumsq(dx, dy);
  if (!(r2.hi > 1e-25f && r2.hi < 1e25f)) return false;
  const dfl r = df_sqrt_rn(r2);
  const dfl q = df_mul(r, g.df_yh);
  const float q1 = (q.hi - 1.0f) + q.lo;
  dfl W, a;
  float E;
  if (q1 < -1.4551915e-11f) {  // -2^-36
    const dfl q2 = df_mul(q, q), q3 = df_mul(q2, q);
    dfl b = df_2sum(2.0f / 3.0f, -q2.hi);
    b = df_fast2sum(b.hi, b.lo - q2.lo);
    dfl c = df_2sum(b.hi, 0.5f * q3.hi);
    c = df_fast2sum(c.hi, (c.lo + b.lo) + 0.5f * q3.lo);
    W = df_mul(g.df_factor, c);
    const float p = 1.5f * q.hi, pe = fmaf(1.5f, q.hi, -p);
    dfl m = df_2sum(-2.0f, p);
    m = df_fast2sum(m.hi, m.lo + fmaf(1.5f, q.lo, pe));
    a = df_mul(df_mul(g.df_factor, m), g.df_yhh);
    E = 4.5474735e-13f;  // 2^-41
  } else if (q1 > 1.4551915e-11f) {
    const dfl t = df_fast2sum(2.0f - q.hi, -q.lo);  // 2 - q.hi is exact
    if (!(t.hi >= 0.001953125f)) return false;
    const dfl t2 = df_mul(t, t);
    W = df_mul(g.df_factor6, df_mul(t2, t));
    // 1 / r: a Newton step in double-float from the FP32 reciprocal
    const float y0 = __frcp_rn(r.hi);
    const float e = fmaf(-r.hi, y0, 1.0f) - r.lo * y0;
    const dfl y = df_fast2sum(y0, y0 * e);
    a = df_mul(df_mul(df_mul(g.df_c3, t2), g.df_yh), y);
    a.hi = -a.hi;
    a.lo = -a.lo;
    E = 4.5474735e-13f * (1.0f + __frcp_rn(t.hi));
  } else {
    return false;
  }
  const dfl g0 = df_mul(a, dx), g1 = df_mul(a, dy);
  *w = W.hi;
  // a zero separation component: a is negative, so the product is a zero of the other sign
  *dw0 = dx.hi == 0.0f ? -dx.hi : g0.hi;
  *dw1 = dy.hi == 0.0f ? -dy.hi : g1.hi;
  return rounds_to_hi(W, E) && (dx.hi == 0.0f || rounds_to_hi(g0, E)) &&
         (dy.hi == 0.0f || rounds_to_hi(g1, E));
}

// the FP64 evaluation of a pair's stored kernel values (out of line: the rare case where h is
// uniform)
static __device__ __noinline__ float3 pair_values_f64(const Dev& D, const Grid& g, int a, int b) {
  double r, dx, dy, mh, w, dw0, dw1;
  exact_test(D, a, b, r, dx, dy, mh);
  if (g.uniform_h) cubic_uniform(g, r, dx, dy, &w, &dw0, &dw1);
  else sph_kernel(D.skf, D.pi, r, dx, dy, mh, &w, &dw0, &dw1);
  return make_float3(f32_rn(w), f32_rn(dw0), f32_rn(dw1));
}

// Pairs created by the particle at sorted position s, in the reference's creation order:
// the rest of its own cell, the cell to its right, then the three cells of the row above.
// FAST = false: W and dW from the reference's FP64 kernel, stored in FP32 (the plain
// form); FAST = true: the FP32 form's evaluation (cubic_mixed, or FP32 for a varying h).
// The pair set is the same.
// Kernel values of one accepted pair (creator a at sorted position s, partner at sorted
// position bs in stencil cell q), packed as the finished half-list entry.
template <bool FAST>
__device__ __forceinline__ int4 half_entry(const Dev& D, const Grid& g, int a, int ta, float xa,
                                           float ya, float ha, float xal, float yal, int bs,
                                           int q) {
  const int b = D.sorted[bs];
  const float cw = (float)g.deltx[0], ch = (float)g.deltx[1];
  // the stencil cell's offset (cells[q]) without indexing a local array
  const int qx = (q == 1 || q == 4) ? 1 : (q == 2 ? -1 : 0), qy = q >= 2 ? 1 : 0;
  const float cx = (float)qx * cw, cy = (float)qy * ch;
  const float4 rb = D.srec[bs];
  const float fx = (xa - rb.x) - cx, fy = (ya - rb.y) - cy;
  float wf, d0f, d1f;
  if (!FAST) {
    if (!(g.uniform_h &&
          cubic_certified(g, D.px[a] - D.px[b], D.py[a] - D.py[b], &wf, &d0f, &d1f))) {
      const float3 v = pair_values_f64(D, g, a, b);
      wf = v.x;
      d0f = v.y;
      d1f = v.z;
    }
  } else if (g.uniform_h) {
    // separation as double-float from the cell-relative hi/lo offsets
    // x_a - x_b = (offset_a - offset_b) - (cell shift) with every term in double-float
    const float2 rl = D.srecl[bs];
    cubic_mixed(g, df_sep(xa, xal, rb.x, rl.x, qx, g.df_cell[0]),
                df_sep(ya, yal, rb.y, rl.y, qy, g.df_cell[1]), &wf, &d0f, &d1f);
  } else {
    float hm = (ha + rb.z) * 0.5f;
    float rf = sqrtf(fx * fx + fy * fy);
    sph_kernel_f32(D.skf, (float)D.pi, rf, fx, fy, hm, &wf, &d0f, &d1f);
  }
  const int pt = pint_type(ta, D.itype[b]);
  return make_int4((int)((unsigned)b | ((unsigned)pt << kHalfTypeShift)), __float_as_int(wf),
                   __float_as_int(d0f), __float_as_int(d1f));
}

// Phase 2 of the plain form, warp-cooperative.  The FP64 kernel values are the plain form's
// cost (FP64 pipe), and a warp whose lanes each evaluate their own creator's pairs runs as
// many iterations as its longest list with the other lanes idle (17.8 of 32 lanes active
// per instruction in the per-lane loop).  Here the warp's accepted pairs are numbered
// creator by creator (a warp scan of the counts) and evaluated 32 at a time, one per lane:
// lane l takes pair base + l, finds its creator among the warp's lanes by a binary search
// over the scanned counts, and writes the finished entry into that creator's list at the
// same place.  Every entry is computed by the same arithmetic as before.  All 32 lanes call
// this (inactive ones with kk = 0).
__device__ __forceinline__ void half_phase2_coop(const Dev& D, int s, int kk, int a, int ta,
                                                 float xa, float ya, float ha) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int incl = kk;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += v;
  }
  const int excl = incl - kk;
  const int total = __shfl_sync(full, incl, 31);
  __syncwarp();  // the phase-1 entries of every lane are visible to the others
  for (int base = 0; base < total; base += 32) {
    const int p = base + lane;
    // the last lane whose first pair is at or before p (it owns p: p < its excl + kk)
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const int e = __shfl_sync(full, excl, lo + step);
      if (e <= p) lo += step;
    }
    const int so = __shfl_sync(full, s, lo), ao = __shfl_sync(full, a, lo);
    const int tao = __shfl_sync(full, ta, lo), eo = __shfl_sync(full, excl, lo);
    const float xo = __shfl_sync(full, xa, lo), yo = __shfl_sync(full, ya, lo);
    const float ho = __shfl_sync(full, ha, lo);
    if (p < total) {
      int4* out = D.half + (size_t)so * D.capH;
      const int m = p - eo;
      const int4 e0 = out[m];
      const Grid& g = D.grid[D.rid[ao]];
      out[m] = half_entry<false>(D, g, ao, tao, xo, yo, ho, 0.0f, 0.0f, e0.x, e0.y);
    }
  }
  __syncwarp();
}

// Phase 1 for the creator at sorted position s: the accepted partners in creation order
// (sorted position, stencil cell) into its half list, its pair count and its list-build
// record.  Returns the number of entries held (at most capH) and the creator's id, type and
// FP32 cell-relative offsets.
template <bool FAST>
__device__ __forceinline__ int half_phase1(const Dev& D, int s, int& a, int& ta, float& xa,
                                           float& ya, float& ha) {
  a = D.sorted[s];
  const Grid& g = D.grid[D.rid[a]];
  const float tau = g.tau;
  int c = D.cell_of[a] - g.cell0;  // local cell in the realisation's grid
  int nx = g.ndiv[0], ny = g.ndiv[1];
  int ix = c % nx, iy = c / nx;
  xa = D.xr[a];
  ya = D.yr[a];
  ha = D.hr[a];
  ta = D.itype[a];
  const float cw = (float)g.deltx[0], ch = (float)g.deltx[1];
  int k = 0;
  int4* out = D.half + (size_t)s * D.capH;
  // stencil cells in creation order: (dix, diy) and the first sorted position to scan
  int cells[5][2] = {{0, 0}, {1, 0}, {-1, 1}, {0, 1}, {1, 1}};
  int gstart[5] = {0, 0, 0, 0, 0};  // where each stencil cell's pairs start in the list
  for (int q = 0; q < 5; q++) {
    gstart[q] = min(k, D.capH);
    int jx = ix + cells[q][0], jy = iy + cells[q][1];
    if (jx < 0 || jx >= nx || jy >= ny) continue;
    int cc = g.cell0 + jy * nx + jx;
    int lo = (q == 0) ? s + 1 : D.cell_start[cc];
    int hi = D.cell_start[cc] + D.cell_cnt[cc];
    float cx = (float)cells[q][0] * cw, cy = (float)cells[q][1] * ch;
    // the kernel values follow in phase 2, so that the lanes of a warp evaluate them
    // together instead of each time one lane accepts a candidate
    for (int bs = lo; bs < hi; bs++) {
      float fx, fy;
      int pf = prefilter(D, xa, ya, ha, D.srec[bs], cx, cy, tau, fx, fy);
      if (pf == 0) continue;
      if (pf == 2) {
        double r, dx, dy, mh;
        if (!exact_test(D, a, D.sorted[bs], r, dx, dy, mh)) continue;
      }
      if (k < D.capH) out[k] = make_int4(bs, q, 0, 0);
      k++;
    }
  }
  if (k > D.capH) {
    atomicOr(D.err, ERR_HALF_CAP);
    k = D.capH;
  }
  D.half_cnt[s] = k;
  // what the list build reads of a creator, in one 16-byte record: where its pairs with
  // stencil cells 1-4 start, its pair count and its id
  D.half_meta[s] = make_int4((int)((unsigned)gstart[1] | ((unsigned)gstart[2] << 16)),
                             (int)((unsigned)gstart[3] | ((unsigned)gstart[4] << 16)), k, a);
  return k;
}

// Task 3 of grid_find_NEW (2_SPH_main_2018.f90:1307-1403): the half-stencil search
// (:1322-1341), the exact test (:1345-1353), kernel (:1371, :1440-1538) and the pair types
// of Pint_Update (3_SPH_material_2018.f90:1574-1634).
// Phase 2 turns each accepted (partner, stencil cell) into the finished entry: the
// partner's id with the pair type in its top bits (kHalfIdMask), so that the list build
// needs neither the partner's id nor its type from memory, and W, dW/dx, dW/dy; within one
// stencil cell the entries ascend in id (a cell is sorted by id) as they do in sorted
// position.  The FP32 form's lanes each finish their own list; the plain form's warps
// share the work (half_phase2_coop), so all of a warp's lanes stay to the end.
template <bool FAST>
__global__ void k_half(Dev D) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = s < D.N2 && s < D.gtot->nactive;
  if (!active && s < D.N2) D.half_cnt[s] = 0;
  if (FAST) {
    if (!active) return;
    int a, ta;
    float xa, ya, ha;
    const int kk = half_phase1<true>(D, s, a, ta, xa, ya, ha);
    const Grid& g = D.grid[D.rid[a]];
    const float xal = D.xrl[a], yal = D.yrl[a];
    int4* out = D.half + (size_t)s * D.capH;
    for (int m = 0; m < kk; m++) {
      const int4 e0 = out[m];
      out[m] = half_entry<true>(D, g, a, ta, xa, ya, ha, xal, yal, e0.x, e0.y);
    }
  } else {
    int a = 0, ta = 0, kk = 0;
    float xa = 0.0f, ya = 0.0f, ha = 0.0f;
    if (active) kk = half_phase1<false>(D, s, a, ta, xa, ya, ha);
    half_phase2_coop(D, s, kk, a, ta, xa, ya, ha);
  }
}

// entries 2j and 2j+1 of a list column in one 32-byte store (ell(): one sector, 32-byte
// aligned), so that no sector of the lists is ever written in halves
__device__ __forceinline__ void store_pair(int4* dst, int4 a, int4 b) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(a.x),
               "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
               : "memory");
}

// -------------------------------------------------------------------------- direct lists
// Where no walk-order keys are wanted, each target's lists are built straight from its 3 x 3
// cell stencil, without the half lists and the search through them.  Scanning the stencil's cells in ascending
// sorted position visits a target's partners in the reference's creation order of their
// pairs: first the creators before it (the row below, the cell to its left, its own cell
// up to it), one pair each, then its own half list (the rest of its cell, the cell to its
// right, the row above).  The lists hold that order.  The FP32 form's sums use it in every
// step; the plain form's walk order reverses the newest pairs in steps where the pair count
// reaches a new maximum (put_walk_order, from the first new pair that k_scan_half finds).
// The pair test is the same symmetric test (prefilter and exact FP64 band test), and the
// kernel values are evaluated with the target in the creator's role: the separation is
// negated exactly (double-float additions and the cell shift are sign-symmetric), so W is
// the same bits as the creator's evaluation and the gradient its exact negation.  Every
// target also counts the partners after it, which is its half-list length (half_cnt), for
// the pair count bookkeeping; dummies and inactive positions are counted by gather_rest.

// the list entry of partner bs (cell offset qx, qy) of a target of type ta with FP32
// cell-relative offsets (xa, xal), (ya, yal) and smoothing length ha: {partner id, W (sign
// bit set for a dummy partner), dW/dx, dW/dy} with the gradient with respect to the target.
// f32: the kernel values in FP32 from the FP32 separation (same-kind entries that only the
// FP32 free-surface detection reads), otherwise r and r/h in double-float (cubic_mixed)
template <bool PLAIN>
__device__ __forceinline__ int4 gather_entry(const Dev& D, const Grid& g, int a, int ta, float xa,
                                             float ya, float ha, float xal, float yal, int bs,
                                             int qx, int qy, bool f32 = false) {
  const int b = D.sorted[bs];
  const float4 rb = D.srec[bs];
  float wf, d0f, d1f;
  if (PLAIN) {
    if (!(g.uniform_h &&
          cubic_certified(g, D.px[a] - D.px[b], D.py[a] - D.py[b], &wf, &d0f, &d1f))) {
      const float3 v = pair_values_f64(D, g, a, b);
      wf = v.x;
      d0f = v.y;
      d1f = v.z;
    }
  } else if (g.uniform_h && !f32) {
    const float2 rl = D.srecl[bs];
    cubic_mixed(g, df_sep(xa, xal, rb.x, rl.x, qx, g.df_cell[0]),
                df_sep(ya, yal, rb.y, rl.y, qy, g.df_cell[1]), &wf, &d0f, &d1f);
  } else {
    // the cell shift qx * (float)deltx without conversions on the FP64 pipe
    const float cw = f32_rn(g.deltx[0]), ch = f32_rn(g.deltx[1]);
    const float cx = qx < 0 ? -cw : (qx > 0 ? cw : 0.0f);
    const float cy = qy < 0 ? -ch : (qy > 0 ? ch : 0.0f);
    const float fx = (xa - rb.x) - cx, fy = (ya - rb.y) - cy;
    const float hm = (ha + rb.z) * 0.5f;
    const float rf = sqrtf(fx * fx + fy * fy);
    sph_kernel_f32(D.skf, f32_rn(D.pi), rf, fx, fy, hm, &wf, &d0f, &d1f);
  }
  const int pt = pint_type(ta, __float_as_int(rb.w));
  const int w = __float_as_int(wf);
  return make_int4(b, (pt == 6 || pt == 9) ? (int)((unsigned)w | 0x80000000u) : w,
                   __float_as_int(d0f), __float_as_int(d1f));
}

// the accepted-partner test of the pair search, from either side of the pair
__device__ __forceinline__ bool gather_accept(const Dev& D, int a, float xa, float ya, float ha,
                                              float4 rb, int bs, float cx, float cy, float tau) {
  float fx, fy;
  const int pf = prefilter(D, xa, ya, ha, rb, cx, cy, tau, fx, fy);
  if (pf == 0) return false;
  if (pf == 2) {
    double r, dx, dy, mh;
    return exact_test(D, a, D.sorted[bs], r, dx, dy, mh);
  }
  return true;
}

// Task 3 of grid_find_NEW (2_SPH_main_2018.f90:1307-1403), kernel (:1440-1538) and
// Pint_Update (3_SPH_material_2018.f90:1574-1634) per target of either form, gathering its entries
// from the 3 x 3 cell stencil directly in creation order.
// No same-kind lists (gather_by_group writes them): degS holds 0 unless the outside approach
// reads the counts.  Phase 1 tests the stencil's candidates and keeps the
// accepted ones (sorted position and cell offset) in shared memory; phase 2 evaluates the
// kernel values, so that a warp's lanes evaluate together.  Dynamic shared memory:
// capC ints per thread, entry k of thread j at k * blockDim + j.
template <bool PLAIN>
__device__ __forceinline__ void gather_target(const Dev& D, int s, int col, int* buf) {
  const int bd = blockDim.x, tid = threadIdx.x;
  int nC = 0, nS = 0, nHalf = 0;
  if (s < D.gtot->nactive) {
    const int a = D.sorted[s];
    const int ta = D.itype[a];
    const Grid& g = D.grid[D.rid[a]];
    const float tau = g.tau;
    const int c = D.cell_of[a] - g.cell0;
    const int nx = g.ndiv[0], ny = g.ndiv[1];
    const int ix = c % nx, iy = c / nx;
    const float xa = D.xr[a], ya = D.yr[a], ha = D.hr[a];
    const float cw = (float)g.deltx[0], ch = (float)g.deltx[1];
    // same-kind partners before the target matter only for the outside approach's
    // isolated-node test, which reads the full same-kind count; otherwise only the
    // ones after it are tested, for the half-list count
    const bool all_same = D.outside;
    // a uniform smoothing length makes the prefilter's bounds constant (the same FP32
    // expressions as prefilter(), so the same decisions)
    float s2lo = 0.0f, s2hi = 0.0f;
    if (g.uniform_h) {
      const float sv = (float)D.scale_k * ((ha + ha) * 0.5f);
      const float s2 = sv * sv;
      s2lo = s2 * (1.0f - tau);
      s2hi = s2 * (1.0f + tau);
    }
    // the stencil row by row: a row's three cells are one contiguous run of sorted
    // positions; a candidate's cell follows from the run's cell boundaries
    for (int qy = -1; qy <= 1; qy++) {
      const int jy = iy + qy;
      if (jy < 0 || jy >= ny) continue;
      const int row0 = g.cell0 + jy * nx;
      const int cr = row0 + (ix + 1 < nx ? ix + 1 : ix);
      const int lo = D.cell_start[row0 + (ix > 0 ? ix - 1 : 0)];
      const int hi = D.cell_start[cr] + D.cell_cnt[cr];
      const int b0 = D.cell_start[row0 + ix];                         // the centre cell
      const int b1 = ix + 1 < nx ? D.cell_start[row0 + ix + 1] : hi;  // the right cell
      const float cy = qy < 0 ? -ch : (qy > 0 ? ch : 0.0f);  // (float)qy * ch
      for (int bs = lo; bs < hi; bs++) {
        if (bs == s) continue;
        const float4 rb = D.srec[bs];
        const bool same = __float_as_int(rb.w) == ta;
        if (same && !all_same && bs < s) continue;
        const int qx = bs < b0 ? -1 : (bs < b1 ? 0 : 1);
        const float cx = qx < 0 ? -cw : (qx > 0 ? cw : 0.0f);  // (float)qx * cw
        bool acc;
        if (g.uniform_h) {
          const float fx = (xa - rb.x) - cx, fy = (ya - rb.y) - cy;
          const float d2 = fx * fx + fy * fy;
          if (d2 > s2hi) continue;
          acc = d2 < s2lo;
          if (!acc) {
            double r, dx, dy, mh;
            acc = exact_test(D, a, D.sorted[bs], r, dx, dy, mh);
          }
        } else {
          acc = gather_accept(D, a, xa, ya, ha, rb, bs, cx, cy, tau);
        }
        if (!acc) continue;
        nHalf += bs > s;
        const int code = (qy + 1) * 3 + (qx + 1);  // cell offset, kept in the top 4 bits
        if (same) {
          nS++;
        } else {
          if (nC < D.capC) buf[(size_t)nC * bd + tid] = bs | (code << kHalfTypeShift);
          nC++;
        }
      }
    }
    if (!all_same) nS = 0;  // not counted: no step kernel reads the same-kind lists or counts
    if (nHalf > D.capH) {
      atomicOr(D.err, ERR_HALF_CAP);
      nHalf = D.capH;
    }
    if (nC > D.capC || nS > D.capS) {
      atomicOr(D.err, ERR_LIST_CAP);
      nC = min(nC, D.capC);
      nS = min(nS, D.capS);
    }
    const float xal = PLAIN ? 0.0f : D.xrl[a], yal = PLAIN ? 0.0f : D.yrl[a];
    // phase 2: the entries, stored in pairs (whole 32-byte sectors)
    int4 pend = make_int4(0, 0, 0, 0);
    for (int k = 0; k < nC; k++) {
      const unsigned v = (unsigned)buf[(size_t)k * bd + tid];
      const int code = (int)(v >> kHalfTypeShift);
      const int4 e = gather_entry<PLAIN>(D, g, a, ta, xa, ya, ha, xal, yal, (int)(v & kHalfIdMask),
                                         code % 3 - 1, code / 3 - 1, false);
      if (k & 1) store_pair(D.cross + ell(k - 1, col, D.N2), pend, e);
      else pend = e;
      // the lanes of a warp write entry k of adjacent columns together: whole sectors
      if (D.use_crossW) D.crossW[(size_t)k * D.N2 + col] = make_int2(e.x, e.y);
    }
    if (nC & 1) D.cross[ell(nC - 1, col, D.N2)] = pend;
  }
  D.degC[col] = nC;
  D.degS[col] = nS;
  D.half_cnt[s] = nHalf;
}

// The same gather by G lanes a target: they test G candidates at a time, keep the accepted ones
// in order (their places from a ballot) and share the kernel values.  The same decisions and
// values; all 32 lanes of a warp take part (act: the group has a target).  Two reasons to
// take it: the serial chain of about 100 tests and up to 36 evaluations a target is G times
// shorter where the problem cannot fill the chip, and a group's buffers are shared, so that G times
// as many warps fit a multiprocessor where two lists are buffered (launch_gather).  SAME: the
// same-kind entries are written too, for the steps that read them (XSPH, artificial viscosity
// or stress, the FP32 free-surface detection; those that no step kernel reads hold FP32 kernel
// values, Dev::same_f32).
template <bool SAME, bool PLAIN, int G>
__device__ __forceinline__ void gather_by_group(const Dev& D, int s, int col, bool act, int* bufC) {
  constexpr unsigned all = 0xffffffffu;
  const int q = threadIdx.x & (G - 1), sh = threadIdx.x & 31 & ~(G - 1);
  const unsigned below = (1u << q) - 1u;
  int* bufS = bufC + D.capC;
  auto group = [&](bool b) { return (__ballot_sync(all, b) >> sh) & ((1u << G) - 1u); };
  const bool on = act && s < D.gtot->nactive;
  const int a = D.sorted[s];
  const int ta = D.itype[a];
  const Grid& g = D.grid[D.rid[a]];
  const float tau = g.tau;
  const int nx = g.ndiv[0], ny = g.ndiv[1];
  const int c = on ? D.cell_of[a] - g.cell0 : 0;
  const int ix = c % nx, iy = c / nx;
  const float xa = D.xr[a], ya = D.yr[a], ha = D.hr[a];
  const float cw = (float)g.deltx[0], ch = (float)g.deltx[1];
  const bool all_same = SAME || D.outside;
  float s2lo = 0.0f, s2hi = 0.0f;
  if (g.uniform_h) {
    const float sv = (float)D.scale_k * ((ha + ha) * 0.5f);
    const float s2 = sv * sv;
    s2lo = s2 * (1.0f - tau);
    s2hi = s2 * (1.0f + tau);
  }
  int nC = 0, nS = 0, nHalf = 0;
  for (int qy = -1; qy <= 1; qy++) {
    const int jy = iy + qy;
    int lo = 0, hi = 0, b0 = 0, b1 = 0;
    if (on && jy >= 0 && jy < ny) {
      const int row0 = g.cell0 + jy * nx;
      const int cr = row0 + (ix + 1 < nx ? ix + 1 : ix);
      lo = D.cell_start[row0 + (ix > 0 ? ix - 1 : 0)];
      hi = D.cell_start[cr] + D.cell_cnt[cr];
      b0 = D.cell_start[row0 + ix];
      b1 = ix + 1 < nx ? D.cell_start[row0 + ix + 1] : hi;
    }
    const float cy = qy < 0 ? -ch : (qy > 0 ? ch : 0.0f);
    const int nmax = (int)__reduce_max_sync(all, (unsigned)(hi - lo));
    for (int j = 0; j < nmax; j += G) {
      const int bs = lo + j + q;
      bool acc = false, same = false;
      int qx = 0;
      if (bs < hi && bs != s) {
        const float4 rb = D.srec[bs];
        same = __float_as_int(rb.w) == ta;
        if (!same || all_same || bs > s) {
          qx = bs < b0 ? -1 : (bs < b1 ? 0 : 1);
          const float cx = qx < 0 ? -cw : (qx > 0 ? cw : 0.0f);
          if (g.uniform_h) {
            const float fx = (xa - rb.x) - cx, fy = (ya - rb.y) - cy;
            const float d2 = fx * fx + fy * fy;
            acc = d2 < s2lo;
            if (!acc && !(d2 > s2hi)) {
              double r, dx, dy, mh;
              acc = exact_test(D, a, D.sorted[bs], r, dx, dy, mh);
            }
          } else {
            acc = gather_accept(D, a, xa, ya, ha, rb, bs, cx, cy, tau);
          }
        }
      }
      const unsigned mC = group(acc && !same), mS = group(acc && same);
      nHalf += __popc(group(acc && bs > s));
      const int code = bs | (((qy + 1) * 3 + (qx + 1)) << kHalfTypeShift);
      if (acc) {
        const int k = same ? nS + __popc(mS & below) : nC + __popc(mC & below);
        if (!same && k < D.capC) bufC[k] = code;
        if (SAME && same && k < D.capS) bufS[k] = code;
      }
      nC += __popc(mC);
      nS += __popc(mS);
    }
  }
  __syncwarp();
  if (!act) return;
  if (!all_same) nS = 0;
  if (nHalf > D.capH || nC > D.capC || nS > D.capS) {
    if (q == 0) {
      if (nHalf > D.capH) atomicOr(D.err, ERR_HALF_CAP);
      if (nC > D.capC || nS > D.capS) atomicOr(D.err, ERR_LIST_CAP);
    }
    nHalf = min(nHalf, D.capH);
    nC = min(nC, D.capC);
    nS = min(nS, D.capS);
  }
  const float xal = PLAIN ? 0.0f : D.xrl[a], yal = PLAIN ? 0.0f : D.yrl[a];
  auto finish = [&](const int* buf, int n, int4* list, int2* compact, bool f32) {
    for (int k = q; k < n; k += G) {
      const unsigned v = (unsigned)buf[k];
      const int code = (int)(v >> kHalfTypeShift);
      const int4 e = gather_entry<PLAIN>(D, g, a, ta, xa, ya, ha, xal, yal, (int)(v & kHalfIdMask),
                                         code % 3 - 1, code / 3 - 1, f32);
      list[ell(k, col, D.N2)] = e;
      if (compact) compact[(size_t)k * D.N2 + col] = make_int2(e.x, e.y);
    }
  };
  finish(bufC, nC, D.cross, D.use_crossW ? D.crossW : nullptr, false);
  if (SAME) finish(bufS, nS, D.same, nullptr, D.same_f32);
  if (q == 0) {
    D.degC[col] = nC;
    D.degS[col] = nS;
    D.half_cnt[s] = nHalf;
  }
}

// every sorted position that is not a stress-point or node target: the half-list length
// of an active dummy (its pairs with the particles after it in its half stencil), zero
// counts for inactive positions and dummies' list columns
__device__ __forceinline__ void gather_rest(const Dev& D, int a) {
  const int s = D.spos[a];
  const int col = D.lcol[s];
  D.degC[col] = 0;
  D.degS[col] = 0;
  int k = 0;
  if (s < D.gtot->nactive) {
    const Grid& g = D.grid[D.rid[a]];
    const int c = D.cell_of[a] - g.cell0;
    const int nx = g.ndiv[0], ny = g.ndiv[1];
    const int ix = c % nx, iy = c / nx;
    const float xa = D.xr[a], ya = D.yr[a], ha = D.hr[a];
    const float cw = (float)g.deltx[0], ch = (float)g.deltx[1];
    const int cells[5][2] = {{0, 0}, {1, 0}, {-1, 1}, {0, 1}, {1, 1}};
    for (int q = 0; q < 5; q++) {
      const int jx = ix + cells[q][0], jy = iy + cells[q][1];
      if (jx < 0 || jx >= nx || jy >= ny) continue;
      const int cc = g.cell0 + jy * nx + jx;
      const int lo = q == 0 ? s + 1 : D.cell_start[cc];
      const int hi = D.cell_start[cc] + D.cell_cnt[cc];
      const float cx = (float)cells[q][0] * cw, cy = (float)cells[q][1] * ch;
      for (int bs = lo; bs < hi; bs++)
        k += gather_accept(D, a, xa, ya, ha, D.srec[bs], bs, cx, cy, g.tau);
    }
    if (k > D.capH) {
      atomicOr(D.err, ERR_HALF_CAP);
      k = D.capH;
    }
  }
  D.half_cnt[s] = k;
}

// the stress-point targets [0, bs blocks), the node targets [bs, bn), the dummies: one launch
template <bool PLAIN>
__global__ void __launch_bounds__(512, 2) k_fgather(Dev D, int bs, int bn) {
  extern __shared__ int gbuf[];
  const int ns = D.NT - D.NN, b = blockIdx.x;
  if (b < bs) {
    const int k = b * blockDim.x + threadIdx.x;
    if (k < ns) gather_target<PLAIN>(D, D.tgtS[k], k, gbuf);
  } else if (b < bn) {
    const int k = (b - bs) * blockDim.x + threadIdx.x;
    if (k < D.NN) gather_target<PLAIN>(D, D.tgtN[k], ns + k, gbuf);
  } else {
    const int k = (b - bn) * blockDim.x + threadIdx.x;
    if (D.NT + k < D.N2) gather_rest(D, D.NT + k);
  }
}

template <bool SAME, bool PLAIN, int G>
__global__ void __launch_bounds__(128) k_fgatherg(Dev D, int bs, int bn) {
  extern __shared__ int gbuf[];
  const int ns = D.NT - D.NN, b = blockIdx.x, per = blockDim.x / G, w = threadIdx.x / G;
  int* buf = gbuf + (size_t)w * (D.capC + (SAME ? D.capS : 0));
  if (b < bs) {
    const int k = b * per + w, kk = k < ns ? k : 0;
    gather_by_group<SAME, PLAIN, G>(D, D.tgtS[kk], kk, k < ns, buf);
  } else if (b < bn) {
    const int k = (b - bs) * per + w, kk = k < D.NN ? k : 0;
    gather_by_group<SAME, PLAIN, G>(D, D.tgtN[kk], ns + kk, k < D.NN, buf);
  } else {
    const int k = (b - bn) * blockDim.x + threadIdx.x;
    if (D.NT + k < D.N2) gather_rest(D, D.NT + k);
  }
}

// The sorted position of the K-th partner (from 0) of the creator at sorted position s: its
// half stencil in ascending sorted position, which is its creation order
__device__ __forceinline__ int creator_partner(const Dev& D, int s, int64_t K) {
  const int a = D.sorted[s];
  const Grid& g = D.grid[D.rid[a]];
  const int c = D.cell_of[a] - g.cell0, nx = g.ndiv[0], ny = g.ndiv[1];
  const int ix = c % nx, iy = c / nx;
  const float xa = D.xr[a], ya = D.yr[a], ha = D.hr[a];
  const float cw = (float)g.deltx[0], ch = (float)g.deltx[1];
  for (int q = 0; q < 5; q++) {
    const int dx = (q == 1 || q == 4) ? 1 : (q == 2 ? -1 : 0), dy = q >= 2 ? 1 : 0;
    const int jx = ix + dx, jy = iy + dy;
    if (jx < 0 || jx >= nx || jy >= ny) continue;
    const int cc = g.cell0 + jy * nx + jx;
    const int lo = q == 0 ? s + 1 : D.cell_start[cc], hi = D.cell_start[cc] + D.cell_cnt[cc];
    for (int bs = lo; bs < hi; bs++)
      if (gather_accept(D, a, xa, ya, ha, D.srec[bs], bs, (float)dx * cw, (float)dy * ch, g.tau) &&
          K-- == 0)
        return bs;
  }
  return D.N2;
}

// Pair counts: half_off, the exclusive scan of the half-list lengths within kScan sorted
// positions, and half_bs, the scan of the blocks' sums (readers add the two: half_first), then
// the pair bookkeeping of every realisation (its pairs are the half lists of its sorted
// range), both by the last block
__device__ __forceinline__ int64_t half_first(const Dev& D, int s) {
  return D.half_off[s] + D.half_bs[s / kScan];
}
__global__ void __launch_bounds__(kBlock) k_scan_half(Dev D) {
  __shared__ long long sh[kBlock / 32];
  const int i0 = blockIdx.x * kScan + threadIdx.x * kPer;
  int h[kPer];
  long long l = 0;
#pragma unroll
  for (int q = 0; q < kPer; q++) h[q] = i0 + q < D.N2 ? D.half_cnt[i0 + q] : 0;
#pragma unroll
  for (int q = 0; q < kPer; q++) l += h[q];
  long long tot;
  long long run = block_exclusive(l, sh, tot);
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    if (i0 + q <= D.N2) D.half_off[i0 + q] = run;  // one past the end: the total
    run += h[q];
  }
  if (threadIdx.x == 0) D.half_bs[blockIdx.x] = tot;
  if (!last_block(D.tick + 2)) return;
  const long long all = scan_sums(reinterpret_cast<long long*>(D.half_bs), (int)gridDim.x, sh);
  __syncthreads();
  auto first = [&](int s) -> int64_t {
    return (int64_t)__ldcg((const long long*)&D.half_off[s]) +
           (int64_t)__ldcg((const long long*)&D.half_bs[s / kScan]);
  };
  const GridTotal gt = *D.gtot;
  for (int r = threadIdx.x; r < D.R; r += blockDim.x) {
    const Grid& g = D.grid[r];
    int64_t lo = 0, hi = 0;
    if (!gt.overflow) {
      lo = first(D.cell_start[g.cell0]);
      hi = first(D.cell_start[g.cell0 + g.ncells]);
    }
    PairMeta m = D.meta[r];
    m.m_prev = m.m;
    m.n = hi - lo;
    m.base = lo;
    if (m.n > m.m) m.m = m.n;
    if (D.walk_order && m.n > m.m_prev) {
      // the first new pair: its creator is the last sorted position whose pairs start at or
      // before it
      const int64_t B = m.base + m.m_prev;
      int a = D.cell_start[g.cell0], b = D.cell_start[g.cell0 + g.ncells];
      while (b - a > 1) {
        const int mid = a + (b - a) / 2;
        if (first(mid) <= B) a = mid;
        else b = mid;
      }
      m.newc = a;
      m.newo = creator_partner(D, a, B - first(a));
    }
    D.meta[r] = m;
  }
  // walk-order keys hold 2 x position in 32 bits
  if (threadIdx.x == 0 && all > 1073741823LL) atomicOr(D.err, ERR_NPAIRS);
}

template <bool KEYS>
__device__ __forceinline__ void reverse_ell(int4* base, int32_t* key, int N2, int col, int lo,
                                            int hi) {
  // reverse entries [lo, hi) of list column col (and their keys)
  hi--;
  while (lo < hi) {
    int4 t = base[ell(lo, col, N2)];
    base[ell(lo, col, N2)] = base[ell(hi, col, N2)];
    base[ell(hi, col, N2)] = t;
    if (KEYS) {
      int32_t k = key[(size_t)lo * N2 + col];
      key[(size_t)lo * N2 + col] = key[(size_t)hi * N2 + col];
      key[(size_t)hi * N2 + col] = k;
    }
    lo++;
    hi--;
  }
}

// Per-target lists.  The pairs a target t meets, in creation order, are: first the pairs
// created by particles before t in sorted order (each holds t in its half list), then
// t's own half list.  The linked list of the reference is walked as: pairs created this
// step beyond the previous list length m (newest first), then pairs 0..m-1 in creation
// order; the lists are written in that walk order.
// KEYS: also write the walk-order key of every entry (for the free-surface detection)
template <bool KEYS>
__device__ __forceinline__ void lists_target(const Dev& D, int s, int4& pendC, int4& pendS) {
  int nC = 0, nS = 0, newC = 0, newS = 0;
  const int col = D.lcol[s];
  if (s < D.gtot->nactive) {
    int t = D.sorted[s];
    int tt = D.itype[t];
    if (!is_dummy(tt)) {
      const int r = D.rid[t];
      const Grid& g = D.grid[r];
      const PairMeta meta = D.meta[r];
      const bool reorder = meta.n > meta.m_prev;
      const int c0g = g.cell0;
      int c = D.cell_of[t] - c0g;  // local cell
      int nx = g.ndiv[0];
      int ix = c % nx, iy = c / nx;
      int lo[2], hi[2];
      if (iy > 0) {
        int c0 = c0g + (iy - 1) * nx + (ix > 0 ? ix - 1 : 0);
        int c1 = c0g + (iy - 1) * nx + (ix + 1 < nx ? ix + 1 : ix);
        lo[0] = D.cell_start[c0];
        hi[0] = D.cell_start[c1] + D.cell_cnt[c1];
      } else {
        lo[0] = hi[0] = 0;
      }
      lo[1] = D.cell_start[c0g + (ix > 0 ? c - 1 : c)];
      hi[1] = s;
      // key of an entry: its position in the walk order of the realisation's list, and
      // whether the target is pair_i (creator of a same-type pair; the stress-point of a
      // node--stress-point pair)
      auto push = [&](int u, int pt, int w, float gx, float gy, int64_t cidx, bool own) {
        bool same = (pt == 2 || pt == 3);
        // a wall (dummy) partner (pair types 6 and 9 of a non-dummy target) is marked by the
        // sign bit of W (W >= 0): readers skip or branch on it without loading its type
        int4 e = make_int4(u, (pt == 6 || pt == 9) ? (int)((unsigned)w | 0x80000000u) : w,
                           __float_as_int(gx), __float_as_int(gy));
        const int64_t rel = cidx - meta.base;
        bool isnew = reorder && rel >= meta.m_prev;
        int64_t wp = !reorder ? rel : isnew ? meta.n - 1 - rel : (meta.n - meta.m_prev) + rel;
        int role = same ? (own ? 1 : 0) : (pt == 1 && is_sp(tt) ? 1 : 0);
        int32_t key = (int32_t)(2 * wp + role);
        // an even entry waits in pendS / pendC for its odd partner, and the two are stored
        // together; a last even entry is stored alone after the walk
        if (same) {
          if (nS < D.capS && (KEYS || D.same_entries)) {
            if (nS & 1) store_pair(D.same + ell(nS - 1, col, D.N2), pendS, e);
            else pendS = e;
            if (KEYS) D.keyS[(size_t)nS * D.N2 + col] = key;
          }
          nS++;
          newS += isnew;
        } else if (pt != 0) {
          if (nC < D.capC) {
            if (nC & 1) store_pair(D.cross + ell(nC - 1, col, D.N2), pendC, e);
            else pendC = e;
            if (KEYS) D.keyC[(size_t)nC * D.N2 + col] = key;
          }
          nC++;
          newC += isnew;
        }
      };
      // the creators before s, in ascending sorted position: each holds s at most once in
      // its (ascending) half list, among the pairs it made with s's cell, whose place in
      // the list k_half recorded (half_meta: the starts of its five stencil cells).  The
      // stencil cell of s seen from a creator follows from the creator's cell: below-left,
      // below, below-right (region 0), left, own (region 1).  kG lower-bound searches run
      // interleaved, so that their dependent loads overlap; the hits are pushed in creator
      // order.
      constexpr int kG = 4;
      const int n0 = hi[0] - lo[0], ncand = n0 + (hi[1] - lo[1]);
      const int rowb = c0g + (iy - 1) * nx;  // first cell of the row below
      const int b1 = iy > 0 ? D.cell_start[rowb + ix] : 0;  // the cell below s's cell
      const int b2 = (iy > 0 && ix + 1 < nx) ? D.cell_start[rowb + ix + 1] : hi[0];
      const int own0 = D.cell_start[c0g + c];
      for (int i0 = 0; i0 < ncand; i0 += kG) {
        int as[kG], pos[kG], len[kG], cnt[kG], cid[kG];
        int4 mt[kG];
#pragma unroll
        for (int q = 0; q < kG; q++) {
          const int i = i0 + q;
          as[q] = i < n0 ? lo[0] + i : lo[1] + (i - n0);
          mt[q] = i < ncand ? D.half_meta[as[q]] : make_int4(0, 0, 0, 0);
          cnt[q] = mt[q].z;
          cid[q] = mt[q].w;
        }
#pragma unroll
        for (int q = 0; q < kG; q++) {
          const int i = i0 + q;
          const unsigned g12 = (unsigned)mt[q].x, g34 = (unsigned)mt[q].y;
          const int gs[6] = {0, (int)(g12 & 0xFFFFu), (int)(g12 >> 16), (int)(g34 & 0xFFFFu),
                             (int)(g34 >> 16), cnt[q]};
          // stencil cell of s from the creator: 0 own, 1 right, 2 up-left, 3 up, 4 up-right
          const int st = i < n0 ? (as[q] < b1 ? 4 : as[q] < b2 ? 3 : 2) : (as[q] < own0 ? 1 : 0);
          const int g0 = st == 0 ? gs[0] : st == 1 ? gs[1] : st == 2 ? gs[2] : st == 3 ? gs[3] : gs[4];
          const int g1 = st == 0 ? gs[1] : st == 1 ? gs[2] : st == 2 ? gs[3] : st == 3 ? gs[4] : gs[5];
          pos[q] = g0;
          len[q] = i < ncand ? max(g1 - g0, 0) : 0;
        }
        bool more = true;
        while (more) {
          int v[kG];
#pragma unroll
          for (int q = 0; q < kG; q++)
            v[q] = len[q] > 0 ? (int)((unsigned)D.half[(size_t)as[q] * D.capH + pos[q] +
                                                       (len[q] >> 1)].x & kHalfIdMask)
                              : 0;
          more = false;
#pragma unroll
          for (int q = 0; q < kG; q++)
            if (len[q] > 0) {
              const int half = len[q] >> 1;
              if (v[q] < t) {
                pos[q] += half + 1;
                len[q] -= half + 1;
              } else {
                len[q] = half;
              }
              more |= len[q] > 0;
            }
        }
#pragma unroll
        for (int q = 0; q < kG; q++)
          if (pos[q] < cnt[q]) {
            const int4 e = D.half[(size_t)as[q] * D.capH + pos[q]];
            if ((int)((unsigned)e.x & kHalfIdMask) == t)
              push(cid[q], (int)((unsigned)e.x >> kHalfTypeShift), e.y,
                   -__int_as_float(e.z), -__int_as_float(e.w), half_first(D, as[q]) + pos[q], false);
          }
      }
      {
        int n = D.half_cnt[s];
        const int4* h = D.half + (size_t)s * D.capH;
        for (int k = 0; k < n; k++) {
          int4 e = h[k];
          push((int)((unsigned)e.x & kHalfIdMask), (int)((unsigned)e.x >> kHalfTypeShift), e.y,
               __int_as_float(e.z), __int_as_float(e.w), half_first(D, s) + k, true);
        }
      }
      {
        const int wc = min(nC, D.capC), ws = min(nS, D.capS);
        if (wc & 1) D.cross[ell(wc - 1, col, D.N2)] = pendC;
        if ((ws & 1) && (KEYS || D.same_entries)) D.same[ell(ws - 1, col, D.N2)] = pendS;
      }
      if (nC > D.capC || nS > D.capS) {
        atomicOr(D.err, ERR_LIST_CAP);
        nC = min(nC, D.capC);
        nS = min(nS, D.capS);
        newC = newS = 0;
      }
      // walk order: [new entries, descending creation] + [old entries, ascending]
      if (newC > 0) {
        reverse_ell<KEYS>(D.cross, D.keyC, D.N2, col, 0, nC);
        reverse_ell<KEYS>(D.cross, D.keyC, D.N2, col, newC, nC);
      }
      if (newS > 0 && (KEYS || D.same_entries)) {
        reverse_ell<KEYS>(D.same, D.keyS, D.N2, col, 0, nS);
        reverse_ell<KEYS>(D.same, D.keyS, D.N2, col, newS, nS);
      }
    }
  }
  D.degC[col] = nC;
  D.degS[col] = nS;
}

// every target's cross and same lists, built from the creators' half lists in the walk
// order of the reference's pair linked list (its reuse and relinking,
// 2_SPH_main_2018.f90:1309-1401).
// dynamic shared memory: 2 x blockDim int4, the waiting even entries of each thread's two
// lists (in registers they cost the list build, which waits on its gathers, an eighth of
// its resident warps)
template <bool KEYS>
__global__ void k_lists(Dev D) {
  extern __shared__ int4 lists_pend[];
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < D.N2)
    lists_target<KEYS>(D, s, lists_pend[threadIdx.x], lists_pend[blockDim.x + threadIdx.x]);
}

}  // namespace

// per-target lists (k_lists), one thread per sorted position; keys: with the walk-order
// keys (and the same-kind entries); same: the same-kind entries even when no step kernel
// reads them (the FP32 free-surface detection does)
void launch_lists(Ctx& c, bool keys, bool same = false) {
  Dev D = c.d;
  if (same) D.same_entries = 1;
  const int b = Ctx::block_for(D.N2, c.blk[TK_LISTS]), nb = (D.N2 + b - 1) / b;
  const size_t pend = 2 * sizeof(int4) * (size_t)b;
  if (keys) k_lists<true><<<nb, b, pend, c.stream>>>(D);
  else k_lists<false><<<nb, b, pend, c.stream>>>(D);
}

// The lists straight from the cell stencil and the remaining positions' counts.  Lanes a target:
// fewer as the problem fills the chip by itself, since a group's ballots and partly filled
// passes cost it two to three times the instructions a target (slopes of the FP32 form, no
// same-kind lists, us with 8 / 4 / 2 lanes / 1: 17,000 targets 26 / - / - / 52; 29,000 30 / 24 /
// 33 / 54; 80,000 57 / 50 / 57 / 58; 320,000 195 / 164 / 152 / 158; 2 million 1188 / 991 / 880 /
// 762; with same-kind lists, 2 million, plain, 2082 / 1792 / 1728 / 2551: one lane's buffers
// leave too few warps a multiprocessor, so that form is not built).  Dynamic shared memory: the
// list capacity for each target of a block, blocks halved until it is within 48 KB.
void launch_gather(Ctx& c, bool same, const Dev& D) {
  const size_t per_target = sizeof(int) * (size_t)(D.capC + (same ? D.capS : 0));
  const int G = D.NT <= 16000 ? 8 : (D.NT <= 100000 ? 4 : (same || D.NT <= 400000 ? 2 : 1));
  if (G == 1) {
    int b = std::min(c.blk[TK_HALF], 512);  // k_fgather's launch bounds
    while (b > 32 && per_target * (size_t)b > 49152) b >>= 1;
    const int bs = (D.NT - D.NN + b - 1) / b, bn = bs + (D.NN + b - 1) / b;
    const int nb = bn + (D.N2 - D.NT + b - 1) / b;
    auto k = D.fast ? k_fgather<false> : k_fgather<true>;
    k<<<nb, b, per_target * b, c.stream>>>(D, bs, bn);
    return;
  }
  int b = Ctx::block_for((int64_t)D.NT * G, 128);
  while (b > 32 && per_target * (b / G) > 49152) b >>= 1;
  const int per = b / G;
  const int bs = (D.NT - D.NN + per - 1) / per, bn = bs + (D.NN + per - 1) / per;
  const int nb = bn + (D.N2 - D.NT + b - 1) / b;
  auto form = [&](auto f, auto p) {
    constexpr bool S = decltype(f)::value, P = decltype(p)::value;
    return G == 8 ? k_fgatherg<S, P, 8> : (G == 4 ? k_fgatherg<S, P, 4> : k_fgatherg<S, P, 2>);
  };
  const std::true_type yes;
  const std::false_type no;
  auto k = same ? (D.fast ? form(yes, no) : form(yes, yes)) : (D.fast ? form(no, no) : form(no, yes));
  k<<<nb, b, per_target * per, c.stream>>>(D, bs, bn);
}

int launch_pair_build(Ctx& c) {
  Dev& D = c.d;
  cudaStream_t st = c.stream;
  const int nb = (D.N2 + kBlock - 1) / kBlock;
  const int b = Ctx::block_for(D.N2, kBlock), nbs = (D.N2 + b - 1) / b;
  c.mark("bbox");
  // 256 to 2048 particles a block: at least as many blocks as fit the chip while there are
  const int per = std::min(8, std::max(1, nb / 608));
  k_bbox<<<(nb + per - 1) / per, kBlock, 0, st>>>(D, per);
  c.mark("cell_count");
  k_cell_count<<<nbs, b, 0, st>>>(D);
  c.mark("scan_cells");
  k_scan_cells<<<(D.cell_cap + 1 + kScan - 1) / kScan, kBlock, 0, st>>>(D);
  c.mark("cell_fill");
  k_cell_fill<<<nbs, b, 0, st>>>(D);
  c.mark("cell_rank");
  k_cell_rank<<<nbs, b, 0, st>>>(D);
  // variant bit 2: a download follows most steps; the exact detection wants the keys, the
  // FP32 detection only the same-kind entries
  const bool want = (c.step_variant & 4) != 0;
  const bool direct = c.lists_direct();
  if (direct) {
    c.mark("gather");
    launch_gather(c, c.same_now(), D);
  } else {
    c.mark("half");
    const int h = Ctx::block_for(D.N2, c.blk[TK_HALF]);
    if (c.precision == SPS_PREC_FP32_FAST) k_half<true><<<(D.N2 + h - 1) / h, h, 0, st>>>(D);
    else k_half<false><<<(D.N2 + h - 1) / h, h, 0, st>>>(D);
  }
  c.mark("scan_half");
  k_scan_half<<<(D.N2 + 1 + kScan - 1) / kScan, kBlock, 0, st>>>(D);
  if (!direct) {
    c.mark("lists");
    launch_lists(c, c.surf_every || (want && !c.surface_f32()), want);
  }
  c.half_stale = direct || c.fused();
  return 0;
}

// both lists of every target from creation order to walk order: in a step that re-interpolates
// before the one-launch stages' preparation, which does it otherwise, and after a rebuild.  Once
// for each gather: it reverses the new pairs of a list.
__global__ void k_walk_order(Dev D) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < D.NT) put_target_walk_order(D, k, D.colid[k], k >= D.NT - D.NN);
}
static void walk_order(Ctx& c, Dev D, bool same) {
  D.same_entries = same;
  const int b = Ctx::block_for(D.NT, kBlock);
  k_walk_order<<<(D.NT + b - 1) / b, b, 0, c.stream>>>(D);
}
void launch_walk_order(Ctx& c) { walk_order(c, c.d, c.same_now()); }

// The device view of the last pair build for a rebuild after the step: the FP64 positions
// the build's exact band test read (x0x, x0y hold them from the step's start, before
// anything moved; the smoothing lengths are constant when the lists are gathered, and an upload
// keeps the ones that it replaces), so the rebuild decides every pair as the build did.  The
// cell-frame offsets and sorted records are the build's own.
Dev build_view(Ctx& c) {
  Dev D = c.d;
  D.px = D.x0x;
  D.py = D.x0y;
  if (c.builds > 0 && c.hbuilt_of == c.builds) {
    // (of a batch, the realisations that no upload has replaced)
    for (size_t r = 0; r < c.hr.size(); r++) {
      if (c.hr[r].kept == c.builds) continue;
      c.hr[r].kept = c.builds;
      const Real& M = c.real[r];
      const int64_t seg[3][2] = {{M.node0, M.nnode}, {M.sp0, M.nsp}, {M.dum0, M.ndum}};
      for (const auto& q : seg)
        if (q[1] > 0)
          SPS_CUDA_CHECK(cudaMemcpyAsync(c.hbuilt + q[0], D.hsml + q[0], sizeof(double) * q[1],
                                         cudaMemcpyDeviceToDevice, c.stream));
    }
    D.hsml = c.hbuilt;
  }
  return D;
}

// the half lists of the last pair build, when it gathered the lists directly: the same pairs,
// counts and creation order
void ensure_half_lists(Ctx& c) {
  if (!c.half_stale) return;
  const int nb = c.grid_of(TK_HALF, c.d.N2), b = c.blk[TK_HALF];
  if (c.d.fast) k_half<true><<<nb, b, 0, c.stream>>>(build_view(c));
  else k_half<false><<<nb, b, 0, c.stream>>>(build_view(c));
  c.half_stale = false;
}

// the lists of the last step again, now with their walk-order keys (the on-demand
// free-surface detection; the lists are rebuilt identically)
void launch_lists_keys(Ctx& c) {
  ensure_half_lists(c);
  launch_lists(c, true);
}

// the lists of the last step again with the same-kind entries (the FP32 detection)
void launch_lists_same(Ctx& c) {
  if (c.lists_direct()) {
    const Dev D = build_view(c);
    launch_gather(c, true, D);
    if (D.walk_order) walk_order(c, D, true);
  } else {
    ensure_half_lists(c);
    launch_lists(c, false, true);
  }
}

}  // namespace sps
