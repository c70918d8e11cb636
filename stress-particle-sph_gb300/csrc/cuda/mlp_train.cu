// mlp_train.cu -- training of the constitutive surrogate (include/sps_surrogate.h):
// forward, backward and Adam kernels, the BF16 fragment packing, and the tensor-core
// prediction path.
//
// Every layer is handled as one matrix product with the bias folded in: the activations
// carry a trailing column of ones and the parameters of a layer, W (K x N) followed by b
// (N), are read as one (K + 1) x N matrix.  So
//   forward   Z   = [A, 1] . [W; b]
//   backward  d[W; b] = [A, 1]^T . dZ,   dA = dZ . W^T
// A minibatch is three launches:
//   k_rows    32 rows a block: the whole forward pass, the loss and the backward pass down to
//             every layer's dZ, the network in shared memory
//   k_wgrad   the four layers' weight gradients, their long reductions (over the rows) split
//             into partial products
//   k_update  the partial products summed in a fixed order, Adam, the next forward pass's
//             rounded weights, the loss sums
// Training is deterministic: the sums of Z and dA are single FP32 multiply-add chains in
// ascending index, whatever the tiling; a weight gradient is at most kSplit such chains over
// consecutive rows, added in order; a loss is a tree over 256 rows at a time, added in order on the host.
// An epoch's order (Fisher-Yates over all rows) is drawn on the host before an epoch's first
// launch: 0.37 ms of the 1.54 that an epoch of 65,536 rows takes.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "common.cuh"
#include "mlp.cuh"
#include "sps_surrogate.h"

static_assert(sps::MLP_NPARAM == SPS_MLP_NPARAM, "parameter count");
static_assert(sps::MLP_TUPLE == SPS_MLP_TUPLE, "tuple size");

namespace {

using namespace sps;

constexpr int kSplit = 16;  // partial products of a weight gradient

#define MLP_CHECK(call)                                                                   \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      throw std::runtime_error(std::string(#call) + ": " + cudaGetErrorString(e_));      \
  } while (0)

__device__ __forceinline__ float bf16r(float v) {
  return __bfloat162float(__float2bfloat16_rn(v));
}

// layer geometry: parameter offset, input width K, output width N
struct Layer {
  int off, K, N;
};
constexpr Layer kLayers[4] = {{MLP_W1, MLP_IN, MLP_H},
                              {MLP_W2, MLP_H, MLP_H},
                              {MLP_W3, MLP_H, MLP_H},
                              {MLP_W4, MLP_H, MLP_OUT}};

__device__ __forceinline__ bool is_bias(int i) {
  return (i >= MLP_B1 && i < MLP_W2) || (i >= MLP_B2 && i < MLP_W3) ||
         (i >= MLP_B3 && i < MLP_W4) || i >= MLP_B4;
}

// the weights the forward pass uses: BF16-rounded weights (quantize), FP32 biases
__global__ void k_quantize(const float* __restrict__ P, float* __restrict__ Wq, int quantize) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= MLP_NPARAM) return;
  float v = P[i];
  Wq[i] = (quantize && !is_bias(i)) ? bf16r(v) : v;
}

// ---- one minibatch ------------------------------------------------------------------------

constexpr int kRows = 32;        // rows a block, four a warp
constexpr int kHS = MLP_H + 4;   // row stride of H = [silu(Z), 1] and of W in shared memory
constexpr int kXS = 20;          // row stride of X = [inputs (14), 0, 0, 1]
constexpr int kWgradTiles = 2 + 6 + 6 + 3;  // 64 x 64 tiles of the four gradients

struct RowsSmem {
  float w1[(MLP_IN + 1) * kHS];
  float w2[(MLP_H + 1) * kHS], w3[(MLP_H + 1) * kHS];
  float w4[(MLP_H + 1) * MLP_OUT];
  float a[kRows * kHS];  // a warp's four rows: activations, then dZ
  float dy[kRows * MLP_OUT];
};

// z of a warp's four rows and a lane's columns lane + 32 c: the chain over k of A(row, k) W(k, n)
// (K values of A in shared memory, then the bias row)
template <int K>
__device__ __forceinline__ void layer_forward(const float* __restrict__ A, int as,
                                              const float* __restrict__ W, int lane,
                                              float (*z)[4]) {
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) z[r][c] = 0.0f;
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    float4 a[4];
#pragma unroll
    for (int r = 0; r < 4; r++) a[r] = *reinterpret_cast<const float4*>(A + r * as + k);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      float b[4];
#pragma unroll
      for (int c = 0; c < 4; c++) b[c] = W[(k + q) * kHS + lane + 32 * c];
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float v = q == 0 ? a[r].x : q == 1 ? a[r].y : q == 2 ? a[r].z : a[r].w;
#pragma unroll
        for (int c = 0; c < 4; c++) z[r][c] = fmaf(v, b[c], z[r][c]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float b = W[K * kHS + lane + 32 * c];
#pragma unroll
    for (int r = 0; r < 4; r++) z[r][c] = fmaf(1.0f, b, z[r][c]);
  }
}
// dA of the same rows and columns: the chain over the outputs j of dZ(row, j) W(n, j)
__device__ __forceinline__ void layer_backward(const float* __restrict__ dZ,
                                               const float* __restrict__ W, int lane,
                                               float (*d)[4]) {
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) d[r][c] = 0.0f;
#pragma unroll 2
  for (int j = 0; j < MLP_H; j += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int r = 0; r < 4; r++) a[r] = *reinterpret_cast<const float4*>(dZ + r * kHS + j);
#pragma unroll
    for (int c = 0; c < 4; c++) b[c] = *reinterpret_cast<const float4*>(W + (lane + 32 * c) * kHS + j);
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) {
        d[r][c] = fmaf(a[r].x, b[c].x, d[r][c]);
        d[r][c] = fmaf(a[r].y, b[c].y, d[r][c]);
        d[r][c] = fmaf(a[r].z, b[c].z, d[r][c]);
        d[r][c] = fmaf(a[r].w, b[c].w, d[r][c]);
      }
  }
}

// Rows r < n of a minibatch (data rows perm[start + r]): X, H = [silu(Z), 1] of the hidden
// layers (BF16-rounded when quantize), dY = 2 (Y - T) / (4 n), dZ of the hidden layers, and the
// rows' squared errors.  A warp owns four rows from the inputs to dZ of the first layer, so
// warps meet only where the network is loaded; its Z stay in registers.  167 KB of shared
// memory, one block an SM: 128 blocks for a minibatch of 4096.  Bound by the shared-memory
// reads of the weights (4 wavefronts for 16 multiply-adds a lane).  With the other two kernels
// a minibatch of 4096 takes three launches in place of twenty-seven.
__global__ void __launch_bounds__(256, 1) k_rows(const float* __restrict__ data,
                                                 const int* __restrict__ perm, long start, int n,
                                                 int quantize, const float* __restrict__ Wq,
                                                 float* __restrict__ X, float* __restrict__ H1,
                                                 float* __restrict__ H2, float* __restrict__ H3,
                                                 float* __restrict__ dY, float* __restrict__ dZ1,
                                                 float* __restrict__ dZ2, float* __restrict__ dZ3,
                                                 float* __restrict__ lrow) {
  extern __shared__ __align__(16) uint8_t rows_raw[];
  RowsSmem& S = *reinterpret_cast<RowsSmem*>(rows_raw);
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  for (int i = tid; i < (MLP_IN + 1) * MLP_H; i += 256)
    S.w1[(i >> 7) * kHS + (i & 127)] = Wq[MLP_W1 + i];
  for (int i = tid; i < (MLP_H + 1) * MLP_H; i += 256) {
    S.w2[(i >> 7) * kHS + (i & 127)] = Wq[MLP_W2 + i];
    S.w3[(i >> 7) * kHS + (i & 127)] = Wq[MLP_W3 + i];
  }
  for (int i = tid; i < (MLP_H + 1) * MLP_OUT; i += 256) S.w4[i] = Wq[MLP_W4 + i];
  const int row0 = blockIdx.x * kRows + 4 * w;
  float* A = S.a + 4 * w * kHS;
  // inputs: lane k of a row its column k (rows past n stay zero and store nothing)
#pragma unroll
  for (int r = 0; r < 4; r++) {
    float v = lane == MLP_IN ? 1.0f : 0.0f;
    if (row0 + r < n) {
      if (lane < MLP_NIN) {
        v = data[(size_t)perm[start + row0 + r] * MLP_TUPLE + lane];
        if (quantize) v = bf16r(v);
      }
      if (lane < kXS) X[(size_t)(row0 + r) * kXS + lane] = v;
    }
    if (lane < kXS) A[r * kHS + lane] = v;
  }
  __syncthreads();

  float z1[4][4], z2[4][4], z3[4][4];
  auto activate = [&](const float (*z)[4], float* __restrict__ H) {
    __syncwarp();  // every lane has read the rows
#pragma unroll
    for (int r = 0; r < 4; r++) {
#pragma unroll
      for (int c = 0; c < 4; c++) {
        float v = silu(z[r][c]);
        if (quantize) v = bf16r(v);
        A[r * kHS + lane + 32 * c] = v;
        if (row0 + r < n) H[(size_t)(row0 + r) * kHS + lane + 32 * c] = v;
      }
      if (lane == 0) {
        A[r * kHS + MLP_H] = 1.0f;
        if (row0 + r < n) H[(size_t)(row0 + r) * kHS + MLP_H] = 1.0f;
      }
    }
    __syncwarp();
  };
  layer_forward<MLP_IN>(A, kHS, S.w1, lane, z1);
  activate(z1, H1);
  layer_forward<MLP_H>(A, kHS, S.w2, lane, z2);
  activate(z2, H2);
  layer_forward<MLP_H>(A, kHS, S.w3, lane, z3);
  activate(z3, H3);
  {  // output layer and loss: lane 8 r + c holds output c of row r
    const int r = lane >> 3, c = lane & 7, row = row0 + r;
    float y = 0.0f;
#pragma unroll 4
    for (int k = 0; k <= MLP_H; k++) y = fmaf(A[r * kHS + k], S.w4[k * MLP_OUT + c], y);
    const float sc = 2.0f / (4.0f * (float)n);
    float d = 0.0f;
    if (row < n && c < MLP_NOUT) d = y - data[(size_t)perm[start + row] * MLP_TUPLE + MLP_NIN + c];
    float l = 0.0f;
#pragma unroll
    for (int q = 0; q < MLP_NOUT; q++) {
      const float dq = __shfl_sync(0xffffffffu, d, (lane & 24) + q);
      l = fmaf(dq, dq, l);
    }
    S.dy[(4 * w + r) * MLP_OUT + c] = sc * d;
    if (row < n) {
      dY[(size_t)row * MLP_OUT + c] = sc * d;
      if (c == 0) lrow[row] = l;
    }
    __syncwarp();
  }
  // dZ = dA silu'(Z), kept as the warp's rows
  auto through = [&](const float (*d)[4], const float (*z)[4], float* __restrict__ dZ) {
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float zz = z[r][c];
        const float sg = 1.0f / (1.0f + expf(-zz));
        const float v = d[r][c] * (sg * (1.0f + zz * (1.0f - sg)));
        A[r * kHS + lane + 32 * c] = v;
        if (row0 + r < n) dZ[(size_t)(row0 + r) * MLP_H + lane + 32 * c] = v;
      }
    __syncwarp();
  };
  float d[4][4];
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int c = 0; c < 4; c++) {
      float v = 0.0f;
#pragma unroll
      for (int k = 0; k < MLP_OUT; k++)
        v = fmaf(S.dy[(4 * w + r) * MLP_OUT + k], S.w4[(lane + 32 * c) * MLP_OUT + k], v);
      d[r][c] = v;
    }
  through(d, z3, dZ3);
  layer_backward(A, S.w3, lane, d);
  through(d, z2, dZ2);
  layer_backward(A, S.w2, lane, d);
  through(d, z1, dZ1);
}

struct WgradLayer {
  const float *A, *dZ;  // A (n x (K + 1), stride as), dZ (n x N)
  int as, K, N, off;
};
struct WgradArgs {
  WgradLayer l[4];
};
// part[z][i]: the weight gradient d[W; b] = [A, 1]^T . dZ of the rows of split z, every layer's at
// its parameters' place; 64 x 64 tiles (blockIdx.x), 256 threads with 4 x 4 outputs each
__global__ void __launch_bounds__(256) k_wgrad(WgradArgs args, int n, int kchunk,
                                               float* __restrict__ part) {
  __shared__ __align__(16) float As[16][68];
  __shared__ __align__(16) float Bs[16][68];
  int tile = blockIdx.x, li = 0;
  if (tile >= 2) {
    tile -= 2;
    li = 1 + tile / 6;
    tile = li < 3 ? tile % 6 : tile - 12;
    if (li > 3) li = 3;
  }
  const WgradLayer L = args.l[li];
  const int M = L.K + 1, N = L.N, nt = (N + 63) / 64;
  const int m0 = tile / nt * 64, n0 = tile % nt * 64;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int kbeg = blockIdx.y * kchunk, kend = min(n, kbeg + kchunk);
  float acc[4][4] = {};
  const int mm = tid & 63, k4 = tid >> 6;  // a thread's column and rows k4 + 4 i of a step
  float ra[4], rb[4];
  auto fetch = [&](int kb) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int k = kb + k4 + 4 * i;
      ra[i] = m0 + mm < M && k < kend ? L.A[(size_t)k * L.as + m0 + mm] : 0.0f;
      rb[i] = n0 + mm < N && k < kend ? L.dZ[(size_t)k * N + n0 + mm] : 0.0f;
    }
  };
  fetch(kbeg);
  for (int kb = kbeg; kb < kend; kb += 16) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      As[k4 + 4 * i][mm] = ra[i];
      Bs[k4 + 4 * i][mm] = rb[i];
    }
    __syncthreads();
    if (kb + 16 < kend) fetch(kb + 16);  // the next step's rows while this one is summed
#pragma unroll
    for (int kk = 0; kk < 16; kk++) {
      const float4 a = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
  float* C = part + (size_t)blockIdx.y * MLP_NPARAM + L.off;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int c = n0 + tx * 4 + j;
      if (c < N) C[(size_t)m * N + c] = acc[i][j];
    }
  }
}

// The gradient (the splits summed in order), with `adam` the update and the rounded weights of
// the next forward pass; the blocks after the parameters' sum 256 rows' squared errors each
// into lossp
__global__ void __launch_bounds__(256) k_update(const float* __restrict__ part, int nsplit,
                                                float* __restrict__ G, float* __restrict__ P,
                                                float* __restrict__ Wq, float* __restrict__ Mo,
                                                float* __restrict__ Vo, int adam, int quantize,
                                                float lr, float b1, float b2, float eps, float bc1,
                                                float bc2, const float* __restrict__ lrow, int n,
                                                float* __restrict__ lossp) {
  constexpr int pb = (MLP_NPARAM + 255) / 256;
  if ((int)blockIdx.x >= pb) {
    __shared__ float sh[256];
    const int b = blockIdx.x - pb, r = b * 256 + threadIdx.x;
    sh[threadIdx.x] = r < n ? lrow[r] : 0.0f;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
      if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
      __syncthreads();
    }
    if (threadIdx.x == 0) lossp[b] = sh[0];
    return;
  }
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= MLP_NPARAM) return;
  float g = 0.0f;
#pragma unroll 4
  for (int z = 0; z < nsplit; z++) g += part[(size_t)z * MLP_NPARAM + i];
  G[i] = g;
  if (!adam) return;
  float m = b1 * Mo[i] + (1.0f - b1) * g;
  float v = b2 * Vo[i] + (1.0f - b2) * (g * g);
  Mo[i] = m;
  Vo[i] = v;
  const float p = P[i] - lr * (m / bc1) / (sqrtf(v / bc2) + eps);
  P[i] = p;
  Wq[i] = (quantize && !is_bias(i)) ? bf16r(p) : p;
}

// B-operand registers of mma.m16n8k16 (row.col, BF16) for every tile and lane:
// lane = 4 g + t holds {W[k0 + 2t][n0 + g], W[k0 + 2t + 1][n0 + g]} and the same at
// k0 + 8 + 2t; biases copied as FP32
__global__ void k_pack(const float* __restrict__ P, uint2* __restrict__ frag,
                       float* __restrict__ bias) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < MLP_BIAS) {
    int src = i < MLP_H ? MLP_B1 + i
              : i < 2 * MLP_H ? MLP_B2 + (i - MLP_H)
              : i < 3 * MLP_H ? MLP_B3 + (i - 2 * MLP_H)
                              : MLP_B4 + (i - 3 * MLP_H);
    bias[i] = P[src];
  }
  if (i >= MLP_FRAG_U2) return;
  int tile = i >> 5, lane = i & 31, g = lane >> 2, t = lane & 3;
  int off, N, local, NT;
  if (tile < MLP_T1) {
    off = MLP_W1, N = MLP_H, NT = 16, local = tile;
  } else if (tile < MLP_T1 + MLP_T2) {
    off = MLP_W2, N = MLP_H, NT = 16, local = tile - MLP_T1;
  } else if (tile < MLP_T1 + MLP_T2 + MLP_T3) {
    off = MLP_W3, N = MLP_H, NT = 16, local = tile - MLP_T1 - MLP_T2;
  } else {
    off = MLP_W4, N = MLP_OUT, NT = 1, local = tile - MLP_T1 - MLP_T2 - MLP_T3;
  }
  int kt = local / NT, nt = local % NT;
  int n = nt * 8 + g, k = kt * 16 + 2 * t;
  const float* W = P + off;
  frag[i] = make_uint2(pack_bf16(W[k * N + n], W[(k + 1) * N + n]),
                       pack_bf16(W[(k + 8) * N + n], W[(k + 9) * N + n]));
}

// y (n x 4) = network(x (n x 14)) by the tensor-core code of the step; 4 warps per
// block, 32 rows per warp, every lane of a warp takes part in both 16-row tiles
__global__ void __launch_bounds__(128) k_predict(const uint2* __restrict__ frag,
                                                 const float* __restrict__ bias,
                                                 const float* __restrict__ x, int n,
                                                 float* __restrict__ y) {
  __shared__ float xs[4][32][16];
  __shared__ float ys[4][32][8];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long row = (blockIdx.x * 4L + w) * 32 + lane;
  for (int k = 0; k < 16; k++)
    xs[w][lane][k] = (row < n && k < MLP_NIN) ? x[row * MLP_NIN + k] : 0.0f;
  __syncwarp();
  mlp_tile16(frag, bias, &xs[w][0][0], &ys[w][0][0], lane);
  mlp_tile16(frag, bias, &xs[w][16][0], &ys[w][16][0], lane);
  __syncwarp();
  if (row < n)
    for (int k = 0; k < MLP_NOUT; k++) y[row * MLP_NOUT + k] = ys[w][lane][k];
}

uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

double uniform01(uint64_t& s) { return (splitmix(s) >> 11) * 0x1.0p-53; }

}  // namespace

struct sps_mlp {
  sps_mlp_config cfg{};
  cudaStream_t stream = nullptr;
  std::vector<void*> allocs;
  float *P = nullptr, *Wq = nullptr, *G = nullptr, *Mo = nullptr, *Vo = nullptr;
  float *part = nullptr, *X = nullptr, *dY = nullptr, *lrow = nullptr;
  float *H[3] = {}, *dZ[3] = {};
  float* lossp = nullptr;
  int lossp_cap = 0;
  float* data = nullptr;
  int64_t ndata = 0, data_cap = 0;
  int* perm = nullptr;
  int64_t perm_cap = 0;
  int* ident = nullptr;
  float* gtuples = nullptr;
  uint2* frag = nullptr;
  float* bias = nullptr;
  void* tc_img = nullptr;   // the network as the tensor-core kernel's shared-memory image
  float* tc_bias = nullptr;
  int* tc_err = nullptr;
  float *px = nullptr, *py = nullptr;
  int64_t pred_cap = 0;
  bool tensor_memory_path = true;  // sps_mlp_predict: tcgen05 (else the warp-level mma.sync)
  int64_t adam_t = 0;
  uint64_t rng = 0;
  std::string err;

  template <typename T>
  T* alloc(size_t n) {
    void* p = nullptr;
    MLP_CHECK(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)));
    allocs.push_back(p);
    return static_cast<T*>(p);
  }
  void release(void* p) {
    if (!p) return;
    for (auto& a : allocs)
      if (a == p) {
        cudaFree(a);
        a = nullptr;
      }
  }
  ~sps_mlp() {
    if (stream) cudaStreamSynchronize(stream);
    for (void* p : allocs)
      if (p) cudaFree(p);
    if (stream) cudaStreamDestroy(stream);
  }

  // forward, loss and backward of n rows (data rows perm[start ...]) with the weights Wq; the
  // gradient into G, per-256-row squared errors into lossp[lo ...]; adam: one update of the
  // parameters and Wq with the learning rate lr
  void minibatch(const float* rows, const int* order, long start, int n, int lo, bool adam,
                 float lr, float bc1, float bc2) {
    k_rows<<<(n + kRows - 1) / kRows, 256, sizeof(RowsSmem), stream>>>(
        rows, order, start, n, cfg.quantize, Wq, X, H[0], H[1], H[2], dY, dZ[0], dZ[1], dZ[2], lrow);
    const int kchunk = ((n + kSplit - 1) / kSplit + 15) / 16 * 16;
    const int nsplit = (n + kchunk - 1) / kchunk;
    WgradArgs args = {{{X, dZ[0], kXS, MLP_IN, MLP_H, MLP_W1},
                       {H[0], dZ[1], kHS, MLP_H, MLP_H, MLP_W2},
                       {H[1], dZ[2], kHS, MLP_H, MLP_H, MLP_W3},
                       {H[2], dY, kHS, MLP_H, MLP_OUT, MLP_W4}}};
    k_wgrad<<<dim3(kWgradTiles, nsplit), 256, 0, stream>>>(args, n, kchunk, part);
    k_update<<<(MLP_NPARAM + 255) / 256 + (n + 255) / 256, 256, 0, stream>>>(
        part, nsplit, G, P, Wq, Mo, Vo, adam ? 1 : 0, cfg.quantize, lr, cfg.beta1, cfg.beta2,
        cfg.eps, bc1, bc2, lrow, n, lossp + lo);
  }
  void quantize() {
    k_quantize<<<(MLP_NPARAM + 255) / 256, 256, 0, stream>>>(P, Wq, cfg.quantize);
  }
  void ensure_lossp(int n) {
    if (n <= lossp_cap) return;
    release(lossp);
    lossp = alloc<float>(n);
    lossp_cap = n;
  }
};

namespace {

int mfail(sps_mlp* m, int rc, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  std::vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (m) m->err = buf;
  return rc;
}

}  // namespace

namespace sps {
// used by the step's surrogate installation (sps_api.cu)
void mlp_pack(sps_mlp* m, uint2* frag, float* bias, cudaStream_t st) {
  k_pack<<<(MLP_FRAG_U2 + 255) / 256, 256, 0, st>>>(m->P, frag, bias);
}
cudaStream_t mlp_stream(sps_mlp* m) { return m->stream; }
const float* mlp_params(sps_mlp* m) { return m->P; }
}  // namespace sps

extern "C" {

int sps_mlp_create(const sps_mlp_config* cfg, sps_mlp** out) {
  if (!cfg || !out) return SPS_ERR_ARG;
  *out = nullptr;
  if (cfg->batch < 64 || cfg->batch > 65536 || cfg->batch % 64) return SPS_ERR_ARG;
  sps_mlp* m = new (std::nothrow) sps_mlp;
  if (!m) return SPS_ERR_CUDA;
  try {
    m->cfg = *cfg;
    m->rng = cfg->seed;
    MLP_CHECK(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
    const int B = cfg->batch;
    m->P = m->alloc<float>(MLP_NPARAM);
    m->Wq = m->alloc<float>(MLP_NPARAM);
    m->G = m->alloc<float>(MLP_NPARAM);
    m->Mo = m->alloc<float>(MLP_NPARAM);
    m->Vo = m->alloc<float>(MLP_NPARAM);
    m->part = m->alloc<float>((size_t)kSplit * MLP_NPARAM);
    m->X = m->alloc<float>((size_t)B * kXS);
    m->dY = m->alloc<float>((size_t)B * MLP_OUT);
    m->lrow = m->alloc<float>(B);
    for (int l = 0; l < 3; l++) {
      m->H[l] = m->alloc<float>((size_t)B * kHS);
      m->dZ[l] = m->alloc<float>((size_t)B * MLP_H);
    }
    MLP_CHECK(cudaFuncSetAttribute(k_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(RowsSmem)));
    m->ident = m->alloc<int>(B);
    m->gtuples = m->alloc<float>((size_t)B * MLP_TUPLE);
    m->frag = m->alloc<uint2>(MLP_FRAG_U2);
    m->tc_img = m->alloc<uint8_t>(sps::mlp_tc_image_bytes());
    m->tc_bias = m->alloc<float>(sps::mlp_tc_bias_count());
    m->tc_err = m->alloc<int>(1);
    m->bias = m->alloc<float>(MLP_BIAS);
    m->ensure_lossp((B + 255) / 256);
    // Glorot-uniform weights, zero biases and padding
    std::vector<float> p(MLP_NPARAM, 0.0f);
    uint64_t s = cfg->seed ^ 0x5eed5eed5eedull;
    for (const Layer& L : kLayers) {
      int kin = (L.off == MLP_W1) ? MLP_NIN : L.K;
      int nout = (L.off == MLP_W4) ? MLP_NOUT : L.N;
      double a = std::sqrt(6.0 / (kin + nout));
      for (int k = 0; k < kin; k++)
        for (int n = 0; n < nout; n++) p[L.off + k * L.N + n] = (float)((2.0 * uniform01(s) - 1.0) * a);
    }
    std::vector<int> id(B);
    for (int i = 0; i < B; i++) id[i] = i;
    MLP_CHECK(cudaMemcpyAsync(m->P, p.data(), sizeof(float) * MLP_NPARAM, cudaMemcpyHostToDevice, m->stream));
    MLP_CHECK(cudaMemcpyAsync(m->ident, id.data(), sizeof(int) * B, cudaMemcpyHostToDevice, m->stream));
    MLP_CHECK(cudaMemsetAsync(m->Mo, 0, sizeof(float) * MLP_NPARAM, m->stream));
    MLP_CHECK(cudaMemsetAsync(m->Vo, 0, sizeof(float) * MLP_NPARAM, m->stream));
    MLP_CHECK(cudaStreamSynchronize(m->stream));
  } catch (const std::exception& e) {
    delete m;
    return SPS_ERR_CUDA;
  }
  *out = m;
  return SPS_OK;
}

int sps_mlp_get_params(sps_mlp* m, float* params) {
  if (!m || !params) return SPS_ERR_ARG;
  try {
    MLP_CHECK(cudaMemcpyAsync(params, m->P, sizeof(float) * MLP_NPARAM, cudaMemcpyDeviceToHost, m->stream));
    MLP_CHECK(cudaStreamSynchronize(m->stream));
  } catch (const std::exception& e) {
    return mfail(m, SPS_ERR_CUDA, "%s", e.what());
  }
  return SPS_OK;
}

int sps_mlp_set_params(sps_mlp* m, const float* params) {
  if (!m || !params) return SPS_ERR_ARG;
  try {
    MLP_CHECK(cudaMemcpyAsync(m->P, params, sizeof(float) * MLP_NPARAM, cudaMemcpyHostToDevice, m->stream));
    MLP_CHECK(cudaMemsetAsync(m->Mo, 0, sizeof(float) * MLP_NPARAM, m->stream));
    MLP_CHECK(cudaMemsetAsync(m->Vo, 0, sizeof(float) * MLP_NPARAM, m->stream));
    MLP_CHECK(cudaStreamSynchronize(m->stream));
    m->adam_t = 0;
  } catch (const std::exception& e) {
    return mfail(m, SPS_ERR_CUDA, "%s", e.what());
  }
  return SPS_OK;
}

int sps_mlp_set_data(sps_mlp* m, const float* tuples, int64_t n) {
  if (!m || n < 0 || (n > 0 && !tuples)) return SPS_ERR_ARG;
  if (n > (int64_t)1 << 30) return mfail(m, SPS_ERR_CAPACITY, "at most 2^30 tuples");
  try {
    if (n > m->data_cap) {
      m->release(m->data);
      m->release(m->perm);
      m->data = m->alloc<float>((size_t)n * MLP_TUPLE);
      m->perm = m->alloc<int>(n);
      m->data_cap = m->perm_cap = n;
    }
    if (n)
      MLP_CHECK(cudaMemcpyAsync(m->data, tuples, sizeof(float) * MLP_TUPLE * n,
                                cudaMemcpyHostToDevice, m->stream));
    MLP_CHECK(cudaStreamSynchronize(m->stream));
    m->ndata = n;
  } catch (const std::exception& e) {
    return mfail(m, SPS_ERR_CUDA, "%s", e.what());
  }
  return SPS_OK;
}

int sps_mlp_train(sps_mlp* m, int32_t epochs, float lr, float* loss) {
  if (!m || epochs < 0) return SPS_ERR_ARG;
  const int B = m->cfg.batch;
  const int64_t nmb = m->ndata / B;
  if (epochs > 0 && nmb == 0) return mfail(m, SPS_ERR_STATE, "fewer tuples than one minibatch");
  const int per = (B + 255) / 256;
  if (!(lr > 0.0f)) lr = m->cfg.lr;
  try {
    m->ensure_lossp((int)(nmb * per));
    std::vector<int> perm(m->ndata);
    std::vector<float> lp;
    if (epochs > 0) m->quantize();  // k_update keeps the rounded weights from here on
    for (int ep = 0; ep < epochs; ep++) {
      for (int64_t i = 0; i < m->ndata; i++) perm[i] = (int)i;
      for (int64_t i = m->ndata - 1; i > 0; i--) {  // Fisher-Yates
        int64_t j = (int64_t)(splitmix(m->rng) % (uint64_t)(i + 1));
        std::swap(perm[i], perm[j]);
      }
      MLP_CHECK(cudaMemcpyAsync(m->perm, perm.data(), sizeof(int) * m->ndata,
                                cudaMemcpyHostToDevice, m->stream));
      for (int64_t b = 0; b < nmb; b++) {
        m->adam_t++;
        float bc1 = (float)(1.0 - std::pow((double)m->cfg.beta1, (double)m->adam_t));
        float bc2 = (float)(1.0 - std::pow((double)m->cfg.beta2, (double)m->adam_t));
        m->minibatch(m->data, m->perm, b * B, B, (int)(b * per), true, lr, bc1, bc2);
      }
      MLP_CHECK(cudaGetLastError());
      lp.resize(nmb * per);
      MLP_CHECK(cudaMemcpyAsync(lp.data(), m->lossp, sizeof(float) * lp.size(),
                                cudaMemcpyDeviceToHost, m->stream));
      MLP_CHECK(cudaStreamSynchronize(m->stream));
      double s = 0.0;
      for (float v : lp) s += v;
      if (loss) loss[ep] = (float)(s / ((double)nmb * B * MLP_NOUT));
    }
  } catch (const std::exception& e) {
    return mfail(m, SPS_ERR_CUDA, "%s", e.what());
  }
  return SPS_OK;
}

int sps_mlp_grad(sps_mlp* m, const float* tuples, int32_t n, float* grad, float* loss) {
  if (!m || !tuples || !grad || n <= 0 || n > m->cfg.batch) return SPS_ERR_ARG;
  try {
    MLP_CHECK(cudaMemcpyAsync(m->gtuples, tuples, sizeof(float) * MLP_TUPLE * n,
                              cudaMemcpyHostToDevice, m->stream));
    m->quantize();
    m->minibatch(m->gtuples, m->ident, 0, n, 0, false, 0.0f, 1.0f, 1.0f);
    MLP_CHECK(cudaGetLastError());
    std::vector<float> lp((n + 255) / 256);
    MLP_CHECK(cudaMemcpyAsync(grad, m->G, sizeof(float) * MLP_NPARAM, cudaMemcpyDeviceToHost, m->stream));
    MLP_CHECK(cudaMemcpyAsync(lp.data(), m->lossp, sizeof(float) * lp.size(), cudaMemcpyDeviceToHost, m->stream));
    MLP_CHECK(cudaStreamSynchronize(m->stream));
    double s = 0.0;
    for (float v : lp) s += v;
    if (loss) *loss = (float)(s / (4.0 * n));
  } catch (const std::exception& e) {
    return mfail(m, SPS_ERR_CUDA, "%s", e.what());
  }
  return SPS_OK;
}

int sps_mlp_predict(sps_mlp* m, const float* x, int32_t n, float* y) {
  if (!m || n < 0 || (n > 0 && (!x || !y))) return SPS_ERR_ARG;
  if (n == 0) return SPS_OK;
  try {
    if (n > m->pred_cap) {
      m->release(m->px);
      m->release(m->py);
      m->px = m->alloc<float>((size_t)n * MLP_NIN);
      m->py = m->alloc<float>((size_t)n * MLP_NOUT);
      m->pred_cap = n;
    }
    MLP_CHECK(cudaMemcpyAsync(m->px, x, sizeof(float) * MLP_NIN * n, cudaMemcpyHostToDevice, m->stream));
    int herr = 0;
    if (m->tensor_memory_path) {
      // the step's inference: 128-row tiles on tcgen05 with tensor-memory accumulators
      int dev = 0, nsm = 0;
      MLP_CHECK(cudaGetDevice(&dev));
      MLP_CHECK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
      MLP_CHECK(sps::mlp_tc_prepare());
      sps::mlp_tc_pack(m->P, m->tc_img, m->tc_bias, m->stream);
      MLP_CHECK(cudaMemsetAsync(m->tc_err, 0, sizeof(int), m->stream));
      MLP_CHECK(sps::mlp_tc_forward(m->tc_img, m->tc_bias, m->px, MLP_NIN, MLP_NIN, nullptr, n,
                                    m->py, MLP_NOUT, m->tc_err, 1, sps::mlp_tc_grid(n, nsm),
                                    m->stream));
      MLP_CHECK(cudaMemcpyAsync(&herr, m->tc_err, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    } else {
      // the warp-level mma.sync inference
      sps::mlp_pack(m, m->frag, m->bias, m->stream);
      k_predict<<<(n + 127) / 128, 128, 0, m->stream>>>(m->frag, m->bias, m->px, n, m->py);
    }
    MLP_CHECK(cudaGetLastError());
    MLP_CHECK(cudaMemcpyAsync(y, m->py, sizeof(float) * MLP_NOUT * n, cudaMemcpyDeviceToHost, m->stream));
    MLP_CHECK(cudaStreamSynchronize(m->stream));
    if (herr) return mfail(m, SPS_ERR_CUDA, "tensor-core inference: a wait ran out");
  } catch (const std::exception& e) {
    return mfail(m, SPS_ERR_CUDA, "%s", e.what());
  }
  return SPS_OK;
}

int sps_mlp_set_inference(sps_mlp* m, int32_t tensor_memory) {
  if (!m || (tensor_memory != 0 && tensor_memory != 1)) return SPS_ERR_ARG;
  m->tensor_memory_path = tensor_memory == 1;
  return SPS_OK;
}

int sps_mlp_last_error(sps_mlp* m, char* buf, int32_t len) {
  if (!m || !buf || len <= 0) return 0;
  std::snprintf(buf, (size_t)len, "%s", m->err.c_str());
  return (int)m->err.size();
}

void sps_mlp_destroy(sps_mlp* m) { delete m; }

}  // extern "C"
