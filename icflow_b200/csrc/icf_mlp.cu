// icf_mlp.cu -- the learned Newton warm start: a per-node MLP 15 -> 64 -> 64 -> 3
// with GELU, BF16 weights and FP32 accumulation, with its own training.
//
// No counterpart in the reference: icFlow starts every Newton loop from
// du = v h (ImplicitModel3.cs:149-156).  The network predicts a correction
// to that guess from each node's (u, v, a, du_{n-1}, du_{n-2}) (15 inputs,
// normalised with fixed per-input shifts and scales); the guess is
// du = v h + out_scale * net(x).  With a zero network the plain guess comes
// back unchanged.
//
// Forward: one warp per 16 nodes, bf16 mma.sync m16n8k16 with FP32
// accumulators; each layer's accumulator fragments are re-used in registers
// as the next layer's A fragments (the C layout of two adjacent 8-column
// tiles is the A layout of one 16-column k-step).  Weights sit in shared
// memory as bf16.  Rounding points: the inputs and the two hidden activations
// are rounded to bf16 before each product; biases, GELU and all sums are
// FP32.
//
// Training: forward, FP32 CUDA-core backward and weight-gradient partials of 32
// nodes per block in one kernel, a fixed order reduction of the partials (no
// atomics: a gradient is identical run to run), and Adam on FP32 master
// weights, after which the bf16 copies are refreshed.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <utility>
#include <cstring>
#include <string>
#include <vector>

#include "icf_internal.cuh"

#define NI 15   // inputs
#define NH 64   // hidden width
#define NO 3    // outputs
// parameter layout: W1[64][15] b1[64] W2[64][64] b2[64] W3[3][64] b3[3]
#define OFF_W1 0
#define OFF_B1 (OFF_W1 + NH * NI)
#define OFF_W2 (OFF_B1 + NH)
#define OFF_B2 (OFF_W2 + NH * NH)
#define OFF_W3 (OFF_B2 + NH)
#define OFF_B3 (OFF_W3 + NO * NH)
#define NPAR (OFF_B3 + NO)

struct icf_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string err;
  float *d_master = nullptr;  // FP32 parameters (NPAR)
  float *d_m = nullptr, *d_v = nullptr;  // Adam moments
  __nv_bfloat16 *d_wb = nullptr;  // bf16 weights, padded: W1 64x16, W2 64x64, W3 8x64
  float *d_norm = nullptr;        // in_shift[15], in_scale[15], out_scale[3]
  long long adam_t = 0;
  // inputs, outputs, targets (or output gradients), activations of
  // forward_trace, gradient partials and losses, with their elements
  float *d_x = nullptr, *d_out = nullptr, *d_y = nullptr;
  float *d_z1 = nullptr, *d_h1 = nullptr, *d_z2 = nullptr, *d_h2 = nullptr;
  float *d_part = nullptr, *d_loss = nullptr, *d_grad = nullptr;
  long long x_cap = 0, out_cap = 0, y_cap = 0, z1_cap = 0, h1_cap = 0, z2_cap = 0, h2_cap = 0, part_cap = 0,
            loss_cap = 0;
};

namespace {

constexpr int WB_W1 = 0, WB_W2 = NH * 16, WB_W3 = WB_W2 + NH * NH, WB_N = WB_W3 + 8 * NH;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
// d/dz GELU = Phi(z) + z phi(z)
__device__ __forceinline__ float gelu_d(float z) {
  const float Phi = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
  const float phi = 0.39894228040143268f * expf(-0.5f * z * z);
  return Phi + z * phi;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ void mma_bf16(float c[4], const uint32_t a[4], const uint32_t b[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// B fragment of W (row-major [rows][ld] bf16) for n-tile j, k-step kk:
// element (k, n) = W[8j + n][16kk + k]
__device__ __forceinline__ void bfrag(const __nv_bfloat16 *W, int ld, int j, int kk, int lane, uint32_t b[2]) {
  const int g = lane >> 2, t = lane & 3;
  const __nv_bfloat16 *row = W + (size_t)(8 * j + g) * ld + 16 * kk + 2 * t;
  b[0] = *reinterpret_cast<const uint32_t *>(row);
  b[1] = *reinterpret_cast<const uint32_t *>(row + 8);
}

struct fwd_out {
  float z1[8][4], z2[8][4], y[4];
};

// Forward of 16 nodes [r0, r0 + 16) (rows >= n read as zeros).  Inputs are
// normalised here.  Returns the pre-activations and the output fragment.
__device__ __forceinline__ void mlp_forward16(const float *__restrict__ x, int n, int r0, const __nv_bfloat16 *sW,
                                              const float *sB, const float *sNorm, int lane, fwd_out &f) {
  const int g = lane >> 2, t = lane & 3;
  // A fragment of the normalised inputs (16 x 16, column 15 zero)
  auto xin = [&](int r, int c) -> float {
    if (r >= n || c >= NI) return 0.f;
    return (x[(size_t)r * NI + c] - sNorm[c]) * sNorm[NI + c];
  };
  uint32_t a[4];
  a[0] = pack_bf16(xin(r0 + g, 2 * t), xin(r0 + g, 2 * t + 1));
  a[1] = pack_bf16(xin(r0 + g + 8, 2 * t), xin(r0 + g + 8, 2 * t + 1));
  a[2] = pack_bf16(xin(r0 + g, 2 * t + 8), xin(r0 + g, 2 * t + 9));
  a[3] = pack_bf16(xin(r0 + g + 8, 2 * t + 8), xin(r0 + g + 8, 2 * t + 9));
  // layer 1
#pragma unroll
  for (int j = 0; j < 8; j++) {
    f.z1[j][0] = f.z1[j][1] = f.z1[j][2] = f.z1[j][3] = 0.f;
    uint32_t b[2];
    bfrag(sW + WB_W1, 16, j, 0, lane, b);
    mma_bf16(f.z1[j], a, b);
    const float b0 = sB[OFF_B1 + 8 * j + 2 * t], b1 = sB[OFF_B1 + 8 * j + 2 * t + 1];
    f.z1[j][0] += b0; f.z1[j][1] += b1; f.z1[j][2] += b0; f.z1[j][3] += b1;
  }
  // layer 2: A fragments from GELU(z1) of tiles 2kk, 2kk + 1
#pragma unroll
  for (int j = 0; j < 8; j++) f.z2[j][0] = f.z2[j][1] = f.z2[j][2] = f.z2[j][3] = 0.f;
#pragma unroll
  for (int kk = 0; kk < 4; kk++) {
    uint32_t ah[4];
    ah[0] = pack_bf16(gelu(f.z1[2 * kk][0]), gelu(f.z1[2 * kk][1]));
    ah[1] = pack_bf16(gelu(f.z1[2 * kk][2]), gelu(f.z1[2 * kk][3]));
    ah[2] = pack_bf16(gelu(f.z1[2 * kk + 1][0]), gelu(f.z1[2 * kk + 1][1]));
    ah[3] = pack_bf16(gelu(f.z1[2 * kk + 1][2]), gelu(f.z1[2 * kk + 1][3]));
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint32_t b[2];
      bfrag(sW + WB_W2, NH, j, kk, lane, b);
      mma_bf16(f.z2[j], ah, b);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const float b0 = sB[OFF_B2 + 8 * j + 2 * t], b1 = sB[OFF_B2 + 8 * j + 2 * t + 1];
    f.z2[j][0] += b0; f.z2[j][1] += b1; f.z2[j][2] += b0; f.z2[j][3] += b1;
  }
  // layer 3 (W3 padded to 8 rows)
  f.y[0] = f.y[1] = f.y[2] = f.y[3] = 0.f;
#pragma unroll
  for (int kk = 0; kk < 4; kk++) {
    uint32_t ah[4];
    ah[0] = pack_bf16(gelu(f.z2[2 * kk][0]), gelu(f.z2[2 * kk][1]));
    ah[1] = pack_bf16(gelu(f.z2[2 * kk][2]), gelu(f.z2[2 * kk][3]));
    ah[2] = pack_bf16(gelu(f.z2[2 * kk + 1][0]), gelu(f.z2[2 * kk + 1][1]));
    ah[3] = pack_bf16(gelu(f.z2[2 * kk + 1][2]), gelu(f.z2[2 * kk + 1][3]));
    uint32_t b[2];
    bfrag(sW + WB_W3, NH, 0, kk, lane, b);
    mma_bf16(f.y, ah, b);
  }
  const int c0 = 2 * t, c1 = 2 * t + 1;
  if (c0 < NO) { f.y[0] += sB[OFF_B3 + c0]; f.y[2] += sB[OFF_B3 + c0]; }
  if (c1 < NO) { f.y[1] += sB[OFF_B3 + c1]; f.y[3] += sB[OFF_B3 + c1]; }
}

__device__ __forceinline__ void load_params(const __nv_bfloat16 *wb, const float *master, const float *norm,
                                            __nv_bfloat16 *sW, float *sB, float *sNorm) {
  for (int i = threadIdx.x; i < WB_N; i += blockDim.x) sW[i] = wb[i];
  for (int i = threadIdx.x; i < NPAR; i += blockDim.x) sB[i] = master[i];
  for (int i = threadIdx.x; i < 2 * NI + NO; i += blockDim.x) sNorm[i] = norm[i];
  __syncthreads();
}

// inference: y[n][3] = network output (normalised output units)
__global__ void __launch_bounds__(256) k_mlp_infer(int n, const float *__restrict__ x, const __nv_bfloat16 *wb,
                                                   const float *master, const float *norm, float *__restrict__ y) {
  __shared__ __nv_bfloat16 sW[WB_N];
  __shared__ float sB[NPAR];
  __shared__ float sNorm[2 * NI + NO];
  load_params(wb, master, norm, sW, sB, sNorm);
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int r0 = 16 * warp; r0 < n; r0 += 16 * nwarps) {
    fwd_out f;
    mlp_forward16(x, n, r0, sW, sB, sNorm, lane, f);
    const int g = lane >> 2, t = lane & 3;
    const int c0 = 2 * t, c1 = 2 * t + 1;
    if (r0 + g < n) {
      if (c0 < NO) y[(size_t)(r0 + g) * NO + c0] = f.y[0];
      if (c1 < NO) y[(size_t)(r0 + g) * NO + c1] = f.y[1];
    }
    if (r0 + g + 8 < n) {
      if (c0 < NO) y[(size_t)(r0 + g + 8) * NO + c0] = f.y[2];
      if (c1 < NO) y[(size_t)(r0 + g + 8) * NO + c1] = f.y[3];
    }
  }
}

// forward that keeps Z1, H1 = bf16(GELU(Z1)), Z2 and H2 (forward_trace)
__global__ void __launch_bounds__(256) k_mlp_trace(int n, const float *__restrict__ x, const __nv_bfloat16 *wb,
                                                   const float *master, const float *norm, float *__restrict__ z1,
                                                   float *__restrict__ h1, float *__restrict__ z2,
                                                   float *__restrict__ h2) {
  __shared__ __nv_bfloat16 sW[WB_N];
  __shared__ float sB[NPAR];
  __shared__ float sNorm[2 * NI + NO];
  load_params(wb, master, norm, sW, sB, sNorm);
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int r0 = 16 * warp;
  if (r0 >= n) return;
  fwd_out f;
  mlp_forward16(x, n, r0, sW, sB, sNorm, lane, f);
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int j = 0; j < 8; j++)
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int r = r0 + g + (e >= 2 ? 8 : 0), c = 8 * j + 2 * t + (e & 1);
      if (r < n) {
        z1[(size_t)r * NH + c] = f.z1[j][e];
        h1[(size_t)r * NH + c] = bf16r(gelu(f.z1[j][e]));
        z2[(size_t)r * NH + c] = f.z2[j][e];
        h2[(size_t)r * NH + c] = bf16r(gelu(f.z2[j][e]));
      }
    }
}

// ---- gradient: forward, backward and weight gradients of 32 nodes per block -----
// Everything of the 32 nodes stays in shared memory; a block writes only its
// partial of every weight and bias gradient,
//   dW1 = dZ1^T Xn, db1 = sum dZ1, dW2 = dZ2^T H1, db2 = sum dZ2,
//   dW3 = dY^T H2, db3 = sum dY
// (Xn the bf16-rounded normalised inputs), and of the loss.  The backward is
// dZ2 = (dY W3) * gelu'(Z2), dZ1 = (dZ2 W2) * gelu'(Z1) with W the bf16 values,
// FP32 throughout; the partials of NODES nodes, of CHUNK nodes and of all are
// added in this order (k_mlp_reduce), so a gradient is identical run to run.
//
// What bounds it: at a training batch (4096 nodes, 128 blocks, one wave) the
// chain of a block's phases.  As four kernels with the activations in global
// memory, the weight gradients by one block per 1024 nodes (4 blocks, 262 us) and
// the backward by one thread per node (32 blocks, 131 us), the batch took 424 us
// on the device (437 us a call with its host copies); now 22 us and 7 us (91 us a
// call, bound by the copies of the 295 KB batch from pageable memory).
constexpr int NODES = 32;
constexpr int CHUNK = 1024;  // nodes whose partials are added first
constexpr int LDH = NH + 4;  // padded row of a node's hidden values

struct grad_smem {
  __nv_bfloat16 W[WB_N];
  float W2[NH * NH];  // the bf16 values
  float W3[NO * NH];
  float B1[NH], B2[NH], B3[NO + 1];
  float x[NODES][16];                    // normalised, rounded to bf16; column 15 zero
  float z1[NODES][LDH], z2[NODES][LDH];  // pre-activations, later dZ1 and dZ2
  float h1[NODES][LDH], h2[NODES][LDH];  // bf16 values
  float dy[NODES][4];
};

// A fragment of 16 rows, columns 16 kk ..: bf16 values held as floats
template <int LD>
__device__ __forceinline__ void afrag(const float (*H)[LD], int r0, int kk, int lane, uint32_t a[4]) {
  const int g = lane >> 2, t = lane & 3, c = 16 * kk + 2 * t;
  a[0] = pack_bf16(H[r0 + g][c], H[r0 + g][c + 1]);
  a[1] = pack_bf16(H[r0 + g + 8][c], H[r0 + g + 8][c + 1]);
  a[2] = pack_bf16(H[r0 + g][c + 8], H[r0 + g][c + 9]);
  a[3] = pack_bf16(H[r0 + g + 8][c + 8], H[r0 + g + 8][c + 9]);
}

// tgt: the loss is the mean squared error against it; tgt == nullptr: dyin is
// dL/d(output)
__global__ void __launch_bounds__(256) k_mlp_grad(int n, const float *__restrict__ x, const float *__restrict__ tgt,
                                                  const float *__restrict__ dyin, const __nv_bfloat16 *wb,
                                                  const float *master, const float *norm, float *__restrict__ part,
                                                  float *__restrict__ loss_part) {
  extern __shared__ __align__(16) unsigned char raw[];
  grad_smem &S = *reinterpret_cast<grad_smem *>(raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b0 = blockIdx.x * NODES;
  for (int i = tid; i < WB_N / 2; i += 256) reinterpret_cast<uint32_t *>(S.W)[i] = reinterpret_cast<const uint32_t *>(wb)[i];
  for (int i = tid; i < NH * NH; i += 256) S.W2[i] = __bfloat162float(wb[WB_W2 + i]);
  for (int i = tid; i < NO * NH; i += 256) S.W3[i] = __bfloat162float(wb[WB_W3 + i]);
  if (tid < NH) {
    S.B1[tid] = master[OFF_B1 + tid];
    S.B2[tid] = master[OFF_B2 + tid];
  }
  if (tid < NO) S.B3[tid] = master[OFF_B3 + tid];
  for (int i = tid; i < NODES * 16; i += 256) {
    const int r = i / 16, c = i % 16;
    S.x[r][c] = b0 + r < n && c < NI ? bf16r((x[(size_t)(b0 + r) * NI + c] - norm[c]) * norm[NI + c]) : 0.f;
  }
  __syncthreads();
  // layers 1 and 2: warp w computes the hidden units 8 w .. 8 w + 7 of all nodes
  const int g = lane >> 2, t = lane & 3, c0 = 8 * warp + 2 * t;
#pragma unroll
  for (int layer = 1; layer <= 2; layer++) {
    float (*Z)[LDH] = layer == 1 ? S.z1 : S.z2, (*H)[LDH] = layer == 1 ? S.h1 : S.h2;
    const float bb0 = layer == 1 ? S.B1[c0] : S.B2[c0], bb1 = layer == 1 ? S.B1[c0 + 1] : S.B2[c0 + 1];
#pragma unroll
    for (int r0 = 0; r0 < NODES; r0 += 16) {
      float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int kk = 0; kk < (layer == 1 ? 1 : 4); kk++) {
        uint32_t a[4], b[2];
        if (layer == 1) {
          afrag(S.x, r0, 0, lane, a);
          bfrag(S.W + WB_W1, 16, warp, 0, lane, b);
        } else {
          afrag(S.h1, r0, kk, lane, a);
          bfrag(S.W + WB_W2, NH, warp, kk, lane, b);
        }
        mma_bf16(z, a, b);
      }
      z[0] += bb0; z[1] += bb1; z[2] += bb0; z[3] += bb1;
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int r = r0 + g + (e >= 2 ? 8 : 0), c = c0 + (e & 1);
        const bool ok = b0 + r < n;
        Z[r][c] = z[e];
        H[r][c] = ok ? bf16r(gelu(z[e])) : 0.f;
      }
    }
    __syncthreads();
  }
  // layer 3, its error and loss: one warp per 16 nodes
  if (warp < NODES / 16) {
    const int r0 = 16 * warp;
    float l = 0.f;
    if (tgt != nullptr) {
      float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int kk = 0; kk < 4; kk++) {
        uint32_t a[4], b[2];
        afrag(S.h2, r0, kk, lane, a);
        bfrag(S.W + WB_W3, NH, 0, kk, lane, b);
        mma_bf16(y, a, b);
      }
      const float inv = 2.0f / (float)(n * NO);
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int r = r0 + g + (e >= 2 ? 8 : 0), c = 2 * t + (e & 1);
        if (c >= NO) continue;
        float v = 0.f;
        if (b0 + r < n) {
          const float d = (y[e] + S.B3[c]) - tgt[(size_t)(b0 + r) * NO + c];
          v = inv * d;
          l += d * d;
        }
        S.dy[r][c] = v;
      }
    } else {
      for (int i = lane; i < 16 * NO; i += 32) {
        const int r = r0 + i / NO, c = i % NO;
        S.dy[r][c] = b0 + r < n ? dyin[(size_t)(b0 + r) * NO + c] : 0.f;
      }
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
    if (lane == 0) loss_part[(NODES / 16) * blockIdx.x + warp] = l;
  }
  __syncthreads();
  // dZ2 in place of Z2
  for (int i = tid; i < NODES * NH; i += 256) {
    const int r = i / NH, j = i % NH;
    const float dh = S.dy[r][0] * S.W3[j] + S.dy[r][1] * S.W3[NH + j] + S.dy[r][2] * S.W3[2 * NH + j];
    S.z2[r][j] = b0 + r < n ? dh * gelu_d(S.z2[r][j]) : 0.f;
  }
  __syncthreads();
  // dZ1 in place of Z1: eight units of one node per thread
  {
    const int r = tid / 8, i0 = 8 * (tid % 8);
    float dh[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int j = 0; j < NH; j++) {
      const float d = S.z2[r][j];
      const float4 wa = *reinterpret_cast<const float4 *>(S.W2 + NH * j + i0);
      const float4 wc = *reinterpret_cast<const float4 *>(S.W2 + NH * j + i0 + 4);
      dh[0] += d * wa.x; dh[1] += d * wa.y; dh[2] += d * wa.z; dh[3] += d * wa.w;
      dh[4] += d * wc.x; dh[5] += d * wc.y; dh[6] += d * wc.z; dh[7] += d * wc.w;
    }
#pragma unroll
    for (int k = 0; k < 8; k++) S.z1[r][i0 + k] = b0 + r < n ? dh[k] * gelu_d(S.z1[r][i0 + k]) : 0.f;
  }
  __syncthreads();
  // the partials: a 4 x 4 tile of dW2 per thread, four inputs of a unit of dW1,
  // then dW3 and the biases
  float *P = part + (size_t)blockIdx.x * NPAR;
  {
    const int o0 = 4 * (tid / 16), i0 = 4 * (tid % 16);
    float a[4][4], bs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int p = 0; p < 4; p++)
#pragma unroll
      for (int q = 0; q < 4; q++) a[p][q] = 0.f;
#pragma unroll 4
    for (int r = 0; r < NODES; r++) {
      const float4 d = *reinterpret_cast<const float4 *>(&S.z2[r][o0]), h = *reinterpret_cast<const float4 *>(&S.h1[r][i0]);
      const float dv[4] = {d.x, d.y, d.z, d.w}, hv[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
      for (int p = 0; p < 4; p++) {
        bs[p] += dv[p];
#pragma unroll
        for (int q = 0; q < 4; q++) a[p][q] += dv[p] * hv[q];
      }
    }
#pragma unroll
    for (int p = 0; p < 4; p++) {
#pragma unroll
      for (int q = 0; q < 4; q++) P[OFF_W2 + NH * (o0 + p) + i0 + q] = a[p][q];
      if (i0 == 0) P[OFF_B2 + o0 + p] = bs[p];
    }
  }
  {
    const int o = tid / 4, i0 = 4 * (tid % 4);
    float a[4] = {0.f, 0.f, 0.f, 0.f}, bs = 0.f;
#pragma unroll 4
    for (int r = 0; r < NODES; r++) {
      const float d = S.z1[r][o];
      const float4 v = *reinterpret_cast<const float4 *>(&S.x[r][i0]);
      a[0] += d * v.x; a[1] += d * v.y; a[2] += d * v.z; a[3] += d * v.w;
      bs += d;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (i0 + k < NI) P[OFF_W1 + NI * o + i0 + k] = a[k];
    if (i0 == 0) P[OFF_B1 + o] = bs;
  }
  if (tid < NO * NH) {
    const int o = tid / NH, i = tid % NH;
    float a = 0.f;
    for (int r = 0; r < NODES; r++) a += S.dy[r][o] * S.h2[r][i];
    P[OFF_W3 + tid] = a;
  } else if (tid < NO * NH + NO) {
    float a = 0.f;
    for (int r = 0; r < NODES; r++) a += S.dy[r][tid - NO * NH];
    P[OFF_B3 + tid - NO * NH] = a;
  }
}

// grad[p]: the partials of every CHUNK nodes in order, then the chunks in order
// (32 parameters per block, eight chunks side by side); loss = sum of its
// partials in order / (n NO)
__global__ void __launch_bounds__(256) k_mlp_reduce(int nparts, const float *__restrict__ part, float *__restrict__ grad,
                                                    int nloss, const float *__restrict__ loss_part, float *loss, int n) {
  constexpr int PER = CHUNK / NODES;
  __shared__ float sh[8][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, p = 32 * blockIdx.x + tx;
  const int nch = (nparts + PER - 1) / PER;
  float s = 0.f;
  for (int c0 = 0; c0 < nch; c0 += 8) {
    float a = 0.f;
    if (p < NPAR) {
      const int q0 = (c0 + ty) * PER, q1 = min(nparts, q0 + PER);
#pragma unroll 8
      for (int q = q0; q < q1; q++) a += part[(size_t)q * NPAR + p];
    }
    sh[ty][tx] = a;
    __syncthreads();
    if (ty == 0)
      for (int k = 0; k < 8 && c0 + k < nch; k++) s += sh[k][tx];
    __syncthreads();
  }
  if (ty == 0 && p < NPAR) grad[p] = s;
  if (blockIdx.x == 0 && loss) {
    __shared__ float sl[256];
    float l = 0.f;
    for (int i0 = 0; i0 < nloss; i0 += 256) {
      sl[threadIdx.x] = i0 + (int)threadIdx.x < nloss ? loss_part[i0 + threadIdx.x] : 0.f;
      __syncthreads();
      if (threadIdx.x == 0)
        for (int i = 0; i < min(256, nloss - i0); i++) l += sl[i];
      __syncthreads();
    }
    if (threadIdx.x == 0) *loss = l / (float)(n * NO);
  }
}

// bf16 copies of the weights in the padded layout the forward reads
__global__ void k_mlp_pack(const float *__restrict__ master, __nv_bfloat16 *__restrict__ wb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= WB_N) return;
  float v = 0.f;
  if (i < WB_W2) {
    const int o = i / 16, k = i % 16;
    v = k < NI ? master[OFF_W1 + o * NI + k] : 0.f;
  } else if (i < WB_W3) {
    v = master[OFF_W2 + (i - WB_W2)];
  } else {
    const int o = (i - WB_W3) / NH, k = (i - WB_W3) % NH;
    v = o < NO ? master[OFF_W3 + o * NH + k] : 0.f;
  }
  wb[i] = __float2bfloat16_rn(v);
}

__global__ void k_mlp_adam(float *__restrict__ w, float *__restrict__ m, float *__restrict__ v,
                           const float *__restrict__ g, float lr, float b1c, float b2c) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= NPAR) return;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  m[p] = b1 * m[p] + (1.f - b1) * g[p];
  v[p] = b2 * v[p] + (1.f - b2) * g[p] * g[p];
  const float mh = m[p] / b1c, vh = v[p] / b2c;
  w[p] -= lr * mh / (sqrtf(vh) + eps);
}

__global__ void k_gather_rows(int k, const int *__restrict__ idx, const float *__restrict__ xa,
                              const float *__restrict__ ya, float *__restrict__ x, float *__restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k) return;
  const int r = idx[i];
  for (int c = 0; c < NI; c++) x[(size_t)i * NI + c] = xa[(size_t)r * NI + c];
  for (int c = 0; c < NO; c++) y[(size_t)i * NO + c] = ya[(size_t)r * NO + c];
}

int fail(icf_mlp *m, int code, const std::string &msg) {
  m->err = msg;
  return code;
}
#define MLP_CUDA(m, call)                                                                          \
  do {                                                                                             \
    cudaError_t e_ = (call);                                                                       \
    if (e_ != cudaSuccess) return fail((m), ICF_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// device arrays of at least n elements
int ensure(icf_mlp *m, float **p, long long *cap, long long n) {
  if (n <= *cap && *p) return ICF_OK;
  cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  MLP_CUDA(m, cudaMalloc(p, sizeof(float) * (size_t)n));
  *cap = n;
  return ICF_OK;
}

// the inputs and outputs of n nodes
int ensure_io(icf_mlp *m, long long n) {
  if (ensure(m, &m->d_x, &m->x_cap, NI * n) || ensure(m, &m->d_out, &m->out_cap, NO * n)) return ICF_ERR_CUDA;
  return ICF_OK;
}
// ... and their targets (or output gradients) and the gradient's partials
int ensure_grad(icf_mlp *m, long long n) {
  const long long nb = (n + NODES - 1) / NODES;
  if (ensure(m, &m->d_x, &m->x_cap, NI * n) || ensure(m, &m->d_y, &m->y_cap, NO * n) ||
      ensure(m, &m->d_part, &m->part_cap, NPAR * nb) || ensure(m, &m->d_loss, &m->loss_cap, 1 + (NODES / 16) * nb))
    return ICF_ERR_CUDA;
  return ICF_OK;
}

// gradient of the data already in d_x, d_y (n nodes): d_grad, loss.
// dy_given: d_y holds dL/dy (the caller's loss) instead of targets.
int grad_on_device(icf_mlp *m, int n, float *loss_host, bool dy_given = false) {
  cudaStream_t s = m->stream;
  const int nb = (n + NODES - 1) / NODES;
  float *loss_part = m->d_loss + 1;
  MLP_CUDA(m, cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(grad_smem)));
  k_mlp_grad<<<nb, 256, sizeof(grad_smem), s>>>(n, m->d_x, dy_given ? nullptr : m->d_y, m->d_y, m->d_wb, m->d_master,
                                               m->d_norm, m->d_part, loss_part);
  k_mlp_reduce<<<icf_blocks(NPAR, 32), 256, 0, s>>>(nb, m->d_part, m->d_grad, (NODES / 16) * nb, loss_part, m->d_loss,
                                                   n);
  MLP_CUDA(m, cudaGetLastError());
  if (loss_host) {
    MLP_CUDA(m, cudaMemcpyAsync(loss_host, m->d_loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    MLP_CUDA(m, cudaStreamSynchronize(s));
  }
  return ICF_OK;
}

}  // namespace

extern "C" {

int icf_mlp_create(int device, icf_mlp **out) {
  if (!out) return ICF_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return ICF_ERR_NODEVICE;
  if (device < 0 || device >= ndev) return ICF_ERR_ARG;
  icf_mlp *m = new icf_mlp();
  m->device = device;
  if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) ||
      cudaMalloc(&m->d_master, sizeof(float) * NPAR) || cudaMalloc(&m->d_m, sizeof(float) * NPAR) ||
      cudaMalloc(&m->d_v, sizeof(float) * NPAR) || cudaMalloc(&m->d_grad, sizeof(float) * NPAR) ||
      cudaMalloc(&m->d_wb, sizeof(__nv_bfloat16) * WB_N) || cudaMalloc(&m->d_norm, sizeof(float) * (2 * NI + NO))) {
    delete m;
    return ICF_ERR_CUDA;
  }
  std::vector<float> norm(2 * NI + NO, 0.f);
  for (int i = 0; i < NI; i++) norm[NI + i] = 1.f;
  for (int i = 0; i < NO; i++) norm[2 * NI + i] = 1.f;
  // (copies and fills on the network's stream, here and below: the null stream
  // is not ordered with it)
  cudaStream_t s = m->stream;
  icf_h2d(s, m->d_norm, norm.data(), sizeof(float) * norm.size());
  cudaMemsetAsync(m->d_master, 0, sizeof(float) * NPAR, s);
  cudaMemsetAsync(m->d_m, 0, sizeof(float) * NPAR, s);
  cudaMemsetAsync(m->d_v, 0, sizeof(float) * NPAR, s);
  k_mlp_pack<<<icf_blocks(WB_N, 256), 256, 0, s>>>(m->d_master, m->d_wb);
  if (cudaStreamSynchronize(s) != cudaSuccess) {
    delete m;
    return ICF_ERR_CUDA;
  }
  *out = m;
  return ICF_OK;
}

int icf_mlp_destroy(icf_mlp *m) {
  if (!m) return ICF_ERR_ARG;
  cudaSetDevice(m->device);
  void *p[] = {m->d_master, m->d_m, m->d_v, m->d_wb, m->d_norm, m->d_x, m->d_y, m->d_z1, m->d_h1, m->d_z2,
               m->d_h2, m->d_out, m->d_part, m->d_grad, m->d_loss};
  for (void *q : p) cudaFree(q);
  if (m->stream) cudaStreamDestroy(m->stream);
  delete m;
  return ICF_OK;
}

const char *icf_mlp_last_error(const icf_mlp *m) { return m ? m->err.c_str() : "null network"; }
int icf_mlp_param_count(void) { return NPAR; }

int icf_mlp_set_params(icf_mlp *m, const float *params, const float *norm) {
  if (!m || !params) return ICF_ERR_ARG;
  MLP_CUDA(m, cudaSetDevice(m->device));
  cudaStream_t s = m->stream;
  MLP_CUDA(m, icf_h2d(s, m->d_master, params, sizeof(float) * NPAR));
  if (norm) MLP_CUDA(m, icf_h2d(s, m->d_norm, norm, sizeof(float) * (2 * NI + NO)));
  MLP_CUDA(m, cudaMemsetAsync(m->d_m, 0, sizeof(float) * NPAR, s));
  MLP_CUDA(m, cudaMemsetAsync(m->d_v, 0, sizeof(float) * NPAR, s));
  m->adam_t = 0;
  k_mlp_pack<<<icf_blocks(WB_N, 256), 256, 0, s>>>(m->d_master, m->d_wb);
  MLP_CUDA(m, cudaStreamSynchronize(s));
  return ICF_OK;
}

int icf_mlp_get_params(icf_mlp *m, float *params, float *norm) {
  if (!m || !params) return ICF_ERR_ARG;
  MLP_CUDA(m, cudaSetDevice(m->device));
  MLP_CUDA(m, cudaStreamSynchronize(m->stream));
  MLP_CUDA(m, cudaMemcpy(params, m->d_master, sizeof(float) * NPAR, cudaMemcpyDeviceToHost));
  if (norm) MLP_CUDA(m, cudaMemcpy(norm, m->d_norm, sizeof(float) * (2 * NI + NO), cudaMemcpyDeviceToHost));
  return ICF_OK;
}

int icf_mlp_forward(icf_mlp *m, int n, const float *x, float *y) {
  if (!m || n < 0 || (n && (!x || !y))) return ICF_ERR_ARG;
  if (n == 0) return ICF_OK;
  MLP_CUDA(m, cudaSetDevice(m->device));
  if (ensure_io(m, n)) return ICF_ERR_CUDA;
  cudaStream_t s = m->stream;
  MLP_CUDA(m, cudaMemcpyAsync(m->d_x, x, sizeof(float) * NI * (size_t)n, cudaMemcpyHostToDevice, s));
  const int tiles = (n + 15) / 16;
  int blocks = (tiles + 7) / 8;
  if (blocks > 1184) blocks = 1184;
  k_mlp_infer<<<blocks, 256, 0, s>>>(n, m->d_x, m->d_wb, m->d_master, m->d_norm, m->d_out);
  MLP_CUDA(m, cudaGetLastError());
  MLP_CUDA(m, cudaMemcpyAsync(y, m->d_out, sizeof(float) * NO * (size_t)n, cudaMemcpyDeviceToHost, s));
  MLP_CUDA(m, cudaStreamSynchronize(s));
  return ICF_OK;
}

int icf_mlp_forward_trace(icf_mlp *m, int n, const float *x, float *z1, float *h1, float *z2, float *h2, float *y) {
  if (!m || n <= 0 || !x || !z1 || !h1 || !z2 || !h2 || !y) return ICF_ERR_ARG;
  MLP_CUDA(m, cudaSetDevice(m->device));
  const long long nz = (long long)NH * n;
  if (ensure_io(m, n) || ensure(m, &m->d_z1, &m->z1_cap, nz) || ensure(m, &m->d_h1, &m->h1_cap, nz) ||
      ensure(m, &m->d_z2, &m->z2_cap, nz) || ensure(m, &m->d_h2, &m->h2_cap, nz))
    return ICF_ERR_CUDA;
  cudaStream_t s = m->stream;
  MLP_CUDA(m, cudaMemcpyAsync(m->d_x, x, sizeof(float) * NI * (size_t)n, cudaMemcpyHostToDevice, s));
  const int tiles = (n + 15) / 16;
  k_mlp_trace<<<(tiles + 7) / 8, 256, 0, s>>>(n, m->d_x, m->d_wb, m->d_master, m->d_norm, m->d_z1, m->d_h1, m->d_z2,
                                              m->d_h2);
  int blocks = (tiles + 7) / 8;
  if (blocks > 1184) blocks = 1184;
  k_mlp_infer<<<blocks, 256, 0, s>>>(n, m->d_x, m->d_wb, m->d_master, m->d_norm, m->d_out);
  MLP_CUDA(m, cudaGetLastError());
  const size_t hb = sizeof(float) * NH * (size_t)n;
  MLP_CUDA(m, cudaMemcpyAsync(z1, m->d_z1, hb, cudaMemcpyDeviceToHost, s));
  MLP_CUDA(m, cudaMemcpyAsync(h1, m->d_h1, hb, cudaMemcpyDeviceToHost, s));
  MLP_CUDA(m, cudaMemcpyAsync(z2, m->d_z2, hb, cudaMemcpyDeviceToHost, s));
  MLP_CUDA(m, cudaMemcpyAsync(h2, m->d_h2, hb, cudaMemcpyDeviceToHost, s));
  MLP_CUDA(m, cudaMemcpyAsync(y, m->d_out, sizeof(float) * NO * (size_t)n, cudaMemcpyDeviceToHost, s));
  MLP_CUDA(m, cudaStreamSynchronize(s));
  return ICF_OK;
}

int icf_mlp_grad(icf_mlp *m, int n, const float *x, const float *y, float *grad, float *loss) {
  if (!m || n <= 0 || !x || !y || !grad) return ICF_ERR_ARG;
  MLP_CUDA(m, cudaSetDevice(m->device));
  if (ensure_grad(m, n)) return ICF_ERR_CUDA;
  cudaStream_t s = m->stream;
  MLP_CUDA(m, cudaMemcpyAsync(m->d_x, x, sizeof(float) * NI * (size_t)n, cudaMemcpyHostToDevice, s));
  MLP_CUDA(m, cudaMemcpyAsync(m->d_y, y, sizeof(float) * NO * (size_t)n, cudaMemcpyHostToDevice, s));
  if (grad_on_device(m, n, nullptr)) return ICF_ERR_CUDA;
  MLP_CUDA(m, cudaMemcpyAsync(grad, m->d_grad, sizeof(float) * NPAR, cudaMemcpyDeviceToHost, s));
  if (loss) MLP_CUDA(m, cudaMemcpyAsync(loss, m->d_loss, sizeof(float), cudaMemcpyDeviceToHost, s));
  MLP_CUDA(m, cudaStreamSynchronize(s));
  return ICF_OK;
}

int icf_mlp_grad_dy(icf_mlp *m, int n, const float *x, const float *dy, float *grad) {
  if (!m || n <= 0 || !x || !dy) return ICF_ERR_ARG;
  MLP_CUDA(m, cudaSetDevice(m->device));
  if (ensure_grad(m, n)) return ICF_ERR_CUDA;
  cudaStream_t s = m->stream;
  MLP_CUDA(m, cudaMemcpyAsync(m->d_x, x, sizeof(float) * NI * (size_t)n, cudaMemcpyHostToDevice, s));
  MLP_CUDA(m, cudaMemcpyAsync(m->d_y, dy, sizeof(float) * NO * (size_t)n, cudaMemcpyHostToDevice, s));
  if (grad_on_device(m, n, nullptr, true)) return ICF_ERR_CUDA;
  if (grad) MLP_CUDA(m, cudaMemcpyAsync(grad, m->d_grad, sizeof(float) * NPAR, cudaMemcpyDeviceToHost, s));
  MLP_CUDA(m, cudaStreamSynchronize(s));
  return ICF_OK;
}

int icf_mlp_adam_step(icf_mlp *m, const float *grad, float lr) {
  if (!m || !(lr > 0)) return ICF_ERR_ARG;
  MLP_CUDA(m, cudaSetDevice(m->device));
  cudaStream_t s = m->stream;
  if (grad) MLP_CUDA(m, cudaMemcpyAsync(m->d_grad, grad, sizeof(float) * NPAR, cudaMemcpyHostToDevice, s));
  m->adam_t++;
  const float b1c = 1.f - powf(0.9f, (float)m->adam_t), b2c = 1.f - powf(0.999f, (float)m->adam_t);
  k_mlp_adam<<<icf_blocks(NPAR, 256), 256, 0, s>>>(m->d_master, m->d_m, m->d_v, m->d_grad, lr, b1c, b2c);
  k_mlp_pack<<<icf_blocks(WB_N, 256), 256, 0, s>>>(m->d_master, m->d_wb);
  MLP_CUDA(m, cudaGetLastError());
  MLP_CUDA(m, cudaStreamSynchronize(s));
  return ICF_OK;
}

int icf_mlp_train(icf_mlp *m, int n, const float *x, const float *y, int epochs, int batch, float lr,
                  unsigned long long seed, float *loss_out) {
  if (!m || n <= 0 || !x || !y || epochs < 1 || batch < 16 || !(lr > 0)) return ICF_ERR_ARG;
  MLP_CUDA(m, cudaSetDevice(m->device));
  if (batch > n) batch = n;
  if (ensure_grad(m, batch)) return ICF_ERR_CUDA;
  cudaStream_t s = m->stream;
  // whole data set on the device, shuffled per epoch on the host (seeded)
  float *dx_all = nullptr, *dy_all = nullptr;
  int *d_order = nullptr;
  MLP_CUDA(m, cudaMalloc(&dx_all, sizeof(float) * NI * (size_t)n));
  MLP_CUDA(m, cudaMalloc(&dy_all, sizeof(float) * NO * (size_t)n));
  MLP_CUDA(m, cudaMalloc(&d_order, sizeof(int) * (size_t)n));
  MLP_CUDA(m, icf_h2d(s, dx_all, x, sizeof(float) * NI * (size_t)n));
  MLP_CUDA(m, icf_h2d(s, dy_all, y, sizeof(float) * NO * (size_t)n));
  std::vector<int> order(n);
  for (int i = 0; i < n; i++) order[i] = i;
  unsigned long long st = seed * 6364136223846793005ull + 1442695040888963407ull;
  float last = 0.f;
  int rc = ICF_OK;
  for (int ep = 0; ep < epochs && rc == ICF_OK; ep++) {
    for (int i = n - 1; i > 0; i--) {  // Fisher-Yates with a 64-bit LCG
      st = st * 6364136223846793005ull + 1442695040888963407ull;
      const int j = (int)((st >> 33) % (unsigned long long)(i + 1));
      std::swap(order[i], order[j]);
    }
    if (cudaMemcpyAsync(d_order, order.data(), sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, s) !=
        cudaSuccess) {
      rc = fail(m, ICF_ERR_CUDA, "order upload failed");
      break;
    }
    // contiguous batches of the shuffled order, gathered on the device
    for (int b0 = 0; b0 + batch <= n && rc == ICF_OK; b0 += batch) {
      k_gather_rows<<<icf_blocks(batch, 256), 256, 0, s>>>(batch, d_order + b0, dx_all, dy_all, m->d_x, m->d_y);
      rc = grad_on_device(m, batch, nullptr);
      if (rc) break;
      m->adam_t++;
      const float b1c = 1.f - powf(0.9f, (float)m->adam_t), b2c = 1.f - powf(0.999f, (float)m->adam_t);
      k_mlp_adam<<<icf_blocks(NPAR, 256), 256, 0, s>>>(m->d_master, m->d_m, m->d_v, m->d_grad, lr, b1c, b2c);
      k_mlp_pack<<<icf_blocks(WB_N, 256), 256, 0, s>>>(m->d_master, m->d_wb);
    }
    if (rc == ICF_OK && cudaGetLastError() != cudaSuccess) rc = fail(m, ICF_ERR_CUDA, "training launch failed");
  }
  if (rc == ICF_OK) {
    // loss over the whole set with the final weights (a batch's nodes per pass)
    double tot = 0;
    for (int b0 = 0; b0 < n && rc == ICF_OK; b0 += batch) {
      const int k = std::min(batch, n - b0);
      cudaMemcpyAsync(m->d_x, dx_all + (size_t)b0 * NI, sizeof(float) * NI * (size_t)k, cudaMemcpyDeviceToDevice, s);
      cudaMemcpyAsync(m->d_y, dy_all + (size_t)b0 * NO, sizeof(float) * NO * (size_t)k, cudaMemcpyDeviceToDevice, s);
      float l = 0;
      rc = grad_on_device(m, k, &l);
      tot += (double)l * k;
    }
    last = (float)(tot / n);
  }
  cudaStreamSynchronize(s);  // the host order buffer is reused by the next epoch's upload only after this
  cudaFree(dx_all);
  cudaFree(dy_all);
  cudaFree(d_order);
  if (rc) return rc;
  if (loss_out) *loss_out = last;
  return ICF_OK;
}

}  // extern "C"
