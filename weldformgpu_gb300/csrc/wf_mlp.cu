// wf_mlp.cu — the learned warm start of the Johnson-Cook return map:
// synthetic (state, converged increment) pairs, FP32 training kernels
// (forward, backward, Adam), BF16 tcgen05 tensor-core inference, and a kernel that
// counts Newton iterations with and without the network.
//
// No counterpart in the reference: its return map is a one-shot radial
// return (src/cuda/Mechanical.cu:503-536) with no iterative solve.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/weldform_gb300.h"
#include "wf_common.cuh"
#include "wf_mlp.cuh"
#include "wf_tensor.cuh"

namespace {

// ---- parameter packing for the tensor-core kernels ---------------------------
// The tcgen05 weight image (mlp_umma_cta): B2 = W2 in BF16, K-major core-
// matrix order, then b2, W3 and b3 in FP32 (layer 1 travels as MlpL1).
__global__ void k_mlp_pack_umma(const float* __restrict__ P, uint8_t* __restrict__ out) {
  const float* W2 = P + WF_MLP_OFF_W2;
  for (int k = threadIdx.x; k < WF_UMMA_IMAGE / 4; k += blockDim.x)
    reinterpret_cast<uint32_t*>(out)[k] = 0u;
  __syncthreads();
  for (int e = threadIdx.x; e < WF_MLP_H * WF_MLP_H; e += blockDim.x) {
    const int n = e / WF_MLP_H, k = e % WF_MLP_H;
    *reinterpret_cast<__nv_bfloat16*>(out + WF_UMMA_B2 + umma_kmajor_off(n, k, WF_MLP_H)) =
        __float2bfloat16_rn(W2[n * WF_MLP_H + k]);
  }
  for (int k = threadIdx.x; k < WF_MLP_H; k += blockDim.x) {
    reinterpret_cast<float*>(out + WF_UMMA_BIAS2)[k] = P[WF_MLP_OFF_B2 + k];
    reinterpret_cast<float*>(out + WF_UMMA_W3)[k] = P[WF_MLP_OFF_W3 + k];
  }
  if (threadIdx.x == 0) *reinterpret_cast<float*>(out + WF_UMMA_B3) = P[WF_MLP_OFF_B3];
}

// ---- standalone inference ---------------------------------------------------
__global__ void __launch_bounds__(128) k_mlp_infer_umma(const uint4* __restrict__ image,
                                                        const MlpL1 l1,
                                                        const float4* __restrict__ X, int64_t n,
                                                        float* __restrict__ Y, int* status) {
  extern __shared__ __align__(1024) uint8_t smu[];
  mlp_umma_begin(smu, image);
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool valid = i < n;
  float f[4] = {0.f, 0.f, 0.f, 0.f};
  if (valid) {
    const float4 x = X[i];
    f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w;
  }
  const float y = mlp_umma_cta(smu, image, f, valid, status, l1);
  if (valid) Y[i] = y;
}

__global__ void k_mlp_infer_f32(const float* __restrict__ P, const float4* __restrict__ X,
                                int64_t n, float* __restrict__ Y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 x = X[i];
  const float f[4] = {x.x, x.y, x.z, x.w};
  float h1[WF_MLP_H];
  for (int o = 0; o < WF_MLP_H; o++) {
    float z = P[WF_MLP_OFF_B1 + o];
    for (int k = 0; k < 4; k++) z += P[WF_MLP_OFF_W1 + o * 4 + k] * f[k];
    h1[o] = mlp_silu(z);
  }
  float y = P[WF_MLP_OFF_B3];
  for (int o = 0; o < WF_MLP_H; o++) {
    float z = P[WF_MLP_OFF_B2 + o];
    for (int k = 0; k < WF_MLP_H; k++) z += P[WF_MLP_OFF_W2 + o * WF_MLP_H + k] * h1[k];
    y += P[WF_MLP_OFF_W3 + o] * mlp_silu(z);
  }
  Y[i] = y;
}

// ---- synthetic states with converged FP64 targets ------------------------------
__device__ __forceinline__ uint64_t sm64(uint64_t x) {
  uint64_t z = x + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ double u01d(uint64_t x) { return (double)(sm64(x) >> 11) * (1.0 / 9007199254740992.0); }

struct JcState {
  double ratio, eps_p, rate, T;
};

// rate x thermal factor of the JC law (the rate clamp of Material.cuh:277-279)
__device__ __forceinline__ double jc_rt(const MatParams& M, double rate, double T, double* Th_out) {
  double Th = (T - M.Tt) / (M.Tm - M.Tt);
  Th = Th < 0.0 ? 0.0 : (Th > 0.999 ? 0.999 : Th);
  *Th_out = Th;
  const double sr = rate == 0.0 ? 1.e-5 : rate;
  return (1.0 + M.C * log(sr / M.eps0)) * (1.0 - pow(Th, M.m));
}

// ratio U[1,3], eps_p log-U[1e-4,2], rate log-U[1e-2,1e5] /s, T U[20,550] C
__global__ void k_mlp_synth(StepParams P, double G, int64_t n, uint64_t seed, float4* __restrict__ X,
                            float* __restrict__ Y, float4* __restrict__ S, int32_t* __restrict__ iters) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t base = seed * 0x100000001B3ull + (uint64_t)i * 4ull;
  JcState s;
  s.ratio = 1.0 + 2.0 * u01d(base);
  s.eps_p = 1.0e-4 * pow(2.0e4, u01d(base + 1));
  s.rate = 1.0e-2 * pow(1.0e7, u01d(base + 2));
  s.T = 20.0 + 530.0 * u01d(base + 3);
  double Th;
  const double RT = jc_rt(P.mat, s.rate, s.T, &Th);
  double pwn = pow(s.eps_p, P.mat.n);
  const double sy0 = (P.mat.A + P.mat.B * pwn) * RT;
  const double st = s.ratio * sy0;
  double dl, sy1;
  int it = 0;
  jc_return_cached(P, st, 3.0 * G, s.eps_p, pwn, RT, -1.0, &dl, &sy1, &it);
  const double hi = (st - sy0) / (3.0 * G);
  float f[4];
  mlp_features((float)s.ratio, s.eps_p, (float)s.rate, (float)Th, f);
  X[i] = make_float4(f[0], f[1], f[2], f[3]);
  Y[i] = (float)(dl / hi);
  S[i] = make_float4((float)s.ratio, (float)s.eps_p, (float)s.rate, (float)s.T);
  iters[i] = it;
}

// Newton iterations from the radial start (image == nullptr) or the network's start
__global__ void __launch_bounds__(128) k_mlp_newton_iters(StepParams P, double G,
                                                          const uint4* __restrict__ image,
                                                          const MlpL1 l1,
                                                          const float4* __restrict__ S, int64_t n,
                                                          int32_t* __restrict__ iters,
                                                          int32_t* __restrict__ used,
                                                          float* __restrict__ dl_out, int* status) {
  extern __shared__ __align__(1024) uint8_t smu[];
  mlp_umma_begin(smu, image);
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool valid = i < n;
  const float4 s = valid ? S[i] : make_float4(1.f, 1e-2f, 1.f, 20.f);
  double Th;
  const double RT = jc_rt(P.mat, (double)s.z, (double)s.w, &Th);
  double pwn = pow((double)s.y, P.mat.n);
  const double sy0 = (P.mat.A + P.mat.B * pwn) * RT;
  const double st = (double)s.x * sy0;
  double ratio = -1.0;
  int use = 0;
  if (image) {
    float f[4];
    mlp_features(s.x, (double)s.y, s.z, (float)Th, f);
    const float y = mlp_umma_cta(smu, image, f, valid, status, l1);
    const float yc = mlp_accept(y);
    if (yc > 0.0f) { ratio = (double)yc; use = 1; }
  }
  if (!valid) return;
  double dl, sy1;
  int it = 0;
  jc_return_cached(P, st, 3.0 * G, (double)s.y, pwn, RT, ratio, &dl, &sy1, &it);
  iters[i] = it;
  used[i] = use;
  dl_out[i] = (float)dl;
}

// ---- training: loss and gradient of the mean squared error -------------------
// FP32 throughout.  A block of 512 threads takes tiles of 32 samples (a batch
// of 4,096 is 128 blocks, nearly one per SM; larger sets loop) and keeps its
// weight gradients in registers over its tiles: thread (ts, to) holds one
// sample by four units in the products with W2 and a 2 x 4 block of W2's
// gradient, operands read from shared memory as float4 without bank conflicts.
// Each block writes its sums to its own row of `part`; the rows are added in a
// fixed order by the kernel that uses them (k_adam, k_grad_total), so a run
// gives the same bits every time.  What bounds a training step at this size is
// the latency of its two kernels, not arithmetic (0.1 GFLOP) or memory.  The
// kernel before this one took a sample per thread and walked 64 x 64 products
// serially on 32 blocks: 372 -> 16 us per 4,096 samples (a step with Adam 382
// -> 21 us; 256 threads per block: 17 us; as k_mlp_train 16.5).
constexpr int kTile = 32;              // samples per tile
constexpr int kGradThreads = 512;
constexpr int kGradBlocks = 304;       // most blocks (rows of partial sums): 2 per SM
constexpr int LDA = WF_MLP_H + 4;      // row stride of the tile arrays (16-byte aligned rows)
constexpr int kPartRow = (WF_MLP_NPARAM + 1 + 31) / 32 * 32;   // gradient, then the loss

struct GradShared {
  float W2[WF_MLP_H * LDA];            // [o][k]
  float W1[WF_MLP_H * 4], b1[WF_MLP_H], b2[WF_MLP_H], w3[WF_MLP_H];
  float H1[kTile * LDA], D1[kTile * LDA], G2[kTile * LDA];
  float4 X[kTile];
};

__device__ __forceinline__ void fma4(float4& acc, float a, const float4& b) {
  acc.x += a * b.x; acc.y += a * b.y; acc.z += a * b.z; acc.w += a * b.w;
}
__device__ __forceinline__ float dot4(float acc, const float4& a, const float4& b) {
  acc += a.x * b.x; acc += a.y * b.y; acc += a.z * b.z; acc += a.w * b.w;
  return acc;
}

// The block's sums over its tiles into its row of partial sums.  The parameters
// are read from L2: inside k_mlp_train other blocks have just written them.
__device__ __forceinline__ void grad_block(unsigned char* smem_raw, const float* P,
                                           const float4* __restrict__ X,
                                           const float* __restrict__ Yt, int64_t offset,
                                           int64_t count, float inv_total, int rows, float* row) {
  GradShared& S = *reinterpret_cast<GradShared*>(smem_raw);
  const int t = threadIdx.x;
  const int ts = t >> 4, to = t & 15;          // sample ts; 16 threads share it
  const int64_t tiles = (count + kTile - 1) / kTile;
  // the first tile's samples are on their way while the weights are loaded
  float4 x_next = make_float4(0.f, 0.f, 0.f, 0.f);
  float target_next = 0.0f;
  const auto fetch = [&](int64_t tile) {
    const int64_t gi = tile * kTile + ts;
    const bool v = tile < tiles && gi < count;
    x_next = v ? X[offset + gi] : make_float4(0.f, 0.f, 0.f, 0.f);
    target_next = v ? Yt[offset + gi] : 0.0f;
  };
  fetch(blockIdx.x);
  static_assert(WF_MLP_OFF_W2 % 4 == 0 && WF_MLP_H * WF_MLP_H == 8 * kGradThreads, "16-byte loads");
  float4 wv[2];
#pragma unroll
  for (int q = 0; q < 2; q++)
    wv[q] = __ldcg(reinterpret_cast<const float4*>(P + WF_MLP_OFF_W2) + t + q * kGradThreads);
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int k = 4 * (t + q * kGradThreads);
    *reinterpret_cast<float4*>(S.W2 + (k / WF_MLP_H) * LDA + k % WF_MLP_H) = wv[q];
  }
  if (t < 4 * WF_MLP_H) S.W1[t] = __ldcg(P + WF_MLP_OFF_W1 + t);
  if (t < WF_MLP_H) {
    S.b1[t] = __ldcg(P + WF_MLP_OFF_B1 + t);
    S.b2[t] = __ldcg(P + WF_MLP_OFF_B2 + t);
    S.w3[t] = __ldcg(P + WF_MLP_OFF_W3 + t);
  }
  const float b3 = __ldcg(P + WF_MLP_OFF_B3);
  float4 gW2[2] = {}, gW1[4] = {};             // gW2 rows 2 ts + r, columns 4 to; gW1 of unit 4 to + r
  float4 gb1 = {};                             // units 4 to ..
  float gb2[4] = {}, gw3[4] = {};              // units to + 16 r
  float gb3 = 0.0f, loss = 0.0f;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += rows) {
    const bool valid = tile * kTile + ts < count;
    const float4 x = x_next;
    const float target = target_next;
    fetch(tile + rows);
    __syncthreads();                           // the last tile's arrays are done with
    if (to == 0) S.X[ts] = x;
    {  // layer 1: units 4 to .. 4 to + 3
      float h[4], d[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int o = 4 * to + q;
        const float4 w = *reinterpret_cast<const float4*>(S.W1 + 4 * o);
        const float z = dot4(S.b1[o], w, x);
        const float sg = 1.0f / (1.0f + expf(-z));
        h[q] = valid ? z * sg : 0.0f;
        d[q] = sg * (1.0f + z * (1.0f - sg));
      }
      *reinterpret_cast<float4*>(S.H1 + ts * LDA + 4 * to) = make_float4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<float4*>(S.D1 + ts * LDA + 4 * to) = make_float4(d[0], d[1], d[2], d[3]);
    }
    __syncthreads();
    {  // layer 2, output and its gradient: z2 = b2 + W2 h1 for units to + 16 r
      float z[4];
#pragma unroll
      for (int r = 0; r < 4; r++) z[r] = S.b2[to + 16 * r];
#pragma unroll 4
      for (int k = 0; k < WF_MLP_H; k += 4) {
        const float4 h = *reinterpret_cast<const float4*>(S.H1 + ts * LDA + k);
#pragma unroll
        for (int r = 0; r < 4; r++)
          z[r] = dot4(z[r], *reinterpret_cast<const float4*>(S.W2 + (to + 16 * r) * LDA + k), h);
      }
      float h2[4], d2[4], y = 0.0f;
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float w3 = S.w3[to + 16 * r];
        const float sg = 1.0f / (1.0f + expf(-z[r]));
        h2[r] = z[r] * sg;
        d2[r] = w3 * sg * (1.0f + z[r] * (1.0f - sg));
        y += w3 * h2[r];
      }
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
      const float e = valid ? y + b3 - target : 0.0f;
      const float gy = 2.0f * e * inv_total;
      loss += e * e * inv_total;
      gb3 += gy;
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float g = gy * d2[r];
        gw3[r] += gy * h2[r];
        gb2[r] += g;
        S.G2[ts * LDA + to + 16 * r] = g;
      }
    }
    __syncthreads();
    {  // layer 1's gradient: g1 = (W2^T g2) silu'(z1); gW1 = sum_s g1 x, gb1 = sum_s g1
      float4 g1 = {};
#pragma unroll 4
      for (int o = 0; o < WF_MLP_H; o += 4) {
        const float4 ga = *reinterpret_cast<const float4*>(S.G2 + ts * LDA + o);
        const float av[4] = {ga.x, ga.y, ga.z, ga.w};
#pragma unroll
        for (int q = 0; q < 4; q++)
          fma4(g1, av[q], *reinterpret_cast<const float4*>(S.W2 + (o + q) * LDA + 4 * to));
      }
      const float4 d = *reinterpret_cast<const float4*>(S.D1 + ts * LDA + 4 * to);
      const float g[4] = {g1.x * d.x, g1.y * d.y, g1.z * d.z, g1.w * d.w};
#pragma unroll
      for (int q = 0; q < 4; q++) fma4(gW1[q], g[q], x);
      gb1.x += g[0]; gb1.y += g[1]; gb1.z += g[2]; gb1.w += g[3];
    }
    // gW2[o][k] = sum_s g2[s][o] h1[s][k]
#pragma unroll 8
    for (int s = 0; s < kTile; s++) {
      const float2 g = *reinterpret_cast<const float2*>(S.G2 + s * LDA + 2 * ts);
      const float4 h = *reinterpret_cast<const float4*>(S.H1 + s * LDA + 4 * to);
      fma4(gW2[0], g.x, h);
      fma4(gW2[1], g.y, h);
    }
  }
#pragma unroll
  for (int r = 0; r < 2; r++)
    *reinterpret_cast<float4*>(row + WF_MLP_OFF_W2 + (2 * ts + r) * WF_MLP_H + 4 * to) = gW2[r];
  // the sums held per sample: over the two samples of the warp, then over the
  // warps through shared memory (448 values and two scalars per warp)
  constexpr int kRed = 7 * WF_MLP_H + 2;
  float* red = reinterpret_cast<float*>(smem_raw) + (t >> 5) * kRed;
  float v[30] = {gb1.x,    gb1.y,    gb1.z,    gb1.w,    gb2[0],   gb2[1],   gb2[2],   gb2[3],
                 gw3[0],   gw3[1],   gw3[2],   gw3[3],   gW1[0].x, gW1[0].y, gW1[0].z, gW1[0].w,
                 gW1[1].x, gW1[1].y, gW1[1].z, gW1[1].w, gW1[2].x, gW1[2].y, gW1[2].z, gW1[2].w,
                 gW1[3].x, gW1[3].y, gW1[3].z, gW1[3].w, gb3,      loss};
#pragma unroll
  for (int q = 0; q < 30; q++) v[q] += __shfl_xor_sync(0xffffffffu, v[q], 16);
  __syncthreads();                             // the tile arrays become the reduction buffer
  if ((t & 31) < 16) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      red[4 * to + q] = v[q];
      red[WF_MLP_H + to + 16 * q] = v[4 + q];
      red[2 * WF_MLP_H + to + 16 * q] = v[8 + q];
    }
#pragma unroll
    for (int q = 0; q < 16; q++) red[3 * WF_MLP_H + 16 * to + q] = v[12 + q];
    if (to == 0) {
      red[kRed - 2] = v[28];
      red[kRed - 1] = v[29];
    }
  }
  __syncthreads();
  if (t >= kRed) return;
  const float* all = reinterpret_cast<const float*>(smem_raw) + t;
  float a = 0.0f;
#pragma unroll
  for (int w = 0; w < kGradThreads / 32; w++) a += all[w * kRed];
  const int at = t < WF_MLP_H        ? WF_MLP_OFF_B1 + t
                 : t < 2 * WF_MLP_H  ? WF_MLP_OFF_B2 + t - WF_MLP_H
                 : t < 3 * WF_MLP_H  ? WF_MLP_OFF_W3 + t - 2 * WF_MLP_H
                 : t < 7 * WF_MLP_H  ? WF_MLP_OFF_W1 + t - 3 * WF_MLP_H
                 : t == 7 * WF_MLP_H ? WF_MLP_OFF_B3
                                     : WF_MLP_NPARAM;
  row[at] = a;
}

__global__ void __launch_bounds__(kGradThreads) k_mlp_grad(const float* __restrict__ P,
                                                          const float4* __restrict__ X,
                                                          const float* __restrict__ Yt,
                                                          int64_t offset, int64_t count,
                                                          float inv_total,
                                                          float* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  grad_block(smem_raw, P, X, Yt, offset, count, inv_total, (int)gridDim.x,
             part + (int64_t)blockIdx.x * kPartRow);
}

// The rows' sum of value 32 chunk + lane, on every thread of the eight warps w
// that share a chunk: eight threads per value, each every eighth row.  Every
// thread of the block takes part.
__device__ __forceinline__ float total_of_rows(float (*sum)[32], const float* part, int rows,
                                               int chunk, int w) {
  const int lane = threadIdx.x & 31;
  const float* p = part + chunk * 32 + lane;
  float a = 0.0f;
#pragma unroll 16
  for (int r = w; r < rows; r += 8) a += __ldcg(p + (int64_t)r * kPartRow);
  sum[w][lane] = a;
  __syncthreads();
  a = 0.0f;
  for (int k = 0; k < 8; k++) a += sum[k][lane];
  return a;
}

__global__ void __launch_bounds__(256) k_grad_total(const float* __restrict__ part, int rows,
                                                    float* __restrict__ grad,
                                                    float* __restrict__ loss) {
  __shared__ float sum[8][32];
  const float a = total_of_rows(sum, part, rows, blockIdx.x, threadIdx.x >> 5);
  const int k = blockIdx.x * 32 + threadIdx.x;
  if (threadIdx.x >= 32) return;
  if (k < WF_MLP_NPARAM) grad[k] = a;
  else if (k == WF_MLP_NPARAM) *loss = a;
}

// A step's learning rate and the moments' bias corrections
struct AdamStep {
  float lr, c1, c2;
};
struct AdamState {
  float *P, *m, *v;
};
// one Adam step of value k (the value behind the last parameter is the loss): its
// state is loaded while the gradient is summed
struct AdamValue {
  float p = 0.0f, m = 0.0f, v = 0.0f;
  __device__ __forceinline__ void load(const AdamState& A, int k) {
    if (k >= WF_MLP_NPARAM) return;
    p = __ldcg(A.P + k);
    m = A.m[k];
    v = A.v[k];
  }
  __device__ __forceinline__ void step(const AdamState& A, int k, float gk, const AdamStep& c,
                                       float* loss) const {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    if (k == WF_MLP_NPARAM) *loss = gk;
    if (k >= WF_MLP_NPARAM) return;
    const float mk = b1 * m + (1.0f - b1) * gk;
    const float vk = b2 * v + (1.0f - b2) * gk * gk;
    A.m[k] = mk;
    A.v[k] = vk;
    A.P[k] = p - c.lr * (mk / c.c1) / (sqrtf(vk / c.c2) + eps);
  }
};

__global__ void __launch_bounds__(256) k_adam(AdamState A, const float* __restrict__ part, int rows,
                                              float* __restrict__ loss, AdamStep c) {
  __shared__ float sum[8][32];
  const int k = threadIdx.x < 32 ? blockIdx.x * 32 + threadIdx.x : INT_MAX;
  AdamValue value;
  value.load(A, k);
  const float gk = total_of_rows(sum, part, rows, blockIdx.x, threadIdx.x >> 5);
  value.step(A, k, gk, c, loss);
}

// ---- many training steps in one cooperative launch ------------------------------
// As two launches a step, 4,096 samples take 21 us, several of them the launches
// and the kernels' ramps.  Here the blocks stay: each step is the gradient of
// its rows, a barrier of the grid, Adam on 32 values per half block, and a
// second barrier; the sums and their order are those of the two kernels.
// 16.5 us a step: gradient 10.5 (the tile's products 7, by shared memory reads
// and their latency), Adam 3.7, the barriers 2.4.  The blocks must all be
// resident (a cooperative launch, one block an SM: batches of up to 32 samples
// an SM; larger ones take the two kernels).  A barrier gives up after
// kSpinLimit polls (seconds): the block sets `bad` and leaves, and so do the
// others.
constexpr int kSpinLimit = 1 << 22;
constexpr int64_t kTrainChunk = 1024;        // most steps of a launch

__device__ __forceinline__ bool grid_barrier(unsigned* arrived, unsigned goal, int* bad) {
  __syncthreads();
  bool ok = true;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(arrived, 1u);
    int n = 0;
    unsigned v;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
    } while ((int)(v - goal) < 0 && ++n < kSpinLimit);
    ok = (int)(v - goal) >= 0;
    if (!ok) atomicExch(bad, 1);
  }
  return __syncthreads_and(ok);
}

__global__ void __launch_bounds__(kGradThreads) k_mlp_train(
    AdamState A, const float4* __restrict__ X, const float* __restrict__ Yt, int64_t n,
    int64_t batch, int64_t off, const AdamStep* __restrict__ sched, int steps, float* part,
    float* loss, unsigned* arrived, int* bad) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float sum[2][8][32];
  const int half = threadIdx.x >> 8, w = (threadIdx.x >> 5) & 7, lane = threadIdx.x & 31;
  unsigned goal = 0;
  for (int st = 0; st < steps; st++) {
    const int64_t cnt = min(batch, n - off);
    const int rows = (int)min((cnt + kTile - 1) / kTile, (int64_t)kGradBlocks);
    if ((int)blockIdx.x < rows)
      grad_block(smem_raw, A.P, X, Yt, off, cnt, 1.0f / (float)cnt, rows,
                 part + (int64_t)blockIdx.x * kPartRow);
    goal += gridDim.x;
    if (!grid_barrier(arrived, goal, bad)) return;
    const AdamStep c = sched[st];
    for (int base = 0; base < kPartRow / 32; base += 2 * gridDim.x) {     // whole blocks together
      const int chunk = base + 2 * blockIdx.x + half;
      const bool mine = chunk < kPartRow / 32;
      const int k = mine && w == 0 ? chunk * 32 + lane : INT_MAX;
      AdamValue value;
      value.load(A, k);
      const float gk = total_of_rows(sum[half], part, mine ? rows : 0, mine ? chunk : 0, w);
      value.step(A, k, gk, c, loss + st);
      __syncthreads();
    }
    goal += gridDim.x;
    if (!grid_barrier(arrived, goal, bad)) return;
    off += cnt;
    if (off >= n) off = 0;
  }
}

// partial-sum rows (blocks) of a gradient over `count` samples
int grad_rows(int64_t count) {
  return (int)std::min<int64_t>((count + kTile - 1) / kTile, kGradBlocks);
}
// the opt-in for the gradient kernel's shared memory, on the current device
cudaError_t grad_ready() {
  const cudaError_t e = cudaFuncSetAttribute(
      k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradShared));
  return e != cudaSuccess ? e
                          : cudaFuncSetAttribute(k_mlp_train,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)sizeof(GradShared));
}
// do `blocks` blocks of k_mlp_train run at once on the current device?
bool train_fits(int blocks) {
  int dev = 0, coop = 0, sms = 0, per = 0;
  return cudaGetDevice(&dev) == cudaSuccess &&
         cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop &&
         cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mlp_train, kGradThreads,
                                                       sizeof(GradShared)) == cudaSuccess &&
         blocks <= per * sms;
}

StepParams jc_params(const wf_material* m, double rtol) {
  StepParams P;
  memset(&P, 0, sizeof P);
  P.newton_max_iter = 200;
  P.newton_rtol = rtol;
  P.clamp_homologous = 1;
  MatParams& M = P.mat;
  M.model = m->model;
  M.E = m->E;
  M.A = m->A; M.B = m->B; M.n = m->n; M.C = m->C; M.eps0 = m->eps0; M.m = m->m;
  M.Tm = m->Tm; M.Tt = m->Tt;
  double c = 1.0;
  for (int k = 1; k <= 5; k++) {
    c = c * (m->n - (k - 1)) / k;
    M.bin[k - 1] = c;
  }
  return P;
}

// RAII device buffers for the standalone entry points
struct DevBufs {
  std::vector<void*> ptrs;
  ~DevBufs() {
    for (void* p : ptrs) cudaFree(p);
  }
  template <class T>
  T* get(size_t count) {
    void* p = nullptr;
    if (cudaMalloc(&p, sizeof(T) * (count ? count : 1)) != cudaSuccess) return nullptr;
    ptrs.push_back(p);
    return (T*)p;
  }
};

inline int nb(int64_t n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

// packs FP32 parameters into the BF16 fragment image used by the kernels
int wf_mlp_pack_device(const float* dparams, void* dpacked, cudaStream_t s) {
  k_mlp_pack_umma<<<1, 256, 0, s>>>(dparams, (uint8_t*)dpacked);
  return cudaGetLastError() == cudaSuccess ? WF_OK : WF_ERR_CUDA;
}
size_t wf_mlp_packed_bytes() { return WF_UMMA_IMAGE; }

extern "C" {

int wf_mlp_infer(const float* params, const float* X, int64_t n, int use_tensor_cores, float* Y) {
  if (!params || !X || !Y || n <= 0) return WF_ERR_ARG;
  DevBufs B;
  float* dP = B.get<float>(WF_MLP_NPARAM);
  float4* dX = B.get<float4>(n);
  float* dY = B.get<float>(n);
  if (!dP || !dX || !dY) return WF_ERR_ALLOC;
  cudaMemcpy(dP, params, sizeof(float) * WF_MLP_NPARAM, cudaMemcpyHostToDevice);
  cudaMemcpy(dX, X, sizeof(float) * 4 * n, cudaMemcpyHostToDevice);
  if (use_tensor_cores) {
    uint4* dI = B.get<uint4>(WF_UMMA_IMAGE / 16);
    int* dS = B.get<int>(1);
    if (!dI || !dS) return WF_ERR_ALLOC;
    cudaMemset(dS, 0, sizeof(int));
    k_mlp_pack_umma<<<1, 256>>>(dP, (uint8_t*)dI);
    k_mlp_infer_umma<<<nb(n, 128), 128, WF_UMMA_SMEM>>>(dI, mlp_l1_from(params), dX, n, dY, dS);
    int st = 0;
    cudaMemcpy(&st, dS, sizeof(int), cudaMemcpyDeviceToHost);
    if (st & WF_STATUS_MMA_WAIT) return WF_ERR_CUDA;
  } else {
    k_mlp_infer_f32<<<nb(n, 128), 128>>>(dP, dX, n, dY);
  }
  if (cudaMemcpy(Y, dY, sizeof(float) * n, cudaMemcpyDeviceToHost) != cudaSuccess) return WF_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? WF_OK : WF_ERR_CUDA;
}

int wf_mlp_grad(const float* params, const float* X, const float* Y, int64_t n, float* grad,
                float* loss) {
  if (!params || !X || !Y || !grad || !loss || n <= 0) return WF_ERR_ARG;
  DevBufs B;
  float* dP = B.get<float>(WF_MLP_NPARAM);
  float4* dX = B.get<float4>(n);
  float* dY = B.get<float>(n);
  float* dG = B.get<float>(WF_MLP_NPARAM);
  float* dL = B.get<float>(1);
  if (!dP || !dX || !dY || !dG || !dL) return WF_ERR_ALLOC;
  cudaMemcpy(dP, params, sizeof(float) * WF_MLP_NPARAM, cudaMemcpyHostToDevice);
  cudaMemcpy(dX, X, sizeof(float) * 4 * n, cudaMemcpyHostToDevice);
  cudaMemcpy(dY, Y, sizeof(float) * n, cudaMemcpyHostToDevice);
  const int rows = grad_rows(n);
  float* dR = B.get<float>((size_t)rows * kPartRow);
  if (!dR) return WF_ERR_ALLOC;
  if (grad_ready() != cudaSuccess) return WF_ERR_CUDA;
  k_mlp_grad<<<rows, kGradThreads, sizeof(GradShared)>>>(dP, dX, dY, 0, n, 1.0f / (float)n, dR);
  k_grad_total<<<kPartRow / 32, 256>>>(dR, rows, dG, dL);
  cudaMemcpy(grad, dG, sizeof(float) * WF_MLP_NPARAM, cudaMemcpyDeviceToHost);
  if (cudaMemcpy(loss, dL, sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess) return WF_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? WF_OK : WF_ERR_CUDA;
}

int wf_mlp_train(float* params, const float* X, const float* Y, int64_t n, int64_t steps,
                 int64_t batch, float lr, float* final_loss) {
  if (!params || !X || !Y || n <= 0 || steps <= 0 || batch <= 0) return WF_ERR_ARG;
  // one device block: samples, targets, parameters and moments, partial sums, losses, the steps'
  // rates, the barrier's words
  const int most = grad_rows(std::min<int64_t>(batch, n));
  const auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t bX = up(sizeof(float4) * n), bY = up(sizeof(float) * n),
               bP = up(sizeof(float) * WF_MLP_NPARAM), bR = up(sizeof(float) * most * kPartRow),
               bL = up(sizeof(float) * steps), bS = up(sizeof(AdamStep) * steps);
  DevBufs B;
  char* base = B.get<char>(bX + bY + 3 * bP + bR + bL + bS + 256);
  if (!base) return WF_ERR_ALLOC;
  float4* dX = (float4*)base;
  float* dY = (float*)(base + bX);
  float* dP = (float*)(base + bX + bY);
  const AdamState A{dP, (float*)((char*)dP + bP), (float*)((char*)dP + 2 * bP)};
  float* dR = (float*)((char*)dP + 3 * bP);
  float* dL = (float*)((char*)dR + bR);
  AdamStep* dS = (AdamStep*)((char*)dL + bL);
  unsigned* dB = (unsigned*)((char*)dS + bS);          // barrier arrivals, failure
  std::vector<AdamStep> sched(steps);
  double p1 = 1.0, p2 = 1.0;
  for (int64_t st = 0; st < steps; st++) {
    p1 *= 0.9f;
    p2 *= 0.999f;
    // cosine decay of the learning rate
    sched[st] = AdamStep{lr * 0.5f * (1.0f + cosf(3.14159265f * (float)st / (float)steps)),
                         (float)(1.0 - p1), (float)(1.0 - p2)};
  }
  cudaMemcpy(dP, params, sizeof(float) * WF_MLP_NPARAM, cudaMemcpyHostToDevice);
  cudaMemcpy(dX, X, sizeof(float) * 4 * n, cudaMemcpyHostToDevice);
  cudaMemcpy(dY, Y, sizeof(float) * n, cudaMemcpyHostToDevice);
  cudaMemset(A.m, 0, 2 * bP);
  if (grad_ready() != cudaSuccess) return WF_ERR_CUDA;
  int64_t off = 0, st = 0;
  const auto advance = [&] {                           // the next step's first sample
    off += std::min<int64_t>(batch, n - off);
    if (off >= n) off = 0;
    st++;
  };
  if (train_fits(most)) {
    cudaMemcpy(dS, sched.data(), sizeof(AdamStep) * steps, cudaMemcpyHostToDevice);
    cudaMemset(dB, 0, 2 * sizeof(unsigned));
    while (st < steps) {
      int count = (int)std::min<int64_t>(kTrainChunk, steps - st);
      cudaMemsetAsync(dB, 0, sizeof(unsigned));
      const AdamStep* s0 = dS + st;
      float* l0 = dL + st;
      int* bad = (int*)dB + 1;
      AdamState state = A;
      void* args[] = {&state, &dX, &dY, &n, &batch, &off, &s0, &count, &dR, &l0, &dB, &bad};
      if (cudaLaunchCooperativeKernel((const void*)k_mlp_train, dim3(most), dim3(kGradThreads),
                                      args, sizeof(GradShared), nullptr) != cudaSuccess) {
        cudaGetLastError();                            // not all of its blocks run at once here
        break;
      }
      for (int k = 0; k < count; k++) advance();
    }
    int bad = 0;
    if (cudaMemcpy(&bad, dB + 1, sizeof bad, cudaMemcpyDeviceToHost) != cudaSuccess || bad)
      return WF_ERR_CUDA;
  }
  for (; st < steps; advance()) {
    const int64_t cnt = std::min<int64_t>(batch, n - off);
    const int rows = grad_rows(cnt);
    k_mlp_grad<<<rows, kGradThreads, sizeof(GradShared)>>>(dP, dX, dY, off, cnt, 1.0f / (float)cnt,
                                                          dR);
    k_adam<<<kPartRow / 32, 256>>>(A, dR, rows, dL + st, sched[st]);
  }
  cudaMemcpy(params, dP, sizeof(float) * WF_MLP_NPARAM, cudaMemcpyDeviceToHost);
  if (final_loss) {
    std::vector<float> L(steps);
    cudaMemcpy(L.data(), dL, sizeof(float) * steps, cudaMemcpyDeviceToHost);
    const int64_t k0 = std::max<int64_t>(0, steps - 20);
    double acc = 0.0;
    for (int64_t k = k0; k < steps; k++) acc += L[k];
    *final_loss = (float)(acc / (double)(steps - k0));
  }
  return cudaGetLastError() == cudaSuccess ? WF_OK : WF_ERR_CUDA;
}

int wf_mlp_synth(const wf_material* mat, double G, int64_t n, uint64_t seed, double rtol,
                 float* X, float* Y, float* states, int32_t* iters_radial) {
  if (!mat || !X || !Y || !states || !iters_radial || n <= 0) return WF_ERR_ARG;
  if (mat->model != WF_JOHNSON_COOK) return WF_ERR_ARG;
  DevBufs B;
  float4* dX = B.get<float4>(n);
  float* dY = B.get<float>(n);
  float4* dS = B.get<float4>(n);
  int32_t* dI = B.get<int32_t>(n);
  if (!dX || !dY || !dS || !dI) return WF_ERR_ALLOC;
  StepParams P = jc_params(mat, rtol);
  k_mlp_synth<<<nb(n, 128), 128>>>(P, G, n, seed, dX, dY, dS, dI);
  cudaMemcpy(X, dX, sizeof(float) * 4 * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(Y, dY, sizeof(float) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(states, dS, sizeof(float) * 4 * n, cudaMemcpyDeviceToHost);
  if (cudaMemcpy(iters_radial, dI, sizeof(int32_t) * n, cudaMemcpyDeviceToHost) != cudaSuccess)
    return WF_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? WF_OK : WF_ERR_CUDA;
}

int wf_mlp_newton_iters(const wf_material* mat, double G, const float* params, const float* states,
                        int64_t n, double rtol, int32_t* iters, int32_t* used, float* dl) {
  if (!mat || !states || !iters || !used || !dl || n <= 0) return WF_ERR_ARG;
  DevBufs B;
  float4* dS = B.get<float4>(n);
  int32_t* dI = B.get<int32_t>(n);
  int32_t* dU = B.get<int32_t>(n);
  float* dD = B.get<float>(n);
  float* dP = B.get<float>(WF_MLP_NPARAM);
  uint4* dW = B.get<uint4>(WF_UMMA_IMAGE / 16);
  int* dSt = B.get<int>(1);
  if (!dS || !dI || !dU || !dD || !dP || !dW || !dSt) return WF_ERR_ALLOC;
  cudaMemcpy(dS, states, sizeof(float) * 4 * n, cudaMemcpyHostToDevice);
  cudaMemset(dSt, 0, sizeof(int));
  if (params) {
    cudaMemcpy(dP, params, sizeof(float) * WF_MLP_NPARAM, cudaMemcpyHostToDevice);
    k_mlp_pack_umma<<<1, 256>>>(dP, (uint8_t*)dW);
  }
  StepParams P = jc_params(mat, rtol);
  const MlpL1 l1 = params ? mlp_l1_from(params) : MlpL1{};
  k_mlp_newton_iters<<<nb(n, 128), 128, params ? WF_UMMA_SMEM : 0>>>(
      P, G, params ? dW : nullptr, l1, dS, n, dI, dU, dD, dSt);
  cudaMemcpy(iters, dI, sizeof(int32_t) * n, cudaMemcpyDeviceToHost);
  cudaMemcpy(used, dU, sizeof(int32_t) * n, cudaMemcpyDeviceToHost);
  if (cudaMemcpy(dl, dD, sizeof(float) * n, cudaMemcpyDeviceToHost) != cudaSuccess) return WF_ERR_CUDA;
  int st = 0;
  cudaMemcpy(&st, dSt, sizeof(int), cudaMemcpyDeviceToHost);
  if (st & WF_STATUS_MMA_WAIT) return WF_ERR_CUDA;
  return cudaGetLastError() == cudaSuccess ? WF_OK : WF_ERR_CUDA;
}

}  // extern "C"

static_assert(WF_MLP_NPARAM == WF_MLP_NPARAMS, "MLP parameter count mismatch between header and kernels");
