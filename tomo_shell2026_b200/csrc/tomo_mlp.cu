// Training and inference kernels of the surrogate MLP (see tomo_mlp.cuh).
//
// The network is small (33,793 parameters, 128-wide), and the training set
// is a coarse orientation grid (~10^3 samples), so a step is latency-bound,
// not FLOP-bound.  A step is two launches:
//
//   k_mlp_pass     one CTA per 8 samples: forward pass, loss and the whole
//                  backward pass to the layers' inputs out of shared memory;
//                  activations and pre-activation gradients go to global
//                  memory (3 MB for 936 samples);
//   k_mlp_update   one CTA per 16 x 16 weights (and per 16 of the rest): the
//                  weight gradient over all samples, then the Adam update of
//                  the parameter and of its transposed copy.
//
// The gradient is summed in a fixed order (deterministic): over each 8 samples
// in turn, the sums of eights r, r + 8, r + 16, ... of each r in 0..7, then the
// eight of those.  When each CTA wrote its own gradient of all parameters and a
// second kernel added them up (16 MB written and read a step), a step of 936
// samples took 31 us; now 21 (B200, 300 steps replayed as a graph): 12 of it four
// dependent 128-term products and three activations on one warp per scheduler,
// bound by shared-memory words, 5 the weight gradients, the rest launches.
//
// Weights are row-major [in][out]; the backward pass reads each matrix
// through a transposed copy [out][in] kept in step with the parameters, so
// both passes read weights with consecutive threads on consecutive
// addresses.  FMAs are explicit (the library is built with -fmad=false for
// the exact path; this code is not on it).
#include "tomo_mlp.cuh"

#include <cmath>
#include <cstring>
#include <random>

namespace tomo {

namespace {

constexpr int kSB = 8;           // samples per k_mlp_pass CTA and per partial gradient sum
constexpr int kFB = 64;          // samples per k_mlp_forward CTA and turn at most, eight per warp
constexpr int kH = kMlpHidden;   // 128
constexpr int kParts = 8;        // partial gradient sums per parameter

__device__ __forceinline__ void cp16(void* smem, const void* g)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(g));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }

// Start copying one 128 x 128 matrix into shared memory (one commit group), by
// the threads from `first` on.
__device__ __forceinline__ void stage(const float* __restrict__ src, float* dst, int first = 0)
{
  if ((int)threadIdx.x < first) return;
  for (int k = threadIdx.x - first; k < kH * kH / 4; k += blockDim.x - first) cp16(dst + 4 * k, src + 4 * k);
  cp_commit();
}

// a * w + c for two samples, each rounded once as __fmaf_rn rounds it.
__device__ __forceinline__ float2 fma2(float2 a, float2 w, float2 c)
{
  float2 r;
  asm("{.reg .b64 a, w, c, r;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 w, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 r, a, w, c;\n\tmov.b64 {%0, %1}, r;}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(w.x), "f"(w.y), "f"(c.x), "f"(c.y));
  return r;
}

// out[j][s] = sum over i (in order, from b[j] or zero) of in[i][s] * W[i][j] for
// eight samples and 128 units, by the first two warps: a thread has four units
// x four samples, so that eight shared-memory words serve sixteen products (a
// thread per unit with all eight samples took nine words for eight products,
// and shared memory returns 32 words a cycle: 36 cycles per i instead of 16).
// The next rows are read while these are used; the other warps stage the next
// matrix meanwhile.  3,650 cycles (single products 4,300: a warp by itself on its
// scheduler issues one every other cycle, packed or not).
__device__ __forceinline__ void matmul8(const float (*in)[kSB], const float* W, const float* b, float (*out)[kSB])
{
  constexpr int kRows = 8;
  if (threadIdx.x >= 64) return;
  const int j0 = (threadIdx.x & 31) * 4, s0 = (threadIdx.x >> 5) * 4;
  float2 acc[4][2];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float v = b ? b[j0 + c] : 0.f;
    acc[c][0] = acc[c][1] = make_float2(v, v);
  }
  float4 w[2][kRows], a[2][kRows];
  auto load = [&](int i0, float4* pw, float4* pa) {
#pragma unroll
    for (int k = 0; k < kRows; k++) {
      pw[k] = *reinterpret_cast<const float4*>(W + (i0 + k) * kH + j0);
      pa[k] = *reinterpret_cast<const float4*>(&in[i0 + k][s0]);
    }
  };
  auto use = [&](const float4* pw, const float4* pa) {
#pragma unroll
    for (int k = 0; k < kRows; k++) {
      const float2 x = make_float2(pa[k].x, pa[k].y), y = make_float2(pa[k].z, pa[k].w);
      const float wc[4] = {pw[k].x, pw[k].y, pw[k].z, pw[k].w};
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float2 w2 = make_float2(wc[c], wc[c]);
        acc[c][0] = fma2(x, w2, acc[c][0]);
        acc[c][1] = fma2(y, w2, acc[c][1]);
      }
    }
  };
  load(0, w[0], a[0]);
#pragma unroll 1
  for (int i0 = 0; i0 < kH; i0 += 2 * kRows) {
    load(i0 + kRows, w[1], a[1]);
    use(w[0], a[0]);
    if (i0 + 2 * kRows < kH) load(i0 + 2 * kRows, w[0], a[0]);
    use(w[1], a[1]);
  }
#pragma unroll
  for (int c = 0; c < 4; c++)
    *reinterpret_cast<float4*>(&out[j0 + c][s0]) = make_float4(acc[c][0].x, acc[c][0].y, acc[c][1].x, acc[c][1].y);
}

struct alignas(16) PassShared {
  float w[2][kH * kH];       // the two 128 x 128 matrices in use
  float a[3][kH][kSB];       // tanh outputs of the three hidden layers, samples innermost
  float dz[2][kH][kSB];      // pre-activation gradients, ping-pong
  float mm[kH][kSB];         // a product before its activation
  float x[kSB][kMlpIn];
  float yhat[kSB];
  float dz4[kSB];
};
constexpr size_t kPassSmem = sizeof(PassShared);   // ~153 KB: dynamic, opted in

// What a pass leaves for the weight gradients: [rows][128] each (rows: samples
// rounded up to eights), outputs of the hidden layers, gradients before their
// activations, and the output's gradient [rows].
struct PassOut {
  float *a[3], *d[3], *d4;
};

// One thread per hidden unit and eight samples but for the products (matmul8);
// rows past the last sample hold zero features and a zero output gradient.
__global__ void __launch_bounds__(kH) k_mlp_pass(MlpLayout L, const float* __restrict__ P, const float* __restrict__ WT,
                                                 const float* __restrict__ x, const float* __restrict__ y, int n,
                                                 PassOut O, float* __restrict__ part_loss)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PassShared& S = *reinterpret_cast<PassShared*>(smem_raw);
  const int j = threadIdx.x, warp = j >> 5, lane = j & 31;
  const int s0 = blockIdx.x * kSB, ns = min(kSB, n - s0);
  // everything small that is read from global memory, before the matrices
  if (j < kSB * kMlpIn) {
    const int s = j / kMlpIn, i = j % kMlpIn;
    S.x[s][i] = s < ns ? x[(size_t)(s0 + s) * kMlpIn + i] : 0.f;
  }
  const float w4 = P[L.w[3] + j];
  float w0[kMlpIn], w3[kH / 32];
#pragma unroll
  for (int i = 0; i < kMlpIn; i++) w0[i] = P[L.w[0] + i * kH + j];
#pragma unroll
  for (int k = 0; k < kH / 32; k++) w3[k] = P[L.w[3] + lane + 32 * k];
  const float b0 = P[L.b[0] + j], b3 = P[L.b[3]];
  const float target = j < ns ? y[s0 + j] : 0.f;
  stage(P + L.w[1], S.w[0]);
  __syncthreads();
  float v[kSB];
  // outputs of hidden layer l: shared (samples innermost) and global rows
  auto put = [&](float (*dst)[kSB], float* g) {
    *reinterpret_cast<float4*>(&dst[j][0]) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(&dst[j][4]) = make_float4(v[4], v[5], v[6], v[7]);
#pragma unroll
    for (int s = 0; s < kSB; s++) g[(size_t)(s0 + s) * kH + j] = v[s];
  };
#pragma unroll
  for (int s = 0; s < kSB; s++) {
    float acc = b0;
#pragma unroll
    for (int i = 0; i < kMlpIn; i++) acc = __fmaf_rn(S.x[s][i], w0[i], acc);
    v[s] = tanhf(acc);
  }
  put(S.a[0], O.a[0]);
  cp_wait<0>();
  __syncthreads();
  stage(P + L.w[2], S.w[1], 64);
  matmul8(S.a[0], S.w[0], P + L.b[1], S.mm);
  __syncthreads();
#pragma unroll
  for (int s = 0; s < kSB; s++) v[s] = tanhf(S.mm[j][s]);
  put(S.a[1], O.a[1]);
  cp_wait<0>();
  __syncthreads();
  stage(WT + L.w[2], S.w[0], 64);        // [out][in], for the backward pass
  matmul8(S.a[1], S.w[1], P + L.b[2], S.mm);
  __syncthreads();
#pragma unroll
  for (int s = 0; s < kSB; s++) v[s] = tanhf(S.mm[j][s]);
  put(S.a[2], O.a[2]);
  cp_wait<0>();
  __syncthreads();
  for (int s = warp * 2; s < warp * 2 + 2; s++) {
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < kH / 32; k++) acc = __fmaf_rn(S.a[2][lane + 32 * k][s], w3[k], acc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
    if (lane == 0) S.yhat[s] = acc + b3;
  }
  __syncthreads();
  // loss and output-layer gradient
  if (j < 32) {
    float e = 0.f;
    if (j < kSB) {
      const float d = j < ns ? S.yhat[j] - target : 0.f;
      S.dz4[j] = 2.f * d / (float)n;
      O.d4[s0 + j] = S.dz4[j];
      e = d * d / (float)n;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xFFFFFFFFu, e, o);
    if (j == 0) part_loss[blockIdx.x] = e;
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < kSB; s++) {
    const float a = S.a[2][j][s];
    v[s] = S.dz4[s] * w4 * (1.f - a * a);
  }
  put(S.dz[0], O.d[2]);
  __syncthreads();
  stage(WT + L.w[1], S.w[1], 64);
  matmul8(S.dz[0], S.w[0], nullptr, S.mm);
  __syncthreads();
#pragma unroll
  for (int s = 0; s < kSB; s++) {
    const float a = S.a[1][j][s];
    v[s] = S.mm[j][s] * (1.f - a * a);
  }
  put(S.dz[1], O.d[1]);
  cp_wait<0>();
  __syncthreads();
  matmul8(S.dz[1], S.w[1], nullptr, S.mm);
  __syncthreads();
#pragma unroll
  for (int s = 0; s < kSB; s++) {
    const float a = S.a[0][j][s];
    O.d[0][(size_t)(s0 + s) * kH + j] = S.mm[j][s] * (1.f - a * a);
  }
}

struct alignas(16) ForwardShared {
  float w[2][kH * kH];       // both 128 x 128 matrices, loaded once per CTA
  float a[kH][kFB];          // activations, samples innermost
  float x[kFB][kMlpIn];
};
constexpr size_t kForwardSmem = sizeof(ForwardShared);   // ~161 KB: dynamic, opted in

// Prediction: persistent CTAs of eight warps with eight samples each; a thread
// has four units x eight samples (twelve shared-memory words for 32 products,
// which bound this kernel too).  Eights go to the CTAs in turn, so that a few
// hundred samples take a warp per SM and not eight on a few (a call on 100
// samples took 46-50 us that way, 41 with a CTA per 8 samples, now 36).  Every output
// is summed in the order of the training pass.
// 87,120 samples in 195 us (a CTA per 8 samples, loading both matrices each
// time, and nine words for eight products: about 400).
__global__ void __launch_bounds__(256) k_mlp_forward(MlpLayout L, const float* __restrict__ P,
                                                     const float* __restrict__ x, int n, float* __restrict__ out)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ForwardShared& S = *reinterpret_cast<ForwardShared*>(smem_raw);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int j0 = lane * 4, g = warp * 8;   // units j0 .. j0 + 3, samples g .. g + 7
  stage(P + L.w[1], S.w[0]);
  stage(P + L.w[2], S.w[1]);
  float4 w0[kMlpIn], b[3];
#pragma unroll
  for (int i = 0; i < kMlpIn; i++) w0[i] = *reinterpret_cast<const float4*>(P + L.w[0] + i * kH + j0);
#pragma unroll
  for (int l = 0; l < 3; l++) b[l] = *reinterpret_cast<const float4*>(P + L.b[l] + j0);
  float w3[kH / 32];
#pragma unroll
  for (int k = 0; k < kH / 32; k++) w3[k] = P[L.w[3] + lane + 32 * k];
  const float b3 = P[L.b[3]];
  cp_wait<0>();
  __syncthreads();
  // a warp's eight samples never leave it: no barrier from here on
  for (int s0 = (warp * gridDim.x + blockIdx.x) * 8; s0 < n; s0 += gridDim.x * kFB) {
    const int ns = min(8, n - s0);
    {
      const int s = lane / kMlpIn, i = lane % kMlpIn;
      S.x[g + s][i] = s < ns ? x[(size_t)(s0 + s) * kMlpIn + i] : 0.f;
    }
    __syncwarp();
    float v[4][8];
    auto put = [&](float (*to)[kFB]) {
#pragma unroll
      for (int c = 0; c < 4; c++)
#pragma unroll
        for (int q = 0; q < 2; q++)
          *reinterpret_cast<float4*>(&to[j0 + c][g + 4 * q]) =
              make_float4(tanhf(v[c][4 * q]), tanhf(v[c][4 * q + 1]), tanhf(v[c][4 * q + 2]), tanhf(v[c][4 * q + 3]));
    };
#pragma unroll
    for (int s = 0; s < 8; s++) {
      float4 acc = b[0];
#pragma unroll
      for (int i = 0; i < kMlpIn; i++) {
        const float xi = S.x[g + s][i];
        acc.x = __fmaf_rn(xi, w0[i].x, acc.x); acc.y = __fmaf_rn(xi, w0[i].y, acc.y);
        acc.z = __fmaf_rn(xi, w0[i].z, acc.z); acc.w = __fmaf_rn(xi, w0[i].w, acc.w);
      }
      v[0][s] = acc.x; v[1][s] = acc.y; v[2][s] = acc.z; v[3][s] = acc.w;
    }
    put(S.a);
    __syncwarp();
#pragma unroll
    for (int l = 1; l < 3; l++) {
      const float* W = S.w[l - 1];
      const float bb[4] = {b[l].x, b[l].y, b[l].z, b[l].w};
      float2 acc[4][4];
#pragma unroll
      for (int c = 0; c < 4; c++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[c][q] = make_float2(bb[c], bb[c]);
#pragma unroll 4
      for (int i = 0; i < kH; i++) {
        const float4 w = *reinterpret_cast<const float4*>(W + i * kH + j0);
        const float4 a0 = *reinterpret_cast<const float4*>(&S.a[i][g]), a1 = *reinterpret_cast<const float4*>(&S.a[i][g + 4]);
        const float wc[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const float2 w2 = make_float2(wc[c], wc[c]);
          acc[c][0] = fma2(make_float2(a0.x, a0.y), w2, acc[c][0]);
          acc[c][1] = fma2(make_float2(a0.z, a0.w), w2, acc[c][1]);
          acc[c][2] = fma2(make_float2(a1.x, a1.y), w2, acc[c][2]);
          acc[c][3] = fma2(make_float2(a1.z, a1.w), w2, acc[c][3]);
        }
      }
#pragma unroll
      for (int c = 0; c < 4; c++)
#pragma unroll
        for (int q = 0; q < 4; q++) { v[c][2 * q] = acc[c][q].x; v[c][2 * q + 1] = acc[c][q].y; }
      __syncwarp();
      put(S.a);
      __syncwarp();
    }
    for (int s = 0; s < 8; s++) {
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < kH / 32; k++) acc = __fmaf_rn(S.a[lane + 32 * k][g + s], w3[k], acc);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
      if (lane == 0 && s < ns) out[s0 + s] = acc + b3;
    }
    __syncwarp();
  }
}

// Transposed-copy index of weight p (or -1 for a bias).
__device__ __forceinline__ int transposed_index(const MlpLayout& L, int p)
{
#pragma unroll
  for (int l = 0; l < kMlpLayers; l++) {
    const int r = p - L.w[l];
    if (r >= 0 && r < L.in[l] * L.out[l]) return L.w[l] + (r % L.out[l]) * L.in[l] + r / L.out[l];
  }
  return -1;
}

__device__ __forceinline__ void adam_update(const MlpLayout& L, int p, float gi, float* P, float* WT, float* m,
                                            float* v, float lr, float bc1, float bc2)
{
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float mi = b1 * m[p] + (1.f - b1) * gi;
  const float vi = b2 * v[p] + (1.f - b2) * gi * gi;
  m[p] = mi;
  v[p] = vi;
  const float np = P[p] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  P[p] = np;
  const int q = transposed_index(L, p);
  if (q >= 0) WT[q] = np;
}

constexpr int kTile = 16;                                       // 16 x 16 weights per CTA
constexpr int kTilesPerLayer = (kH / kTile) * (kH / kTile);     // 64
constexpr int kUpdateThreads = 16 * kParts;                      // sixteen per partial sum
constexpr int kSmallPer = 16;                                   // other parameters per CTA
constexpr int kStages = 4;                                      // eights in flight per warp

// The parameters outside the two 128 x 128 matrices, numbered 0 .. kSmall - 1:
// W1, b1, b2, b3, W4, b4.
constexpr int kSmall = kMlpIn * kH + 3 * kH + kH + 1;

// Weight gradients and (update) the Adam step.  Sixteen threads r of a CTA sum
// the partial gradients of the eights r, r + 8, ... (each eight in sample order);
// the eight sums are then added in order.  nblk: eights of samples.
__global__ void __launch_bounds__(kUpdateThreads) k_mlp_update(MlpLayout L, const float* __restrict__ x, PassOut O,
                                                            const float* __restrict__ part_loss, int nblk,
                                                            float* __restrict__ grad, float* __restrict__ loss,
                                                            int update, float* P, float* WT, float* m, float* v,
                                                            float lr, float bc1, float bc2)
{
  __shared__ float red[kParts][kTile * kTile + 1];
  __shared__ __align__(16) float ring[kParts][kStages][2][kSB][kTile];   // activations, gradients
  const int lane = threadIdx.x & 31;
  const int tile = blockIdx.x;
  if (tile < 2 * kTilesPerLayer) {
    // 16 x 16 weights of layer l: sixteen threads with 4 inputs x 4 outputs each,
    // so a warp has two of the partial sums r.  Their eights arrive kStages - 1
    // ahead (a row's 16 inputs and 16 outputs are four 16-byte pieces each, two of
    // either per thread and eight).
    const int l = 1 + tile / kTilesPerLayer, q = tile % kTilesPerLayer;
    const int t = lane & 15, r = threadIdx.x >> 4;
    const int ti = (t >> 2) * 4, tj = (t & 3) * 4;
    const float* A = O.a[l - 1] + q / (kH / kTile) * kTile + (t >> 2) * kH + tj;
    const float* D = O.d[l] + q % (kH / kTile) * kTile + (t >> 2) * kH + tj;
    float acc[4][4];
#pragma unroll
    for (int h = 0; h < 4; h++)
#pragma unroll
      for (int c = 0; c < 4; c++) acc[h][c] = 0.f;
    auto fetch = [&](int b, int k) {
      if (b < nblk) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          cp16(&ring[r][k % kStages][0][(t >> 2) + 4 * h][tj], A + ((size_t)b * kSB + 4 * h) * kH);
          cp16(&ring[r][k % kStages][1][(t >> 2) + 4 * h][tj], D + ((size_t)b * kSB + 4 * h) * kH);
        }
      }
      cp_commit();
    };
#pragma unroll
    for (int k = 0; k < kStages - 1; k++) fetch(r + k * kParts, k);
    const int turns = (nblk + kParts - 1) / kParts;   // the same for both halves of a warp
    for (int k = 0; k < turns; k++) {
      const int b = r + k * kParts;
      cp_wait<kStages - 2>();
      __syncwarp();
      fetch(b + (kStages - 1) * kParts, k + kStages - 1);   // into the stage read one turn ago
      if (b < nblk) {
        float p[4][4];
#pragma unroll
        for (int h = 0; h < 4; h++)
#pragma unroll
          for (int c = 0; c < 4; c++) p[h][c] = 0.f;
#pragma unroll
        for (int s = 0; s < kSB; s++) {
          const float4 a = *reinterpret_cast<const float4*>(&ring[r][k % kStages][0][s][ti]);
          const float4 d = *reinterpret_cast<const float4*>(&ring[r][k % kStages][1][s][tj]);
          const float av[4] = {a.x, a.y, a.z, a.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
          for (int h = 0; h < 4; h++)
#pragma unroll
            for (int c = 0; c < 4; c++) p[h][c] = __fmaf_rn(av[h], dv[c], p[h][c]);
        }
#pragma unroll
        for (int h = 0; h < 4; h++)
#pragma unroll
          for (int c = 0; c < 4; c++) acc[h][c] += p[h][c];
      }
      __syncwarp();
    }
#pragma unroll
    for (int h = 0; h < 4; h++)
#pragma unroll
      for (int c = 0; c < 4; c++) red[r][(ti + h) * kTile + tj + c] = acc[h][c];
    __syncthreads();
    for (int e = threadIdx.x; e < kTile * kTile; e += kUpdateThreads) {
      float gi = 0.f;
#pragma unroll
      for (int k = 0; k < kParts; k++) gi += red[k][e];
      const int w = L.w[l] + (q / (kH / kTile) * kTile + e / kTile) * kH + q % (kH / kTile) * kTile + e % kTile;
      grad[w] = gi;
      if (update) adam_update(L, w, gi, P, WT, m, v, lr, bc1, bc2);
    }
    return;
  }
  if (blockIdx.x == gridDim.x - 1) {
    // the loss: the eights' losses in order
    float e = 0.f;
    float* const part = &ring[0][0][0][0][0];
    for (int b0 = 0; b0 < nblk; b0 += kUpdateThreads) {
      if (b0 + (int)threadIdx.x < nblk) part[threadIdx.x] = part_loss[b0 + threadIdx.x];
      __syncthreads();
      if (threadIdx.x == 0) {
        const int m = min(kUpdateThreads, nblk - b0);
#pragma unroll 8
        for (int k = 0; k < m; k++) e += part[k];
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) *loss = e;
    return;
  }
  // the rest: 16 parameters, a thread per parameter and partial sum; four eights'
  // factors are read before the first is used
  const int t = threadIdx.x & 15, r = threadIdx.x >> 4;
  const int k = (tile - 2 * kTilesPerLayer) * kSmallPer + t;
  int par = -1;
  const float *u = nullptr, *v2 = nullptr;   // the factors' first values; v2 null: the sum of u alone
  int su = kH, sv = 0;                        // and their strides from sample to sample
  if (k < kSmall) {
    int e = k;
    if (e < kMlpIn * kH) {
      par = L.w[0] + e; u = x + e / kH; su = kMlpIn; v2 = O.d[0] + e % kH; sv = kH;
    } else if ((e -= kMlpIn * kH) < 3 * kH) {
      par = L.b[e / kH] + e % kH; u = O.d[e / kH] + e % kH;
    } else if ((e -= 3 * kH) < kH) {
      par = L.w[3] + e; u = O.a[2] + e; v2 = O.d4; sv = 1;
    } else {
      par = L.b[3]; u = O.d4; su = 1;
    }
  }
  float acc = 0.f;
  constexpr int kAhead = 4;
  if (par >= 0)
    for (int b0 = r; b0 < nblk; b0 += kAhead * kParts) {
      float fu[kAhead][kSB], fv[kAhead][kSB];
#pragma unroll
      for (int a = 0; a < kAhead; a++)
#pragma unroll
        for (int s = 0; s < kSB; s++) {
          const int row = (b0 + a * kParts) * kSB + s;
          const bool in = b0 + a * kParts < nblk;
          fu[a][s] = in ? u[(size_t)row * su] : 0.f;
          fv[a][s] = in && v2 ? v2[(size_t)row * sv] : 0.f;
        }
#pragma unroll
      for (int a = 0; a < kAhead; a++) {
        if (b0 + a * kParts >= nblk) break;
        float p = 0.f;
#pragma unroll
        for (int s = 0; s < kSB; s++) p = v2 ? __fmaf_rn(fu[a][s], fv[a][s], p) : p + fu[a][s];
        acc += p;
      }
    }
  red[r][t] = acc;
  __syncthreads();
  if (r == 0 && par >= 0) {
    float gi = 0.f;
#pragma unroll
    for (int q = 0; q < kParts; q++) gi += red[q][t];
    grad[par] = gi;
    if (update) adam_update(L, par, gi, P, WT, m, v, lr, bc1, bc2);
  }
}

__global__ void __launch_bounds__(256) k_mlp_adam(MlpLayout L, const float* __restrict__ grad, float* P, float* WT,
                                                  float* m, float* v, float lr, float bc1, float bc2)
{
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < L.total) adam_update(L, p, grad[p], P, WT, m, v, lr, bc1, bc2);
}

__global__ void k_features(const float* __restrict__ ypr, int n, float* __restrict__ x)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float y = ypr[(size_t)i * 3 + 0], p = ypr[(size_t)i * 3 + 1];
  float4 f;
  sincosf(y, &f.x, &f.y);
  sincosf(p, &f.z, &f.w);
  reinterpret_cast<float4*>(x)[i] = f;
}

#define MLP_TRY(call)                       \
  do {                                      \
    const cudaError_t e_ = (call);          \
    if (e_ != cudaSuccess) return e_;       \
  } while (0)

// Opt the two block kernels into their dynamic shared memory (per device, once).
cudaError_t configure()
{
  static bool done[64];
  int dev = 0;
  MLP_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (done[dev]) return cudaSuccess;
  MLP_TRY(cudaFuncSetAttribute(k_mlp_pass, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPassSmem));
  MLP_TRY(cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kForwardSmem));
  done[dev] = true;
  return cudaSuccess;
}

std::vector<float> transposed(const MlpLayout& L, const float* p)
{
  std::vector<float> t(p, p + L.total);
  for (int l = 0; l < kMlpLayers; l++)
    for (int i = 0; i < L.in[l]; i++)
      for (int o = 0; o < L.out[l]; o++) t[L.w[l] + o * L.in[l] + i] = p[L.w[l] + i * L.out[l] + o];
  return t;
}

}  // namespace

cudaError_t mlp_features(const float* ypr, int n, float* x, cudaStream_t s)
{
  if (n <= 0) return cudaSuccess;
  k_features<<<(n + 255) / 256, 256, 0, s>>>(ypr, n, x);
  return cudaGetLastError();
}

MlpLayout::MlpLayout()
{
  const int dims[kMlpLayers + 1] = {kMlpIn, kMlpHidden, kMlpHidden, kMlpHidden, 1};
  int off = 0;
  for (int l = 0; l < kMlpLayers; l++) {
    in[l] = dims[l];
    out[l] = dims[l + 1];
    w[l] = off;
    off += in[l] * out[l];
    b[l] = off;
    off += out[l];
  }
  total = off;
}

Mlp::~Mlp() { free_all(); }

void Mlp::free_all()
{
  if (fit_exec_) { cudaGraphExecDestroy(fit_exec_); fit_exec_ = nullptr; }
  for (float** p : {&params_, &wt_, &grads_, &m_, &v_, &x_, &y_, &loss_, &part_, &part_loss_})
    if (*p) { cudaFree(*p); *p = nullptr; }
  cap_ = 0; n_ = 0; steps_done_ = 0;
}

cudaError_t Mlp::init(unsigned seed, cudaStream_t s)
{
  std::vector<float> h(L.total, 0.f);
  std::mt19937 rng(seed);
  for (int l = 0; l < kMlpLayers; l++) {
    const float r = std::sqrt(6.f / (float)(L.in[l] + L.out[l]));
    std::uniform_real_distribution<float> U(-r, r);
    for (int k = 0; k < L.in[l] * L.out[l]; k++) h[L.w[l] + k] = U(rng);
  }
  if (!params_) {
    MLP_TRY(cudaMalloc(&params_, sizeof(float) * L.total));
    MLP_TRY(cudaMalloc(&wt_, sizeof(float) * L.total));
    MLP_TRY(cudaMalloc(&grads_, sizeof(float) * L.total));
    MLP_TRY(cudaMalloc(&m_, sizeof(float) * L.total));
    MLP_TRY(cudaMalloc(&v_, sizeof(float) * L.total));
    MLP_TRY(cudaMalloc(&loss_, sizeof(float)));
  }
  MLP_TRY(cudaMemsetAsync(grads_, 0, sizeof(float) * L.total, s));
  return set_params(h.data(), s);
}

cudaError_t Mlp::get_params(float* host, cudaStream_t s) const
{
  if (!params_) return cudaErrorInvalidValue;
  MLP_TRY(cudaMemcpyAsync(host, params_, sizeof(float) * L.total, cudaMemcpyDeviceToHost, s));
  return cudaStreamSynchronize(s);
}

cudaError_t Mlp::set_params(const float* host, cudaStream_t s)
{
  if (!params_) return cudaErrorInvalidValue;
  const std::vector<float> t = transposed(L, host);
  MLP_TRY(cudaMemcpyAsync(params_, host, sizeof(float) * L.total, cudaMemcpyHostToDevice, s));
  MLP_TRY(cudaMemcpyAsync(wt_, t.data(), sizeof(float) * L.total, cudaMemcpyHostToDevice, s));
  MLP_TRY(cudaMemsetAsync(m_, 0, sizeof(float) * L.total, s));
  MLP_TRY(cudaMemsetAsync(v_, 0, sizeof(float) * L.total, s));
  steps_done_ = 0;
  return cudaStreamSynchronize(s);
}

cudaError_t Mlp::reserve(int n)
{
  if (n <= cap_) return cudaSuccess;
  for (float** p : {&x_, &y_, &part_, &part_loss_})
    if (*p) { cudaFree(*p); *p = nullptr; }
  cap_ = 0;
  const size_t nblk = ((size_t)n + kSB - 1) / kSB, rows = nblk * kSB;
  MLP_TRY(cudaMalloc(&x_, sizeof(float) * rows * kMlpIn));
  MLP_TRY(cudaMalloc(&y_, sizeof(float) * rows));
  MLP_TRY(cudaMalloc(&part_, sizeof(float) * rows * (6 * kH + 1)));
  MLP_TRY(cudaMalloc(&part_loss_, sizeof(float) * nblk));
  cap_ = n;
  return cudaSuccess;
}

// The features' rows past the last sample (the weight gradients read whole eights).
cudaError_t Mlp::zero_tail(int n, cudaStream_t s)
{
  const size_t rows = ((size_t)n + kSB - 1) / kSB * kSB;
  if (rows == (size_t)n) return cudaSuccess;
  return cudaMemsetAsync(x_ + (size_t)n * kMlpIn, 0, sizeof(float) * (rows - n) * kMlpIn, s);
}

cudaError_t Mlp::set_data(const float* host_x, const float* host_y, int n, cudaStream_t s)
{
  if (!params_ || n <= 0) return cudaErrorInvalidValue;
  MLP_TRY(reserve(n));
  MLP_TRY(cudaMemcpyAsync(x_, host_x, sizeof(float) * n * kMlpIn, cudaMemcpyHostToDevice, s));
  MLP_TRY(cudaMemcpyAsync(y_, host_y, sizeof(float) * n, cudaMemcpyHostToDevice, s));
  MLP_TRY(zero_tail(n, s));
  n_ = n;
  return cudaStreamSynchronize(s);
}

cudaError_t Mlp::set_data_device(const float* dev_x, const float* dev_y, int n, cudaStream_t s)
{
  if (!params_ || n <= 0) return cudaErrorInvalidValue;
  MLP_TRY(reserve(n));
  MLP_TRY(cudaMemcpyAsync(x_, dev_x, sizeof(float) * n * kMlpIn, cudaMemcpyDeviceToDevice, s));
  MLP_TRY(cudaMemcpyAsync(y_, dev_y, sizeof(float) * n, cudaMemcpyDeviceToDevice, s));
  MLP_TRY(zero_tail(n, s));
  n_ = n;
  return cudaSuccess;
}

cudaError_t Mlp::step(float lr, bool update, cudaStream_t s)
{
  const int n = n_;
  if (n <= 0 || !params_) return cudaErrorInvalidValue;
  const int nblk = (n + kSB - 1) / kSB;
  const size_t rows = (size_t)nblk * kSB;
  PassOut O;
  for (int l = 0; l < 3; l++) { O.a[l] = part_ + l * rows * kH; O.d[l] = part_ + (3 + l) * rows * kH; }
  O.d4 = part_ + 6 * rows * kH;
  MLP_TRY(configure());
  k_mlp_pass<<<nblk, kH, kPassSmem, s>>>(L, params_, wt_, x_, y_, n, O, part_loss_);
  MLP_TRY(cudaGetLastError());
  float bc1 = 1.f, bc2 = 1.f;
  if (update) {
    const int t = steps_done_ + 1;
    bc1 = 1.f - std::pow(0.9f, (float)t);
    bc2 = 1.f - std::pow(0.999f, (float)t);
  }
  const int grid = 2 * kTilesPerLayer + (kSmall + kSmallPer - 1) / kSmallPer + 1;
  k_mlp_update<<<grid, kUpdateThreads, 0, s>>>(L, x_, O, part_loss_, nblk, grads_, loss_, update ? 1 : 0, params_, wt_,
                                            m_, v_, lr, bc1, bc2);
  MLP_TRY(cudaGetLastError());
  if (update) steps_done_++;
  return cudaSuccess;
}

cudaError_t Mlp::grad(cudaStream_t s) { return step(0.f, false, s); }

cudaError_t Mlp::read_grad(float* host, float* loss, cudaStream_t s)
{
  if (host) MLP_TRY(cudaMemcpyAsync(host, grads_, sizeof(float) * L.total, cudaMemcpyDeviceToHost, s));
  if (loss) MLP_TRY(cudaMemcpyAsync(loss, loss_, sizeof(float), cudaMemcpyDeviceToHost, s));
  return cudaStreamSynchronize(s);
}

cudaError_t Mlp::adam(float lr, cudaStream_t s)
{
  if (!params_) return cudaErrorInvalidValue;
  const int t = steps_done_ + 1;
  const float bc1 = 1.f - std::pow(0.9f, (float)t), bc2 = 1.f - std::pow(0.999f, (float)t);
  k_mlp_adam<<<(L.total + 255) / 256, 256, 0, s>>>(L, grads_, params_, wt_, m_, v_, lr, bc1, bc2);
  MLP_TRY(cudaGetLastError());
  steps_done_++;
  return cudaSuccess;
}

cudaError_t Mlp::fit(int steps, float lr, cudaStream_t s, float* final_loss)
{
  if (n_ <= 0 || steps < 0) return cudaErrorInvalidValue;
  if (steps > 0) {
    // Adam's bias corrections are launch arguments, so a graph is tied to
    // the step it starts from as well as to the shapes and buffers
    const bool reuse = fit_exec_ && fit_n_ == n_ && fit_steps_ == steps && fit_lr_ == lr &&
                       fit_start_ == steps_done_ && fit_bufs_[0] == x_ && fit_bufs_[1] == y_ && fit_bufs_[2] == part_;
    if (!reuse) {
      if (fit_exec_) { cudaGraphExecDestroy(fit_exec_); fit_exec_ = nullptr; }
      MLP_TRY(configure());
      const int start = steps_done_;
      MLP_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
      cudaError_t e = cudaSuccess;
      for (int i = 0; i < steps && e == cudaSuccess; i++) e = step(lr, true, s);
      cudaGraph_t g = nullptr;
      const cudaError_t e2 = cudaStreamEndCapture(s, &g);
      steps_done_ = start;
      if (e == cudaSuccess) e = e2;
      if (e == cudaSuccess) e = cudaGraphInstantiate(&fit_exec_, g, 0);
      if (g) cudaGraphDestroy(g);
      if (e != cudaSuccess) { fit_exec_ = nullptr; return e; }
      fit_n_ = n_; fit_steps_ = steps; fit_lr_ = lr; fit_start_ = start;
      fit_bufs_[0] = x_; fit_bufs_[1] = y_; fit_bufs_[2] = part_;
    }
    MLP_TRY(cudaGraphLaunch(fit_exec_, s));
    steps_done_ += steps;
  }
  if (final_loss) {
    MLP_TRY(cudaMemcpyAsync(final_loss, loss_, sizeof(float), cudaMemcpyDeviceToHost, s));
    MLP_TRY(cudaStreamSynchronize(s));
  }
  return cudaSuccess;
}

cudaError_t Mlp::predict_device(const float* dev_x, int n, float* dev_out, cudaStream_t s)
{
  if (!params_ || n <= 0) return cudaErrorInvalidValue;
  MLP_TRY(configure());
  int dev = 0, sms = 0;
  MLP_TRY(cudaGetDevice(&dev));
  MLP_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int eights = n / 8 + (n % 8 != 0);
  k_mlp_forward<<<eights < sms ? eights : sms, 256, kForwardSmem, s>>>(L, params_, dev_x, n, dev_out);
  return cudaGetLastError();
}

}  // namespace tomo
