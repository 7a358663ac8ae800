// FP32 convolution kernels of the preconditioner network (3x3x3 taps on the
// 10^3 region, zero padding; layouts: precond.cu), forward and backward.
//
// Bound: FP32 multiply-adds.  A 32 -> 32 convolution is 27 x 1024 x 1000 of them
// per sample (at 256 samples 7.1 G: 0.19 ms at the chip's 37 T/s), so every
// kernel here is a register-tiled matrix product fed from shared memory by
// conflict-free 16-byte loads, its tile sized so that the multiply-adds of a
// load take at least as long as the load.
// CTAs are persistent (one per SM) over (sample, slab of planes) items, so the
// weights are staged once; the slab height follows from the batch (conv_slab).
// Weight gradients leave the CTAs as partial sums that a second kernel adds in
// a fixed order (no atomics).
//
// 256 samples, us per launch, before (one output at a time per thread; weight
// gradient of one tap per CTA) and now:
//   conv 32 -> 32: 885, 335    weight gradient 32 x 32: 1821, 286
//   conv 3 -> 32:   84, 66     weight gradient 3 x 32:   550, 76
//   conv 32 -> 3:  102, 47     weight gradient 32 x 3:   496, 35
#pragma once

#include "common.cuh"
#include "deposit_core.cuh"
#include "ptx.cuh"

namespace {

constexpr int kPlane = 100;        // voxels of a plane of the region
constexpr int kConvThreads = 256;
constexpr int kTapWarps = 27;      // k_wgrad3: one warp per tap
constexpr int kWgThreads = 32 * kTapWarps;
constexpr int kMaxParts = 304;     // CTAs whose partial weight gradients the workspace holds

__device__ __forceinline__ float sum2(unsigned long long v) {
  const float2 f = *reinterpret_cast<const float2*>(&v);
  return f.x + f.y;
}

// n floats (a multiple of 4) into shared memory, both sides 16-byte aligned
template <int NT>
__device__ __forceinline__ void stage_copy(float* dst, const float* __restrict__ src, int n) {
  for (int t = threadIdx.x; t < n / 4; t += NT) cp_async16(dst + 4 * t, src + 4 * t);
}
__device__ __forceinline__ void stage_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// The planes [z0, z0 + np) of a sample with C channels into rows of RS floats
// per voxel (RS >= C; 3 channels: RS = 4, the fourth 0); planes outside the
// region are left out (nothing reads them).
template <int C, int RS, int NT>
__device__ __forceinline__ void stage_planes(float* s, const float* __restrict__ smp, int z0, int np) {
  const int a = max(z0, 0), b = min(z0 + np, 10);
  const int first = (a - z0) * kPlane, nv = (b - a) * kPlane;
  const float* src = smp + (size_t)a * kPlane * C;
  if constexpr (C == 32) {
    for (int t = threadIdx.x; t < nv * 8; t += NT) cp_async16(s + (first + t / 8) * RS + 4 * (t % 8), src + 4 * t);
  } else {
    for (int v = threadIdx.x; v < nv; v += NT)
      *reinterpret_cast<float4*>(s + (first + v) * RS) = make_float4(src[3 * v], src[3 * v + 1], src[3 * v + 2], 0.f);
  }
}

// ---------------------------------------------------------------------------
// out[s][v][o] = sum_t sum_c W[t][c][o] in[s][v + off_t][c], 32 outputs.  FLIP:
// the weights of the input gradient, W'[t][c][o] = W[26 - t][o][c].
// A thread owns V voxels x 8 outputs; 4 channels cost it V + 8 16-byte shared
// loads and 32 V multiply-adds.  Shared memory delivers one such load per warp
// in 4 cycles and the FP32 pipes take 4 multiply-adds of a warp per cycle, so V
// = 8 balances the two (V = 4 with packed accumulators over even and odd
// channels was bound by the loads: 510 us).  A tap outside the region reads a
// row of zeros.
template <int CIN, int P>
struct ConvShape {
  static constexpr int CP = (CIN + 3) & ~3;            // channels, padded to 4
  static constexpr int RS = CP == 32 ? 36 : CP;        // floats per staged voxel
  static constexpr int V = P == 5 ? 8 : (P == 2 ? 4 : 2);
  static constexpr int NG = (P * kPlane + V - 1) / V;  // voxel groups
  static constexpr int kW = 27 * CP * 32;              // weight floats
  static constexpr size_t kSmem = sizeof(float) * (kW + (P + 2) * kPlane * RS + CP);
};

template <int CIN, bool FLIP, int P>
__global__ void __launch_bounds__(kConvThreads, 1) k_conv32(int items, const float* __restrict__ in,
                                                            const float* __restrict__ W,
                                                            float* __restrict__ out) {
  using Sh = ConvShape<CIN, P>;
  constexpr int CP = Sh::CP, RS = Sh::RS, V = Sh::V, NG = Sh::NG;
  static_assert(4 * NG <= kConvThreads, "a thread per voxel group and 8 outputs");
  extern __shared__ __align__(16) float s_f[];
  float* s_w = s_f;                       // [t][c][o]
  float* s_in = s_w + Sh::kW;             // (P + 2) planes
  float* s_zero = s_in + (P + 2) * kPlane * RS;
  for (int q = threadIdx.x; q < Sh::kW; q += kConvThreads) {
    const int t = q / (CP * 32), c = (q / 32) % CP, o = q % 32;
    s_w[q] = c < CIN ? (FLIP ? W[((26 - t) * 32 + o) * CIN + c] : W[(t * CIN + c) * 32 + o]) : 0.f;
  }
  if (threadIdx.x < CP) s_zero[threadIdx.x] = 0.f;
  const int og = threadIdx.x & 3, vg = threadIdx.x >> 2;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int s = item / (10 / P), z0 = (item % (10 / P)) * P;
    __syncthreads();  // the last item's reads are done
    stage_planes<CIN, RS, kConvThreads>(s_in, in + (size_t)s * 1000 * CIN, z0 - 1, P + 2);
    stage_wait();
    if (vg >= NG) continue;
    float acc[V][8];
    unsigned ok[V];    // taps inside the region
#pragma unroll
    for (int q = 0; q < V; q++) {
      const int v = vg + q * NG, i = v % 10, j = (v / 10) % 10, z = z0 + v / kPlane;
      const unsigned mx = (i > 0 ? 1u : 0u) | 2u | (i < 9 ? 4u : 0u);
      const unsigned my = (j > 0 ? 7u : 0u) | 0x38u | (j < 9 ? 0x1C0u : 0u);
      const unsigned pl = (mx | mx << 3 | mx << 6) & my;
      ok[q] = v < P * kPlane ? (z > 0 ? pl : 0u) | pl << 9 | (z < 9 ? pl << 18 : 0u) : 0u;
#pragma unroll
      for (int o = 0; o < 8; o++) acc[q][o] = 0.f;
    }
    for (int t = 0; t < 27; t++) {
      // staged voxel of the thread's first voxel at this tap (the centre tap of
      // voxel v is staged voxel v + kPlane)
      const int at = vg + kPlane + t % 3 + 10 * ((t / 3) % 3) + kPlane * (t / 9) - 111;
      const float* src[V];
#pragma unroll
      for (int q = 0; q < V; q++) src[q] = (ok[q] >> t) & 1u ? s_in + (at + q * NG) * RS : s_zero;
      const float* w = s_w + t * CP * 32 + og * 8;
#pragma unroll 2
      for (int c = 0; c < CP; c += 4) {
        float ww[4][8];
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
          for (int o = 0; o < 8; o += 4) {
            const float4 f = *reinterpret_cast<const float4*>(w + (c + k) * 32 + o);
            ww[k][o] = f.x; ww[k][o + 1] = f.y; ww[k][o + 2] = f.z; ww[k][o + 3] = f.w;
          }
#pragma unroll
        for (int q = 0; q < V; q++) {
          const float4 f = *reinterpret_cast<const float4*>(src[q] + c);
          const float a[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
          for (int k = 0; k < 4; k++)
#pragma unroll
            for (int o = 0; o < 8; o++) acc[q][o] = fmaf(a[k], ww[k][o], acc[q][o]);
        }
      }
    }
    float* outs = out + ((size_t)s * 1000 + z0 * kPlane) * 32 + og * 8;
#pragma unroll
    for (int q = 0; q < V; q++) {
      const int v = vg + q * NG;
      if (v >= P * kPlane) continue;
      float4* d = reinterpret_cast<float4*>(outs + (size_t)v * 32);
      d[0] = make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
      d[1] = make_float4(acc[q][4], acc[q][5], acc[q][6], acc[q][7]);
    }
  }
}

// 32 -> 3 on the owned voxels (the others are not written): a thread per voxel
// of a slab of 4 owned planes, 3 outputs.
constexpr int kOutThreads = 256;
constexpr int kOutRS = 36;
constexpr size_t kOutSmem = sizeof(float) * (27 * 32 * 4 + 6 * kPlane * kOutRS);

__global__ void __launch_bounds__(kOutThreads, 2) k_conv_out(int items, const float* __restrict__ in,
                                                             const float* __restrict__ W,
                                                             float* __restrict__ out) {
  extern __shared__ __align__(16) float s_f[];
  float* s_w = s_f;                  // [t][c / 2][o (3, padded to 4)][c & 1]
  float* s_in = s_w + 27 * 32 * 4;   // 6 planes
  for (int q = threadIdx.x; q < 27 * 32 * 4; q += kOutThreads) {
    const int t = q / 128, r = q % 128, c = 2 * (r / 8) + (r & 1), o = (r / 2) % 4;
    s_w[q] = o < 3 ? W[(t * 32 + c) * 3 + o] : 0.f;
  }
  const int i = 1 + (threadIdx.x & 7), j = 1 + ((threadIdx.x >> 3) & 7), l = threadIdx.x >> 6;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int s = item >> 1, z0 = 1 + 4 * (item & 1);
    __syncthreads();
    stage_planes<32, kOutRS, kOutThreads>(s_in, in + (size_t)s * 32000, z0 - 1, 6);
    stage_wait();
    unsigned long long acc[3] = {0ull, 0ull, 0ull};
    const float* c0 = s_in + (l * kPlane + (j - 1) * 10 + i - 1) * kOutRS;
    for (int t = 0; t < 27; t++) {
      const float* a = c0 + (t % 3 + 10 * ((t / 3) % 3) + kPlane * (t / 9)) * kOutRS;
      const float* w = s_w + t * 128;
#pragma unroll
      for (int c = 0; c < 32; c += 4) {
        const ulonglong2 av = *reinterpret_cast<const ulonglong2*>(a + c);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const ulonglong2 w01 = *reinterpret_cast<const ulonglong2*>(w + (c / 2 + h) * 8);
          const unsigned long long w2 = *reinterpret_cast<const unsigned long long*>(w + (c / 2 + h) * 8 + 4);
          const unsigned long long x = h ? av.y : av.x;
          ffma2(acc[0], x, w01.x);
          ffma2(acc[1], x, w01.y);
          ffma2(acc[2], x, w2);
        }
      }
    }
    float* o = out + ((size_t)s * 1000 + (z0 + l) * kPlane + j * 10 + i) * 3;
#pragma unroll
    for (int q = 0; q < 3; q++) o[q] = sum2(acc[q]);
  }
}

// ---------------------------------------------------------------------------
// dW[t][c][o] = sum_{s,v} dout[s][v][o] in[s][v + off_t][c], 32 x 32.  A warp
// owns the three taps of one (dy, dz) and one half of the outputs; its lane 4
// channels x 4 outputs of each.  Along a row the inputs of the three taps are a
// sliding window in registers, so a voxel costs two 16-byte loads (4 channels of
// the voxel entering the window, 4 outputs of dout) and 48 multiply-adds; one
// tap per warp with a 4 x 8 tile took three loads for 32 and was bound by them
// (271 us).  Off the row's ends the window holds zeros.  Items are half samples
// (5 planes of dout, 7 of in staged).
constexpr int kWg32Threads = 32 * 18;
constexpr size_t kWg32Smem = sizeof(float) * 12 * kPlane * 32;

__global__ void __launch_bounds__(kWg32Threads, 1) k_wgrad32(int items, const float* __restrict__ dout,
                                                             const float* __restrict__ in,
                                                             float* __restrict__ part) {
  extern __shared__ __align__(16) float s_f[];
  float* s_d = s_f;                      // 5 planes
  float* s_in = s_f + 5 * kPlane * 32;   // 7 planes
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = wid >> 1;
  const int dy = g % 3 - 1, dz = g / 3 - 1;
  const int cq = 4 * (lane & 7), oq = 16 * (wid & 1) + 4 * (lane >> 3);
  const int j0 = max(0, -dy), j1 = min(10, 10 - dy);
  float acc[3][4][4];
#pragma unroll
  for (int t = 0; t < 3; t++)
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int o = 0; o < 4; o++) acc[t][c][o] = 0.f;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int s = item >> 1, z0 = 5 * (item & 1);
    __syncthreads();
    stage_planes<32, 32, kWg32Threads>(s_d, dout + (size_t)s * 32000, z0, 5);
    stage_planes<32, 32, kWg32Threads>(s_in, in + (size_t)s * 32000, z0 - 1, 7);
    stage_wait();
    for (int l = 0; l < 5; l++) {
      const int z = z0 + l + dz;
      if (z < 0 || z > 9) continue;
      for (int j = j0; j < j1; j++) {
        const float* d = s_d + (l * kPlane + j * 10) * 32 + oq;
        const float* a = s_in + ((l + 1 + dz) * kPlane + (j + dy) * 10) * 32 + cq;
        float4 win[3];
        win[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        win[1] = *reinterpret_cast<const float4*>(a);
#pragma unroll
        for (int i = 0; i < 10; i++) {
          win[2] = i < 9 ? *reinterpret_cast<const float4*>(a + (i + 1) * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float4 f = *reinterpret_cast<const float4*>(d + i * 32);
          const float dd[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
          for (int t = 0; t < 3; t++) {
            const float aa[4] = {win[t].x, win[t].y, win[t].z, win[t].w};
#pragma unroll
            for (int c = 0; c < 4; c++)
#pragma unroll
              for (int o = 0; o < 4; o++) acc[t][c][o] = fmaf(aa[c], dd[o], acc[t][c][o]);
          }
          win[0] = win[1];
          win[1] = win[2];
        }
      }
    }
  }
  float* p = part + (size_t)blockIdx.x * 27 * 1024 + 3 * g * 1024 + oq;
#pragma unroll
  for (int t = 0; t < 3; t++)
#pragma unroll
    for (int c = 0; c < 4; c++)
      *reinterpret_cast<float4*>(p + t * 1024 + (cq + c) * 32) =
          make_float4(acc[t][c][0], acc[t][c][1], acc[t][c][2], acc[t][c][3]);
}

// The weight gradients with 3 channels on one side.  A lane owns 4 of the 32
// channels x all 3 of the other side for a quarter of the voxels of a row; the
// four quarters are added at the end.
//   IN3: dW[t][3][32], in has 3 channels (first layer)
//   else dW[t][32][3], dout has 3 channels and is zero off the owned voxels
constexpr size_t kWg3Smem = sizeof(float) * 7 * kPlane * 36;

template <bool IN3>
__global__ void __launch_bounds__(kWgThreads, 1) k_wgrad3(int items, const float* __restrict__ dout,
                                                          const float* __restrict__ in,
                                                          float* __restrict__ part) {
  extern __shared__ __align__(16) float s_f[];
  float* s_wide = s_f;                     // 32 channels: dout (IN3) or in
  float* s_thin = s_f + 7 * kPlane * 32;   // 3 channels, padded to 4
  const int lane = threadIdx.x & 31, t = threadIdx.x >> 5;
  const int dx = t % 3 - 1, dy = (t / 3) % 3 - 1, dz = t / 9 - 1;
  const int wq = 4 * (lane & 7), vs = lane >> 3;
  const int i0 = IN3 ? max(0, -dx) : 1, i1 = IN3 ? min(10, 10 - dx) : 9;
  const int j0 = IN3 ? max(0, -dy) : 1, j1 = IN3 ? min(10, 10 - dy) : 9;
  float acc[3][4];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) acc[a][b] = 0.f;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    // planes of dout: 5 of the region (IN3), or 4 owned ones
    const int s = item >> 1, h = item & 1, np = IN3 ? 5 : 4, z0 = IN3 ? 5 * h : 1 + 4 * h;
    __syncthreads();
    if (IN3) {
      stage_planes<32, 32, kWgThreads>(s_wide, dout + (size_t)s * 32000, z0, 5);
      stage_planes<3, 4, kWgThreads>(s_thin, in + (size_t)s * 3000, z0 - 1, 7);
    } else {
      stage_planes<32, 32, kWgThreads>(s_wide, in + (size_t)s * 32000, z0 - 1, 6);
      stage_planes<3, 4, kWgThreads>(s_thin, dout + (size_t)s * 3000, z0, 4);
    }
    stage_wait();
    for (int l = 0; l < np; l++) {
      const int z = z0 + l + dz;
      if (z < 0 || z > 9) continue;
      for (int j = j0; j < j1; j++) {
        const int vd = l * kPlane + j * 10, vi = (l + 1 + dz) * kPlane + (j + dy) * 10 + dx;
        for (int i = i0 + vs; i < i1; i += 4) {
          const float4 w = *reinterpret_cast<const float4*>(s_wide + (IN3 ? vd + i : vi + i) * 32 + wq);
          const float4 n = *reinterpret_cast<const float4*>(s_thin + (IN3 ? vi + i : vd + i) * 4);
          const float nn[3] = {n.x, n.y, n.z}, ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) acc[a][b] = fmaf(nn[a], ww[b], acc[a][b]);
        }
      }
    }
  }
  float* p = part + (size_t)blockIdx.x * 27 * 96 + t * 96;
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) {
      float v = acc[a][b];
      v += __shfl_xor_sync(0xffffffffu, v, 8);
      v += __shfl_xor_sync(0xffffffffu, v, 16);
      if (vs == 0) p[IN3 ? a * 32 + wq + b : (wq + b) * 3 + a] = v;
    }
}

// g[q] += the sum of the CTAs' partials as an FP32 pair, 4 threads per element
constexpr int kAddThreads = 256;
__global__ void __launch_bounds__(kAddThreads) k_add_parts(int n, int parts, const float* __restrict__ part,
                                                           float* __restrict__ g) {
  __shared__ FF s_sum[4][kAddThreads / 4];
  const int l = threadIdx.x % (kAddThreads / 4), r = threadIdx.x / (kAddThreads / 4);
  const int q = blockIdx.x * (kAddThreads / 4) + l;
  FF s{0.f, 0.f};
  if (q < n) {
#pragma unroll 8
    for (int b = r; b < parts; b += 4) ff_acc(s, part[(size_t)b * n + q], 0.f);
  }
  s_sum[r][l] = s;
  __syncthreads();
  if (r == 0 && q < n) {
#pragma unroll
    for (int k = 1; k < 4; k++) ff_acc(s, s_sum[k][l].s, s_sum[k][l].q);
    g[q] += s.s + s.q;
  }
}

// Slab height of the 32-output convolutions: 5, 2 or 1 planes per item.  Taller
// slabs reuse a weight load for more voxels (relative rates 1, 0.7, 0.45 of the
// tiles of 4, 2 and 1 voxels per thread), shorter ones give a small batch more
// items than one wave of SMs: the height with the least items-per-SM x planes /
// rate.
int conv_slab(int S, int sms) {
  const int p[3] = {5, 2, 1};
  const double rate[3] = {1.0, 0.7, 0.45};
  int best = 0;
  double least = 1e30;
  for (int q = 0; q < 3; q++) {
    const int items = S * (10 / p[q]);
    const double cost = ((items + sms - 1) / sms) * p[q] / rate[q];
    if (cost < least) {
      least = cost;
      best = q;
    }
  }
  return p[best];
}

template <int CIN, bool FLIP, int P>
cudaError_t conv32_p(cudaStream_t st, int S, int sms, int dev, const float* in, const float* W, float* out) {
  constexpr size_t sm = ConvShape<CIN, P>::kSmem;
  static unsigned long long ready = 0;  // per device
  if (!((ready >> dev) & 1ull)) {
    cudaError_t e = cudaFuncSetAttribute(k_conv32<CIN, FLIP, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    ready |= 1ull << dev;
  }
  const int items = S * (10 / P);
  k_conv32<CIN, FLIP, P><<<std::min(items, sms), kConvThreads, sm, st>>>(items, in, W, out);
  return cudaGetLastError();
}

template <int CIN, bool FLIP>
cudaError_t conv32(cudaStream_t st, int S, int sms, int dev, const float* in, const float* W, float* out) {
  switch (conv_slab(S, sms)) {
    case 5: return conv32_p<CIN, FLIP, 5>(st, S, sms, dev, in, W, out);
    case 2: return conv32_p<CIN, FLIP, 2>(st, S, sms, dev, in, W, out);
    default: return conv32_p<CIN, FLIP, 1>(st, S, sms, dev, in, W, out);
  }
}

cudaError_t conv_out(cudaStream_t st, int S, int sms, int dev, const float* in, const float* W, float* out) {
  static unsigned long long ready = 0;
  if (!((ready >> dev) & 1ull)) {
    cudaError_t e = cudaFuncSetAttribute(k_conv_out, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOutSmem);
    if (e != cudaSuccess) return e;
    ready |= 1ull << dev;
  }
  k_conv_out<<<std::min(2 * S, 2 * sms), kOutThreads, kOutSmem, st>>>(2 * S, in, W, out);
  return cudaGetLastError();
}

// kind 0: 32 x 32, 1: 3 x 32 (first layer), 2: 32 x 3 (last layer); g += the gradient
cudaError_t wgrad(cudaStream_t st, int S, int sms, int dev, int kind, const float* dout, const float* in,
                  float* part, float* g) {
  static unsigned long long ready = 0;
  if (!((ready >> dev) & 1ull)) {
    cudaError_t e = cudaFuncSetAttribute(k_wgrad32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWg32Smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_wgrad3<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWg3Smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_wgrad3<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWg3Smem);
    if (e != cudaSuccess) return e;
    ready |= 1ull << dev;
  }
  const int items = 2 * S, grid = std::min({items, sms, kMaxParts});
  const int n = kind == 0 ? 27 * 1024 : 27 * 96;
  if (kind == 0)
    k_wgrad32<<<grid, kWg32Threads, kWg32Smem, st>>>(items, dout, in, part);
  else if (kind == 1)
    k_wgrad3<true><<<grid, kWgThreads, kWg3Smem, st>>>(items, dout, in, part);
  else
    k_wgrad3<false><<<grid, kWgThreads, kWg3Smem, st>>>(items, dout, in, part);
  k_add_parts<<<(4 * n + kAddThreads - 1) / kAddThreads, kAddThreads, 0, st>>>(n, grid, part, g);
  return cudaGetLastError();
}

}  // namespace
