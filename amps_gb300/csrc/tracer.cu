// Batched relativistic test-particle tracing in a dipole + uniform field.
//
// Step: BorisStep of srcEarth/gridless/GridlessParticleMovers.cpp:781-801
// (half drift, momentum rotation with t = q dt B/(2 gamma m), s = 2t/(1+t^2),
// half drift with the new gamma); field Dipole::GetB_Tesla
// (srcEarth/gridless/DipoleInterface.h:99-126) plus a uniform field; step size
// dt = min(dt_max, dphi_max / omega_g) (CutoffRigidityGridless.cpp:1190-1197);
// a particle stops at r < r_in, r > r_out or after max_steps.
//
// One persistent kernel: every lane owns one particle; when lanes finish, the
// warp refills them from a global queue with one atomic per warp, and when the
// queue is empty the CTA packs its particles into fewer warps, so uneven
// lifetimes do not idle lanes.  State is carried in
// normalised units (x / R_E, p / (m c), t c / R_E, B / B_eq) so the FP32
// variant keeps full range; SI is converted at the boundary (k_trace_in / _out).  The FP32
// variant accumulates positions with compensated (Kahan) sums: a half drift is
// ~1e-2 of |x|, so plain FP32 sums would lose ~1e-5 of every displacement.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "ptx.cuh"

namespace {

constexpr double kC = 299792458.0;
constexpr int kRefill = 16;  // steps between refill checks

template <class T>
struct TraceArgs {
  T* x; T* y; T* z; T* px; T* py; T* pz;
  int32_t* status;
  int64_t* steps;
  long long n;
  unsigned long long* queue;     // next particle index
  unsigned long long* total;     // total steps
  unsigned long long* flags;     // [0] iteration cap reached
  T kq;                          // q B_eq R_E / (m c) (signed)
  T ext[3];                      // uniform field / B_eq
  T r_in2, r_out2;
  T dphi, dt_max;
  long long max_steps;
  long long iter_cap;
};

template <class T>
__device__ __forceinline__ T rsq(T v);
template <>
__device__ __forceinline__ float rsq<float>(float v) { return rsqrtf(v); }
template <>
__device__ __forceinline__ double rsq<double>(double v) { return rsqrt(v); }

// Every product and sum of a step is written with these, so where a product is
// rounded on its own and where it is fused is fixed here and not chosen by the
// compiler anew for every change of the code around it: near the cutoff
// trajectories part exponentially, and one rounding decides step counts.
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float mad(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double mad(double a, double b, double c) { return __fma_rn(a, b, c); }

template <class T>
__device__ __forceinline__ T norm2(T x, T y, T z) {
  return mad(z, z, mad(y, y, mul(x, x)));
}
// a b - c d
template <class T>
__device__ __forceinline__ T minor(T a, T b, T c, T d) {
  return mad(a, b, -mul(c, d));
}

template <class T>
__device__ __forceinline__ void field(const TraceArgs<T>& a, T r2, T x, T y, T z, T& bx, T& by, T& bz) {
  const T ir = rsq<T>(r2);
  const T ir2 = mul(ir, ir);
  const T ir3 = mul(ir2, ir);
  const T ir5 = mul(ir3, ir2);
  // moment along +z with unit strength (B_eq R_E^3 in these units): m . r = z
  bx = mad(mul(mul(T(3), x), z), ir5, a.ext[0]);
  by = mad(mul(mul(T(3), y), z), ir5, a.ext[1]);
  bz = add(mad(mul(mul(T(3), z), z), ir5, -ir3), a.ext[2]);
}

// x += h ig with a running compensation c (FP32 only; FP64 sums are plain)
template <class T>
__device__ __forceinline__ void comp_add(T& x, T& c, T h, T ig) {
  if constexpr (sizeof(T) == 4) {
    const T yv = mad(h, ig, -c);
    const T t = add(x, yv);
    c = add(add(t, -x), -yv);
    x = t;
  } else {
    x = mad(h, ig, x);
  }
}

// Threads per CTA and CTAs per SM.  FP64: the narrow pipe (2 lanes per clock and
// SM) is saturated by 8 warps, and one CTA holds the whole SM's particles for
// the compaction below; FP32 needs the warps to hide latency.
template <class T>
struct TraceShape {
  static constexpr int kThreads = sizeof(T) == 8 ? 256 : 512;
  static constexpr int kPerSM = sizeof(T) == 8 ? 1 : 3;
};

// Lane use bounds this kernel: a step costs a warp the same whether 1 or 32 of
// its lanes hold a particle, and lifetimes differ by orders of magnitude.
//   - Start: particle 32 (wid * CTAs + CTA) + lane, so a batch that does not fill
//     the chip is spread over all SMs; the queue serves the rest.
//   - While the queue lasts, idle lanes refill (one atomic per warp).
//   - Then the CTA compacts: whenever its particles fit fewer warps than are
//     running, their states move through shared memory into the first ones
//     (a lane left idle after a refill means that the queue is exhausted).
// gamma, 1/gamma and r^2 at the end of a step are the next step's: they are
// carried instead of formed again (the same expressions of the same values).
// Against the form without compaction, spread start and carrying: 262,144
// protons x 2000 steps FP32 1.68 instead of 2.78 ms; 20,000 x 500 FP64 2.24
// instead of 7.13 ms (79 of 152 SMs had work); 100,000 x 2000 FP64 22 instead of
// 76 ms; 10^6 x 10^5 FP32 104 instead of 154 ms.
template <class T>
__global__ void __launch_bounds__(TraceShape<T>::kThreads, TraceShape<T>::kPerSM) k_trace(TraceArgs<T> a) {
  constexpr int NT = TraceShape<T>::kThreads, NW = NT / 32;
  constexpr int kState = sizeof(T) == 4 ? 9 : 6;  // position, momentum (, FP32: compensation)
  __shared__ T s_v[kState][NT];
  __shared__ long long s_st[NT], s_idx[NT];
  __shared__ int s_cnt[NW];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  long long idx = -1;
  T x = 0, y = 0, z = 0, px = 0, py = 0, pz = 0;
  T cx = 0, cy = 0, cz = 0;  // position compensation (FP32)
  T r2 = 1, g = 1, ig = 1;   // r^2, gamma, 1 / gamma of the state
  long long st = 0;
  unsigned long long my_total = 0;
  bool queue_done = false;
  auto derive = [&]() {
    r2 = norm2(x, y, z);
    g = sqrt(mad(pz, pz, mad(py, py, mad(px, px, T(1)))));
    ig = T(1) / g;
  };
  auto take = [&](unsigned long long mine) {
    if (mine >= (unsigned long long)a.n) return;
    idx = (long long)mine;
    x = a.x[idx]; y = a.y[idx]; z = a.z[idx];
    px = a.px[idx]; py = a.py[idx]; pz = a.pz[idx];
    cx = cy = cz = T(0);
    st = 0;
    derive();
  };
  take(32ull * ((unsigned long long)wid * gridDim.x + blockIdx.x) + lane);  // the queue starts behind these
  int warps = NW;  // warps that hold particles (CTA-uniform)
  for (long long iter = 0;; iter++) {
    // CTA-uniform: iter counts alike in every thread
    if (iter >= a.iter_cap) {
      if (threadIdx.x == 0) atomicAdd(a.flags, 1ull);
      break;
    }
    // refill finished lanes (one atomic per warp)
    const bool need = idx < 0 && wid < warps;
    const unsigned needm = __ballot_sync(0xffffffffu, need);
    if (needm && !queue_done) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(a.queue, (unsigned long long)__popc(needm));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= (unsigned long long)a.n) queue_done = true;
      if (need) take(base + __popc(needm & lanemask_lt()));
    }
    const unsigned livem = __ballot_sync(0xffffffffu, idx >= 0);
    if (lane == 0) s_cnt[wid] = __popc(livem);
    const int live = __syncthreads_count(idx >= 0);
    if (live == 0) break;
    if ((live + 31) / 32 < warps) {
      int pos = __popc(livem & lanemask_lt());
      for (int w = 0; w < wid; w++) pos += s_cnt[w];
      if (idx >= 0) {
        s_v[0][pos] = x; s_v[1][pos] = y; s_v[2][pos] = z;
        s_v[3][pos] = px; s_v[4][pos] = py; s_v[5][pos] = pz;
        if constexpr (kState == 9) { s_v[6][pos] = cx; s_v[7][pos] = cy; s_v[8][pos] = cz; }
        s_st[pos] = st;
        s_idx[pos] = idx;
      }
      __syncthreads();
      const int t = threadIdx.x;
      idx = -1;
      if (t < live) {
        x = s_v[0][t]; y = s_v[1][t]; z = s_v[2][t];
        px = s_v[3][t]; py = s_v[4][t]; pz = s_v[5][t];
        if constexpr (kState == 9) { cx = s_v[6][t]; cy = s_v[7][t]; cz = s_v[8][t]; }
        st = s_st[t];
        idx = s_idx[t];
        derive();
      }
      warps = (live + 31) / 32;
    }
    __syncthreads();  // s_cnt and the states are rewritten
    int status = -1;
    if (idx >= 0) {
#pragma unroll 1
      for (int k = 0; k < kRefill; k++) {
        T bx, by, bz;
        field(a, r2, x, y, z, bx, by, bz);
        const T bm = sqrt(norm2(by, bx, bz));
        T dt = a.dt_max;
        const T om = mul(fabs(a.kq), bm) / g;
        if (om > T(0)) {
          const T lim = a.dphi / om;
          if (lim < dt) dt = lim;
        }
        const T h = mul(T(0.5), dt);
        comp_add(x, cx, mul(h, px), ig);
        comp_add(y, cy, mul(h, py), ig);
        comp_add(z, cz, mul(h, pz), ig);
        const T f = mul(mul(mul(a.kq, dt), T(0.5)), ig);
        const T tx = mul(f, bx), ty = mul(f, by), tz = mul(f, bz);
        const T sfac = T(2) / mad(tz, tz, mad(ty, ty, mad(tx, tx, T(1))));
        const T qx = add(px, minor(py, tz, pz, ty));
        const T qy = add(py, minor(pz, tx, px, tz));
        const T qz = add(pz, minor(px, ty, py, tx));
        px = mad(sfac, minor(qy, tz, qz, ty), px);
        py = mad(sfac, minor(qz, tx, qx, tz), py);
        pz = mad(sfac, minor(qx, ty, qy, tx), pz);
        g = sqrt(mad(pz, pz, mad(py, py, mad(px, px, T(1)))));
        ig = T(1) / g;
        comp_add(x, cx, mul(h, px), ig);
        comp_add(y, cy, mul(h, py), ig);
        comp_add(z, cz, mul(h, pz), ig);
        st++;
        r2 = norm2(x, y, z);
        const T e2 = norm2(y, x, z);  // the end test rounds y^2 first
        if (e2 < a.r_in2) { status = 1; break; }
        if (e2 > a.r_out2) { status = 2; break; }
        if (st >= a.max_steps) { status = 0; break; }
      }
      if (status >= 0) {
        a.x[idx] = x; a.y[idx] = y; a.z[idx] = z;
        a.px[idx] = px; a.py[idx] = py; a.pz[idx] = pz;
        a.status[idx] = status;
        a.steps[idx] = st;
        my_total += (unsigned long long)st;
        idx = -1;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) my_total += __shfl_xor_sync(0xffffffffu, my_total, o);
  if (lane == 0 && my_total) atomicAdd(a.total, my_total);
}

__global__ void k_set_queue(unsigned long long* queue, unsigned long long first) { *queue = first; }

// The caller's interleaved SI arrays <-> normalised component arrays (FP64
// divisions and products rounded as written, then to T): a host loop over them,
// six pageable copies each way and nine allocations took longer than the tracing
// (call of 262,144 FP32 particles x 2000 steps: 6.2 ms, now 4.4).  The SI values
// cross in chunks of kTraceChunk particles (s: the chunk's first in the states of n
// particles), so they take 12.6 MB at any n beside the 36 (FP32) or 60 bytes of a
// particle's state, status and step count; a chunk's 6 MB per array take ten times
// its launch.
constexpr long long kTraceChunk = 1 << 18;
template <class T>
__global__ void __launch_bounds__(256) k_trace_in(long long count, long long n, const double* __restrict__ x,
                                                  const double* __restrict__ p, double r_e, double pscale,
                                                  T* __restrict__ s) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * count) return;
  const long long i = t / 3, d = t - 3 * i;
  s[d * n + i] = (T)(x[t] / r_e);
  s[(3 + d) * n + i] = (T)__dmul_rn(p[t], pscale);
}
template <class T>
__global__ void __launch_bounds__(256) k_trace_out(long long count, long long n, const T* __restrict__ s,
                                                   double r_e, double pscale, double* __restrict__ x,
                                                   double* __restrict__ p) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * count) return;
  const long long i = t / 3, d = t - 3 * i;
  x[t] = __dmul_rn((double)s[d * n + i], r_e);
  p[t] = (double)s[(3 + d) * n + i] / pscale;
}

template <class T>
amps_gpu_status run_trace(long long n, double* x, double* p, int32_t* status, int64_t* steps,
                          double q, double m0, double b_eq, double r_e, const double* b_ext,
                          double r_in, double r_out, long long max_steps, double dphi_max,
                          double dt_max, long long* total_steps, double* kernel_ms) {
  const double pscale = 1.0 / (m0 * kC);
  // one allocation: control words, a chunk's SI arrays, step counts, state, status
  const size_t sn = (size_t)n, ch = (size_t)std::min(n, kTraceChunk);
  const size_t bytes = 64 + ch * 6 * sizeof(double) + sn * (sizeof(int64_t) + 6 * sizeof(T) + sizeof(int32_t));
  char* mem = nullptr;
  cudaStream_t s = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  auto cleanup = [&]() {
    cudaFree(mem);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (s) cudaStreamDestroy(s);
  };
  bool ok = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess;
  ok = ok && cudaMalloc(reinterpret_cast<void**>(&mem), bytes) == cudaSuccess;
  ok = ok && cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess;
  unsigned long long* d_ctl = reinterpret_cast<unsigned long long*>(mem);
  double* d_x = reinterpret_cast<double*>(mem + 64);
  double* d_p = d_x + 3 * ch;
  int64_t* d_steps = reinterpret_cast<int64_t*>(d_p + 3 * ch);
  T* d = reinterpret_cast<T*>(d_steps + sn);
  int32_t* d_st = reinterpret_cast<int32_t*>(d + 6 * sn);
  ok = ok && cudaMemsetAsync(d_ctl, 0, 64, s) == cudaSuccess;
  auto cgrid = [](long long count) { return (unsigned)((3 * count + 255) / 256); };
  for (long long i = 0; ok && i < n; i += kTraceChunk) {
    const long long count = std::min(n - i, kTraceChunk);
    const size_t b = sizeof(double) * 3 * (size_t)count;
    ok = cudaMemcpyAsync(d_x, x + 3 * i, b, cudaMemcpyHostToDevice, s) == cudaSuccess &&
         cudaMemcpyAsync(d_p, p + 3 * i, b, cudaMemcpyHostToDevice, s) == cudaSuccess;
    if (ok) k_trace_in<T><<<cgrid(count), 256, 0, s>>>(count, n, d_x, d_p, r_e, pscale, d + i);
  }
  if (!ok) {
    cudaGetLastError();
    cleanup();
    return AMPS_GPU_CUDA_ERROR;
  }
  TraceArgs<T> a;
  a.x = d; a.y = d + sn; a.z = d + 2 * sn; a.px = d + 3 * sn; a.py = d + 4 * sn; a.pz = d + 5 * sn;
  a.status = d_st; a.steps = d_steps; a.n = n;
  a.queue = d_ctl; a.total = d_ctl + 1; a.flags = d_ctl + 2;
  a.kq = (T)(q * b_eq * r_e / (m0 * kC));
  for (int k = 0; k < 3; k++) a.ext[k] = (T)(b_ext ? b_ext[k] / b_eq : 0.0);
  a.r_in2 = (T)((r_in / r_e) * (r_in / r_e));
  a.r_out2 = (T)((r_out / r_e) * (r_out / r_e));
  a.dphi = (T)dphi_max;
  a.dt_max = (T)(dt_max * kC / r_e);
  a.max_steps = max_steps;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  constexpr int NT = TraceShape<T>::kThreads;
  const int grid = nsm * TraceShape<T>::kPerSM;
  const long long warps = (long long)grid * (NT / 32);
  // a CTA ends when its particles have; the cap is a safety net far above that:
  // the even share of particles of a lane, each at full length, 8 times over (as far
  // as 63 bits go: max_steps may be any)
  const double cap = 8.0 * (double)((n + 32 * warps - 1) / (32 * warps) + 2) * ((double)(max_steps / kRefill) + 3.0) +
                     (double)n + 16.0;
  a.iter_cap = cap < 9.0e18 ? (long long)cap : 9000000000000000000LL;
  cudaEventRecord(e0, s);
  k_set_queue<<<1, 1, 0, s>>>(a.queue, (unsigned long long)(32 * warps));
  k_trace<T><<<grid, NT, 0, s>>>(a);
  cudaEventRecord(e1, s);
  unsigned long long ctl[4];
  cudaError_t err = cudaGetLastError();
  for (long long i = 0; err == cudaSuccess && i < n; i += kTraceChunk) {
    const long long count = std::min(n - i, kTraceChunk);
    const size_t b = sizeof(double) * 3 * (size_t)count;
    k_trace_out<T><<<cgrid(count), 256, 0, s>>>(count, n, d + i, r_e, pscale, d_x, d_p);
    if ((err = cudaGetLastError()) == cudaSuccess) err = cudaMemcpyAsync(x + 3 * i, d_x, b, cudaMemcpyDeviceToHost, s);
    if (err == cudaSuccess) err = cudaMemcpyAsync(p + 3 * i, d_p, b, cudaMemcpyDeviceToHost, s);
  }
  if (err == cudaSuccess) err = cudaMemcpyAsync(ctl, d_ctl, sizeof(ctl), cudaMemcpyDeviceToHost, s);
  if (err == cudaSuccess) err = cudaMemcpyAsync(status, d_st, sizeof(int32_t) * sn, cudaMemcpyDeviceToHost, s);
  if (err == cudaSuccess) err = cudaMemcpyAsync(steps, d_steps, sizeof(int64_t) * sn, cudaMemcpyDeviceToHost, s);
  if (err == cudaSuccess) err = cudaStreamSynchronize(s);
  if (err != cudaSuccess) {
    cleanup();
    return AMPS_GPU_CUDA_ERROR;
  }
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  if (kernel_ms) *kernel_ms = ms;
  if (total_steps) *total_steps = (long long)ctl[1];
  cleanup();
  return ctl[2] ? AMPS_GPU_DEVICE_TIMEOUT : AMPS_GPU_OK;
}

}  // namespace

extern "C" amps_gpu_status amps_gpu_trace_dipole(int device, long long n, double* x, double* p,
                                                 int32_t* status, int64_t* steps, double q,
                                                 double m0, double b_eq, double r_e,
                                                 const double* b_ext, double r_in, double r_out,
                                                 long long max_steps, double dphi_max,
                                                 double dt_max, int precision,
                                                 long long* total_steps, double* kernel_ms) {
  if (n < 0 || (n > 0 && (!x || !p || !status || !steps)) || m0 <= 0.0 || b_eq == 0.0 ||
      r_e <= 0.0 || r_in < 0.0 || r_out <= r_in || max_steps <= 0 || dphi_max <= 0.0 ||
      dt_max <= 0.0 || (precision != 0 && precision != 1))
    return AMPS_GPU_INVALID_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return AMPS_GPU_NO_DEVICE;
  if (device < 0 || device >= ndev) return AMPS_GPU_INVALID_ARG;
  cudaSetDevice(device);
  if (n == 0) {
    if (total_steps) *total_steps = 0;
    return AMPS_GPU_OK;
  }
  if (precision == 0)
    return run_trace<double>(n, x, p, status, steps, q, m0, b_eq, r_e, b_ext, r_in, r_out,
                             max_steps, dphi_max, dt_max, total_steps, kernel_ms);
  return run_trace<float>(n, x, p, status, steps, q, m0, b_eq, r_e, b_ext, r_in, r_out, max_steps,
                          dphi_max, dt_max, total_steps, kernel_ms);
}
