// ECSIM field solve on sm_103a on uniform meshes (FP64 vectors; the inner
// GMRES operator in FP32 arithmetic around an FP64 identity part).
//
//   k_rhs       UpdateRhs with the supports registered by GetStencil
//               (src/pic/ecsim/get_stencil.cpp:1260-1599, ecsim/update_rhs.cpp:285):
//               theta c dt curl B^n - 4 pi theta dt J - (theta c dt)^2 curlcurl E^n
//               - 4 pi theta dt M E^n
//   k_matvec    the assembled row of GetStencil valued by UpdateMatrixElement
//               (pic_field_solver_ecsim.cpp:6004-6019) applied matrix-free:
//               A = I + (theta c dt)^2 (grad div - lap) + 4 pi theta dt M
//               (replaces cLinearSystemCornerNode::MultiplyVector,
//               srcInterface/LinearSystemCornerNode.h:3067-3205)
//   GMRES       restarted GMRES(30), x0 = 0, right preconditioner (none,
//               Jacobi, learned), classical Gram-Schmidt with one
//               re-orthogonalisation; each Arnoldi step is matvec + one
//               cooperative kernel on FP32-pair vectors (k_arnoldi_tile)
//               (the external linear_solver_wrapper of LinearSystemCornerNode.h:3282)
//   k_update_b  UpdateB (:5160-5711)
//   k_c2n_update_e  InterpolateB_C2N (:5715), UpdateE with the wave-energy sum
//   (:5909-6001)
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

#include "common.cuh"
#include "precond.cuh"
#include "ptx.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr int kMaxV = 32;
constexpr int kRedBlocks = 304;  // 2 x 152 SMs
constexpr int kGmOffset = 10240;  // doubles into d_red (12288 doubles)
constexpr int kTolOffset = 12287;  // the solve's tolerance, read by k_first
constexpr int kArnMaxGrid = 1024;  // CTAs of the cooperative Arnoldi step (at most)

struct Taps {
  double K[3][3][27];  // operator taps without the mass matrix
  double f;            // 4 pi theta dt
};

double tap_s(int o) { return o == 0 ? 0.5 : 0.25; }
double tap_d2(int o) { return o == 0 ? -2.0 : 1.0; }
double tap_d1(int o) { return o == 0 ? 0.0 : (o > 0 ? 0.5 : -0.5); }

// Separable form of the compact stencils built by InitDiscritizationStencil
// (pic_field_solver_ecsim.cpp:7121): d2/dx2 = D2(x) S(y) S(z),
// d2/dxdy = D1(x) D1(y) S(z), with S = (1/4, 1/2, 1/4), D2 = (1,-2,1), D1 = (-1/2,0,1/2).
Taps make_taps(const amps_gpu_config& cfg, bool identity) {
  Taps t{};
  double coeff[3], cs[3];
  for (int d = 0; d < 3; d++) {
    coeff[d] = cfg.dt / cfg.dx[d] * cfg.theta;
    cs[d] = coeff[d] * coeff[d];
  }
  for (int dk = -1; dk <= 1; dk++)
    for (int dj = -1; dj <= 1; dj++)
      for (int di = -1; di <= 1; di++) {
        const int o[3] = {di, dj, dk};
        const int s = mm_slot(di, dj, dk);
        double lap[3];
        for (int ax = 0; ax < 3; ax++) {
          double a = 1.0;
          for (int d = 0; d < 3; d++) a *= (d == ax) ? tap_d2(o[d]) : tap_s(o[d]);
          lap[ax] = a;
        }
        for (int p = 0; p < 3; p++)
          for (int q = 0; q < 3; q++) {
            double gd;
            if (p == q) {
              gd = lap[p];
            } else {
              gd = 1.0;
              for (int d = 0; d < 3; d++) gd *= (d == p || d == q) ? tap_d1(o[d]) : tap_s(o[d]);
            }
            double a = 0.0;
            if (p == q) {
              for (int d = 0; d < 3; d++) a -= lap[d] * cs[d];
              if (s == 0 && identity) a += 1.0;
            }
            a += gd * coeff[p] * coeff[q];
            t.K[p][q][s] = a;
          }
      }
  t.f = 4.0 * kPi * cfg.dt * cfg.theta;
  return t;
}

__device__ __forceinline__ void corner_ijk(long long c, int& b, int& i, int& j, int& k) {
  b = (int)(c / AMPS_CPB);
  const int l = (int)(c % AMPS_CPB);
  i = l & 7;
  j = (l >> 3) & 7;
  k = l >> 6;
}

// The operator taps split into FP32 pairs (K = Kh + Kl) for the FP64-accurate
// evaluations below.
struct TapsFF {
  float Kh[3][3][27], Kl[3][3][27];
  double f;
};

TapsFF taps_ff(const Taps& T) {
  TapsFF t;
  for (int p = 0; p < 3; p++)
    for (int q = 0; q < 3; q++)
      for (int s = 0; s < 27; s++) {
        t.Kh[p][q][s] = (float)T.K[p][q][s];
        t.Kl[p][q][s] = (float)(T.K[p][q][s] - (double)t.Kh[p][q][s]);
      }
  t.f = T.f;
  return t;
}

// xh + xl = dinv .* x (dinv may be null), split into FP32 pairs
__global__ void __launch_bounds__(256) k_split(long long n, const double* __restrict__ x,
                                               const double* __restrict__ dinv,
                                               float* __restrict__ xh, float* __restrict__ xl) {
  pdl_wait();
  pdl_next();
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const double v = dinv ? dinv[t] * x[t] : x[t];
    const float h = (float)v;
    xh[t] = h;
    xl[t] = (float)(v - (double)h);
  }
}

struct TapsF {
  float K[3][3][27];
  float f;
};

TapsF taps_f32(const Taps& T) {
  TapsF t;
  for (int p = 0; p < 3; p++)
    for (int q = 0; q < 3; q++)
      for (int s = 0; s < 27; s++) t.K[p][q][s] = (float)T.K[p][q][s];
  t.f = (float)T.f;
  return t;
}

// ---- the 27-point operator ---------------------------------------------------
// A CTA takes 32 consecutive corners (ncor is a multiple of 512) and splits the
// 27 slots into 8 groups (slot s: group s mod 8) over its 2, 4 or 8 warps; lane =
// corner, so the 243 coefficient planes of M are read in whole lines, and a slot's
// neighbour values serve the three components.  The groups' sums meet in shared
// memory and are added in their order, so that a row has the same bits at any CTA
// size (the autotuner chooses it by time).  Bound: latency on small meshes --
// one thread per (component, corner) walked all 27 slots, nine rounds of
// dependent loads -- and reading M (HBM) on large ones.  us per application,
// before and now, at 512 and at 32,768 corners: FP32 operator 15.6 -> 8.0, 18.5 ->
// 13.0 (5.0 and 10.6 back to back); residual operator with its input split 23.2 ->
// 16.1, 30.5 -> 27.2, 9.7 and 21.2 on pairs that are there; RHS with the split of E^n
// 27 -> 15.4, 42 -> 36.8.
constexpr int kOpGroups = 8;  // of slots; a CTA has at most a warp per group

__device__ __forceinline__ void slot_offset(int s, int& di, int& dj, int& dk) {
  const int d0 = s % 3, d1 = (s / 3) % 3, d2 = s / 9;
  di = d0 == 0 ? 0 : (d0 == 1 ? -1 : 1);
  dj = d1 == 0 ? 0 : (d1 == 1 ? -1 : 1);
  dk = d2 == 0 ? 0 : (d2 == 1 ? -1 : 1);
}

// The slots of a group of (K + f M) x at corner c, all three rows, to FP64 accuracy:
// sk the taps, sm the mass matrix's FP32 coefficients, against the split input.
struct RowFF {
  FF sk[3], sm[3];
};
__device__ __forceinline__ RowFF rows_ff(long long ncor, const int* __restrict__ nbr, const float* __restrict__ M,
                                         const float* __restrict__ xh, const float* __restrict__ xl,
                                         const TapsFF& T, long long c, int b, int i, int j, int k, int group) {
  RowFF r;
#pragma unroll
  for (int p = 0; p < 3; p++) r.sk[p] = r.sm[p] = FF{0.f, 0.f};
#pragma unroll 2
  for (int s = group; s < 27; s += kOpGroups) {
    int di, dj, dk;
    slot_offset(s, di, dj, dk);
    const int nb = local_id(nbr, b, i + di, j + dj, k + dk);
    float h[3], lo[3], m[9];
#pragma unroll
    for (int q = 0; q < 3; q++) { h[q] = xh[q * ncor + nb]; lo[q] = xl[q * ncor + nb]; }
#pragma unroll
    for (int e = 0; e < 9; e++) m[e] = M[(size_t)(9 * s + e) * ncor + c];
#pragma unroll
    for (int p = 0; p < 3; p++)
#pragma unroll
      for (int q = 0; q < 3; q++) {
        ff_add2(r.sk[p], T.Kh[p][q][s], T.Kl[p][q][s], h[q], lo[q]);
        ff_add(r.sm[p], m[3 * p + q], h[q], lo[q]);
      }
  }
  return r;
}
// The groups' rows into s_row[6][kOpGroups][32], a warp's after one another, and
// component p of the sum at lane (after the barrier)
__device__ __forceinline__ void rows_store(long long ncor, const int* __restrict__ nbr, const float* __restrict__ M,
                                           const float* __restrict__ xh, const float* __restrict__ xl,
                                           const TapsFF& T, long long c, int b, int i, int j, int k,
                                           float2 (*s_row)[kOpGroups][32], int wid, int warps, int lane) {
  for (int g = wid; g < kOpGroups; g += warps) {
    const RowFF r = rows_ff(ncor, nbr, M, xh, xl, T, c, b, i, j, k, g);
#pragma unroll
    for (int p = 0; p < 3; p++) {
      s_row[p][g][lane] = make_float2(r.sk[p].s, r.sk[p].q);
      s_row[3 + p][g][lane] = make_float2(r.sm[p].s, r.sm[p].q);
    }
  }
}
__device__ __forceinline__ double rows_sum(float2 (*s_row)[kOpGroups][32], int p, int lane, double f) {
  FF a{0.f, 0.f}, m{0.f, 0.f};
#pragma unroll
  for (int g = 0; g < kOpGroups; g++) {
    ff_acc(a, s_row[p][g][lane].x, s_row[p][g][lane].y);
    ff_acc(m, s_row[3 + p][g][lane].x, s_row[3 + p][g][lane].y);
  }
  return ff_value(a) + f * ff_value(m);
}

// y = A (dinv .* x) to FP64 accuracy from the split input (outer residuals)
__global__ void __launch_bounds__(32 * kOpGroups) k_matvec(long long ncor, const int* __restrict__ nbr,
                                                             const float* __restrict__ M,
                                                             const float* __restrict__ xh,
                                                             const float* __restrict__ xl,
                                                             double* __restrict__ y,
                                                             const __grid_constant__ TapsFF T) {
  pdl_wait();
  pdl_next();
  __shared__ float2 s_row[6][kOpGroups][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const long long c = (long long)blockIdx.x * 32 + lane;
  int b, i, j, k;
  corner_ijk(c, b, i, j, k);
  rows_store(ncor, nbr, M, xh, xl, T, c, b, i, j, k, s_row, wid, warps, lane);
  __syncthreads();
  for (int p = wid; p < 3; p += warps) y[p * ncor + c] = rows_sum(s_row, p, lane, T.f);
}

// RHS: theta c dt curl B^n - f J - (curl-curl + f M) E^n, the last term to
// FP64 accuracy from the split E^n (taps without the identity)
__global__ void __launch_bounds__(32 * kOpGroups) k_rhs(long long ncor, const int* __restrict__ nbr,
                                                          const float* __restrict__ M,
                                                          const float* __restrict__ Eh,
                                                          const float* __restrict__ El,
                                                          const double* __restrict__ Bc,
                                                          const double* __restrict__ J,
                                                          double* __restrict__ rhs,
                                                          const __grid_constant__ TapsFF T, double c4x,
                                                          double c4y, double c4z) {
  pdl_wait();
  pdl_next();
  __shared__ float2 s_row[6][kOpGroups][32];
  __shared__ double s_cb[3][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const long long c = (long long)blockIdx.x * 32 + lane;
  int b, i, j, k;
  corner_ijk(c, b, i, j, k);
  // curl B^n from the 2x2 face averages of the 8 cells around the corner,
  // components from the last warp down (the first have one slot more)
  auto Bv = [&](int ii, int jj, int kk, int comp) {
    return Bc[comp * ncor + local_id(nbr, b, ii, jj, kk)];
  };
  for (int p = warps - 1 - wid; p < 3; p += warps) {
    double cb = 0.0;
#pragma unroll
    for (int a = -1; a <= 0; a++)
#pragma unroll
      for (int q = -1; q <= 0; q++) {
        if (p == 0) {
          cb += c4y * (Bv(i + a, j, k + q, 2) - Bv(i + a, j - 1, k + q, 2));
          cb += -c4z * (Bv(i + a, j + q, k, 1) - Bv(i + a, j + q, k - 1, 1));
        } else if (p == 1) {
          cb += c4z * (Bv(i + a, j + q, k, 0) - Bv(i + a, j + q, k - 1, 0));
          cb += -c4x * (Bv(i, j + q, k + a, 2) - Bv(i - 1, j + q, k + a, 2));
        } else {
          cb += c4x * (Bv(i, j + q, k + a, 1) - Bv(i - 1, j + q, k + a, 1));
          cb += -c4y * (Bv(i + q, j, k + a, 0) - Bv(i + q, j - 1, k + a, 0));
        }
      }
    s_cb[p][lane] = cb - T.f * J[p * ncor + c];
  }
  rows_store(ncor, nbr, M, Eh, El, T, c, b, i, j, k, s_row, wid, warps, lane);
  __syncthreads();
  for (int p = wid; p < 3; p += warps) rhs[p * ncor + c] = s_cb[p][lane] - rows_sum(s_row, p, lane, T.f);
}

__global__ void __launch_bounds__(256) k_jacobi(long long ncor, const float* __restrict__ M,
                                                double* __restrict__ dinv, float* __restrict__ dff, double k00,
                                                double k11, double k22, double f) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncor) return;
  // a preconditioner: FP32 arithmetic (FP64 division is slow on this part)
  const float v[3] = {1.0f / fmaf((float)f, M[(size_t)0 * ncor + c], (float)k00),
                      1.0f / fmaf((float)f, M[(size_t)4 * ncor + c], (float)k11),
                      1.0f / fmaf((float)f, M[(size_t)8 * ncor + c], (float)k22)};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    dinv[d * ncor + c] = (double)v[d];
    dff[d * ncor + c] = v[d];  // as pairs: FP32 values
    dff[3 * ncor + d * ncor + c] = 0.f;
  }
}

// ---- reductions ------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Reduce acc[0..nv) over the block and store partial[blockIdx.x*kMaxV + i].
template <int NVM>
__device__ __forceinline__ void block_store_partials(double* acc, int nv, double* partial) {
  __shared__ double s_red[8][NVM];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NVM; i++) {
    if (i < nv) {
      double v = warp_sum(acc[i]);
      if (lane == 0) s_red[wid][i] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < nv) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += s_red[w][threadIdx.x];
    partial[blockIdx.x * kMaxV + threadIdx.x] = t;
  }
}

// x += dinv .* sum_i y_i V_i  (nv from *d_nv when given)
__global__ void __launch_bounds__(256) k_combine(long long n, const double* __restrict__ V,
                                                 const double* __restrict__ y, int nv,
                                                 const int* __restrict__ d_nv,
                                                 const double* __restrict__ dinv,
                                                 double* __restrict__ x) {
  __shared__ double s_y[kMaxV];
  if (d_nv) nv = *d_nv;
  if (threadIdx.x < kMaxV) s_y[threadIdx.x] = threadIdx.x < nv ? y[threadIdx.x] : 0.0;
  __syncthreads();
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    double a = 0.0;
    for (int i = 0; i < nv; i++) a += s_y[i] * V[(size_t)i * n + t];
    x[t] += (dinv ? dinv[t] : 1.0) * a;
  }
}

// GMRES least-squares state on the device: the Hessenberg columns after the
// Givens rotations (row stride kMaxV), the rotations, the rotated right-hand
// side g (|g[j]| = residual norm after j steps), the solution y, and the
// step count jj / converged flag that the host polls.
struct GmState {
  double H[(kMaxV + 1) * kMaxV];
  double cs[kMaxV], sn[kMaxV];
  double g[kMaxV + 1];
  double y[kMaxV];
  double target;
  int jj;    // columns processed in this cycle
  int done;  // |g[jj]| <= target, or breakdown
  double bn2, rn2;  // ||b||^2 (k_first), end-of-cycle ||r||^2 (k_residual)
  unsigned long long timeouts;  // bounded waits that ran out in the solve's Arnoldi steps
  unsigned ticket;  // CTAs of a reducing kernel that have stored their share (0 between kernels)
};
// what the host reads at a time: jj, done, bn2, rn2, timeouts
struct GmStatus {
  int jj, done;
  double bn2, rn2;
  unsigned long long timeouts;
};
static_assert(offsetof(GmState, timeouts) - offsetof(GmState, jj) == offsetof(GmStatus, timeouts), "GmStatus layout");
static_assert(kGmOffset * sizeof(double) + sizeof(GmState) <= kTolOffset * sizeof(double),
              "GmState must fit in d_red");
static_assert(kRedBlocks * kMaxV < kGmOffset, "d_red layout");

// start of a cycle: g = (||r||, 0, ...); *n2 = ||r||^2
__global__ void k_gm_start(GmState* __restrict__ S, const double* __restrict__ n2, double target) {
  if (threadIdx.x != 0) return;
  for (int i = 0; i <= kMaxV; i++) S->g[i] = 0.0;
  S->g[0] = sqrt(*n2);
  S->target = target;
  S->jj = 0;
  S->done = 0;
}

// Sum of acc over the grid, returned in every thread of the CTA that stores its share
// last (true there); partial sums are added in the order of the CTAs.  256 threads.
__device__ __forceinline__ bool grid_sum(double acc, double* __restrict__ partial, unsigned* ticket, double& sum) {
  __shared__ double s_sum;
  __shared__ int s_last;
  double a[1] = {acc};
  block_store_partials<1>(a, 1, partial);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (int bk = threadIdx.x; bk < (int)gridDim.x; bk += 32) t += __ldcg(partial + bk * kMaxV);
    t = warp_sum(t);
    if (threadIdx.x == 0) {
      s_sum = t;
      *ticket = 0u;
    }
  }
  __syncthreads();
  sum = s_sum;
  return true;
}

// Start of a solve from x0 = 0: r = b (in w), x = 0, ||b||^2, and the state of a first
// cycle with the target *tol ||b|| (in memory: a captured launch serves any tolerance).
// (One launch: the copy, the clearing, the norm, its
// reduction and the state took five, ~4 us each on a small mesh.)
__global__ void __launch_bounds__(256) k_first(long long n, const double* __restrict__ b, double* __restrict__ w,
                                               double* __restrict__ x, double* __restrict__ partial,
                                               double* __restrict__ n2, GmState* __restrict__ S,
                                               const double* __restrict__ tol) {
  pdl_wait();
  pdl_next();
  double acc = 0.0;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const double v = b[t];
    w[t] = v;
    x[t] = 0.0;
    acc += v * v;
  }
  double b2;
  if (!grid_sum(acc, partial, &S->ticket, b2)) return;
  if (threadIdx.x <= kMaxV) S->g[threadIdx.x] = threadIdx.x == 0 ? sqrt(b2) : 0.0;
  if (threadIdx.x == 0) {
    *n2 = b2;
    S->target = *tol * sqrt(b2);
    S->jj = 0;
    S->done = 0;
    S->bn2 = b2;
    S->rn2 = -1.0;
    S->timeouts = 0ull;
  }
}

// r = b - r (in place on r) and ||r||^2
__global__ void __launch_bounds__(256) k_residual(long long n, const double* __restrict__ b,
                                                  double* __restrict__ r, double* __restrict__ partial,
                                                  double* __restrict__ n2, GmState* __restrict__ S) {
  pdl_wait();
  pdl_next();
  double acc = 0.0;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const double v = b[t] - r[t];
    r[t] = v;
    acc += v * v;
  }
  double r2;
  if (!grid_sum(acc, partial, &S->ticket, r2) || threadIdx.x != 0) return;
  *n2 = r2;
  S->rn2 = r2;
}

// Arnoldi column jj: h = h1 + h2 (the two CGS passes), h[jj+1] = ||w||; apply
// the previous rotations, form rotation jj, update g.  Frozen once done, so
// steps launched past convergence change nothing the solution uses.  One thread.
__device__ void gm_update(GmState* __restrict__ S, int jj, const double* h1, const double* h2,
                          double n2) {
  if (S->done) return;
  double* H = S->H;
  const double hn = sqrt(n2);
  // the column runs through the rotations in a register
  double a = h1[0] + h2[0];
  const double b = hn;
#pragma unroll 4
  for (int i = 0; i < jj; i++) {
    const double hb = h1[i + 1] + h2[i + 1], c0 = S->cs[i], s0 = S->sn[i];
    H[i * kMaxV + jj] = c0 * a + s0 * hb;
    a = -s0 * a + c0 * hb;
  }
  const double r = sqrt(a * a + b * b);
  const double c = r > 0.0 ? a / r : 1.0, s = r > 0.0 ? b / r : 0.0;
  S->cs[jj] = c;
  S->sn[jj] = s;
  H[jj * kMaxV + jj] = r;
  H[(jj + 1) * kMaxV + jj] = 0.0;
  S->g[jj + 1] = -s * S->g[jj];
  S->g[jj] = c * S->g[jj];
  S->jj = jj + 1;
  if (fabs(S->g[jj + 1]) <= S->target || hn == 0.0) S->done = 1;
}

// y = R^-1 g on the processed columns, by the whole CTA: R staged, then one lane per
// row and a back substitution by columns (reciprocals of the diagonal first, so the
// chain holds a product and an FMA per column).  s_y: kMaxV values.
__device__ __forceinline__ void gm_solve(const GmState* __restrict__ S, double* s_y) {
  __shared__ double s_h[kMaxV][kMaxV + 1];
  const int j = min(S->jj, kMaxV);
  for (int q = threadIdx.x; q < j * j; q += blockDim.x) s_h[q / j][q % j] = S->H[(q / j) * kMaxV + q % j];
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const double d = lane < j ? s_h[lane][lane] : 0.0;
    const double inv = d != 0.0 ? 1.0 / d : 0.0;
    double g = lane < j ? S->g[lane] : 0.0;
    for (int i = j - 1; i >= 0; i--) {
      const double y = __shfl_sync(0xffffffffu, g * inv, i);
      if (lane == i) g = y;
      if (lane < i) g -= s_h[lane][i] * y;
    }
    s_y[lane] = g;
  }
  __syncthreads();
}
__global__ void __launch_bounds__(256) k_gm_solve(GmState* __restrict__ S) {
  __shared__ double s_y[kMaxV];
  gm_solve(S, s_y);
  if (threadIdx.x < kMaxV) S->y[threadIdx.x] = s_y[threadIdx.x];
}

// ---- Krylov vectors in FP32 pairs ----------------------------------------------
// The Arnoldi basis and the operator output are stored as FP32 pairs (hi, lo:
// 48 significant bits, the bytes of a double vector): FP64 arithmetic runs at
// ~1/70 of the FP32 rate on this part, and CGS2 is 4 nv n multiply-adds per
// step, so the sweeps run in pair arithmetic and only the sums over the CTAs
// touch FP64.  One whole Arnoldi step after the operator is one cooperative
// launch (grid-wide barriers between the sweeps); every CTA adds up the per-CTA
// partial sums of a sweep itself.

// a += (xh + xl)(yh + yl)
__device__ __forceinline__ void ff_dot_acc(FF& a, float xh, float xl, float yh, float yl) {
  const float p = __fmul_rn(xh, yh);
  ff_acc(a, p, fmaf(xh, yl, fmaf(xl, yh, fmaf(xh, yh, -p))));
}
__device__ __forceinline__ FF ff_shfl_xor(const FF& a, int o) {
  return FF{__shfl_xor_sync(0xffffffffu, a.s, o), __shfl_xor_sync(0xffffffffu, a.q, o)};
}
__device__ __forceinline__ FF ff_warp_sum(FF a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const FF b = ff_shfl_xor(a, o);
    ff_acc(a, b.s, b.q);
  }
  return a;
}

// One Arnoldi step on pair vectors: CGS2 of w against V_0..V_{nv-1} (h1 = V^T w,
// w' = w - V h1, h2 = V^T w', w'' = w' - V h2), V_nv = w'' / ||w''||, and the
// Givens update of the least-squares state.  Vectors are pair streams: hi at
// V + 2 i ld, lo ld behind it, ld = n rounded up to 4 so that every stream
// starts on 16 bytes.
//
// Bound: reading the basis (n = 1.34M, 15 vectors: 161 MB a sweep).  Two
// persistent CTAs per SM (one computes while the other waits at a barrier); a
// producer warp brings tiles of T elements of every stream into a ring of
// shared-memory stages by tensor copies (all rows of a tile in one: a bulk copy
// per row, 62 of 512 bytes at 30 vectors, kept the copy engine busy longer than
// the bytes; up to 200 KB in flight per SM, which per-thread loads at 2 CTAs per
// SM did not reach), and 8 consumer warps work on the staged tile:
//   - update: a thread owns T / 256 elements (T = 128: two threads split an
//     element's vectors, even and odd);
//   - dots: a warp owns whole vectors (or an element range of one when there
//     are fewer vectors than warps), so the register cost does not grow with
//     nv and no sums cross warps inside the sweep.
// The staged tile serves both halves of the second sweep (w' and then h2), the
// third sweep needs V's hi halves only and sums V h2 in FP32, and tiles are walked
// in alternating directions so a sweep starts on what the last one left in L2: 2.5
// basis reads per step.  ||w''||^2 = ||w'||^2 - ||h2||^2 (V orthonormal) spares a
// sweep and a grid barrier.  Both hold where h2 is no more than the first
// projection's rounding, a few 2^-48 |w|: FP32 is wrong by 2^-24 of V h2, which
// ||h2|| <= 2^-28 ||w'|| (kArnSmallH2, its square) keeps under the pairs' own
// last bit (solves: ||h2||^2 / ||w'||^2 of 1e-29 to 1e-23 in all of 181 steps looked
// at).  Any larger h2 (|w'| far below |w|, or a basis that lost its orthogonality)
// takes the third sweep in full pairs and the norm from its sum, one more grid barrier.
// A CTA whose tiles all fit its stages reads them once.
// Waits give up after `limit` polls (counted in the state): a producer whose stage is
// not freed issues nothing more, a consumer warp whose tile does not come goes on and
// frees nothing more, so that a stage is never filled over a copy still in flight; all
// take part in every barrier, and the producer leaves when its last copies have
// landed.  (64 registers at the tiles of long bases: with 80, which votes or flags at
// the waits cost, the next kernels' early CTAs find no room beside this one, 14 us a
// step of a learned solve on 1.1M unknowns.)
// 1.34M unknowns, mean step of a 55-iteration solve (1 to 30 vectors): 103 us, 4 us
// per vector (the rate of HBM) on ~45 us of barriers and start-up.  Before: 304 us
// with per-thread streams, four basis reads and three barriers; 150 us with one CTA
// per SM and a bulk copy per row.  1.50M unknowns, 1 to 8 vectors: 59 us, before 81.
constexpr int kArnCons = 256;               // consumer threads (8 warps)
constexpr int kArnBlock = kArnCons + 32;    // + the producer warp
constexpr int kArnWarps = kArnCons / 32;
constexpr int kArnMaxStages = 16;
// shared memory of a CTA (two per SM): two tiles of w' and, where two threads
// split an element's vectors, of the odd shares; the rest is the ring
constexpr size_t kArnSmem = 108 * 1024;
constexpr size_t arn_extra(int T) { return sizeof(float) * (T < kArnCons ? 8 : 4) * T; }
constexpr size_t arn_ring(int T) { return kArnSmem - arn_extra(T); }
constexpr int kArnDots = kMaxV;             // dots per sweep: nv, and ||w'||^2
constexpr double kArnSmallH2 = 0x1p-56;     // of ||h2||^2 / ||w'||^2
constexpr int kArnRounds = kArnDots / kArnWarps;  // vectors per warp at most

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// orders this thread's generic writes before later bulk copies of the same addresses
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void bar_consumers() {
  asm volatile("bar.sync 1, %0;" ::"n"(kArnCons) : "memory");
}
__device__ __forceinline__ void bar_all() { asm volatile("bar.sync 2, %0;" ::"n"(kArnBlock) : "memory"); }

// Descriptors of the streams as 2D arrays of ld columns: the 2 nv rows of the
// basis pairs, the nv rows of its hi halves, the 2 rows of w
struct ArnMaps {
  CUtensorMap v, h, w;
};

template <int T>
__global__ void __launch_bounds__(kArnBlock, 2) k_arnoldi_tile(
    const __grid_constant__ ArnMaps maps, long long n, long long ld, float* __restrict__ w, int nv,
    float* __restrict__ vnext, float2* __restrict__ part, GmState* gs, int jj, float* __restrict__ xf,
    const float* __restrict__ dh, int stages, uint32_t limit) {
  cg::grid_group grid = cg::this_grid();
  extern __shared__ __align__(128) float s_ring[];
  __shared__ __align__(8) uint64_t full[kArnMaxStages], empty[kArnMaxStages];
  __shared__ float2 s_red[kArnWarps][kArnRounds];
  __shared__ double s_h1[kMaxV], s_h2[kMaxV], s_n2, s_inv;
  __shared__ float2 s_f[kArnDots];               // the coefficients of the running sweep as pairs
  __shared__ int s_slow;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nblk = gridDim.x;
  constexpr int M = T >= kArnCons ? T / kArnCons : 1;  // chunks of a tile = elements per thread
  constexpr int C = T / M;                             // elements per chunk (a copy's width)
  constexpr int G = kArnCons / C;                      // threads per element
  const int tiles = (int)((n + T - 1) / T);
  const int nt = (tiles - (int)blockIdx.x + nblk - 1) / nblk;  // this CTA's tiles (grid <= tiles)
  const bool resident = nt <= stages;
  // a stage: M chunks of 2 nv + 2 rows of C floats (V_0 hi, lo, V_1 hi, .., w hi,
  // lo; the third sweep: V_0 hi, V_1 hi, .., D in the first nv + 1 rows)
  const int chunk_f = (2 * nv + 2) * C;
  const size_t stage_f = (size_t)M * chunk_f;
  // w' of two tiles (hi, lo): the next tile's is written while slow warps still
  // read this one's; G = 2: the odd vectors' share of the update, likewise
  float* s_w = s_ring + stages * stage_f;
  float2* s_part = reinterpret_cast<float2*>(s_w + 4 * T);
  auto tile_of = [&](int k) { return (long long)blockIdx.x + (long long)k * nblk; };
  auto count_of = [&](int k) { return (int)min((long long)T, n - tile_of(k) * T); };
  pdl_next();
  if (tid == 0) {
    for (int s = 0; s < stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kArnWarps);
    }
    fence_mbar_init();
  }
  __syncthreads();

  if (wid == kArnWarps) {
    // ---- producer warp: tile k of the sweep as the ring's use number c; pairs of
    // V, or its hi halves (and D)
    int end = resident ? nt : 3 * nt;  // of the uses; lower where it gave up
    auto issue = [&](int c, int k, bool pairs, const float* D) {
      const int s = c % stages;
      if (c >= stages && !mbar_wait_bounded(&empty[s], ((c / stages) - 1) & 1, limit)) {
        if (lane == 0) atomicAdd(&gs->timeouts, 1ull);
        end = min(end, c);
      }
      if (lane == 0 && c < end) {
        const long long e0 = tile_of(k) * T;
        const int count = count_of(k);
        const uint32_t dbytes = D ? (uint32_t)((count + 3) & ~3) * 4u : 0u;
        mbar_arrive_expect_tx(&full[s], (uint32_t)(T * 4 * (pairs ? 2 * nv + 2 : nv + 2)) + dbytes);
        for (int m = 0; m < M; m++) {
          float* dst = s_ring + (size_t)s * stage_f + m * chunk_f;
          tensor_copy_2d(dst, pairs ? &maps.v : &maps.h, (int)(e0 + m * C), 0, &full[s]);
          tensor_copy_2d(dst + 2 * nv * C, &maps.w, (int)(e0 + m * C), 0, &full[s]);
          const int dc = min(C, count - m * C);
          if (D && dc > 0) bulk_copy_g2s(dst + nv * C, D + e0 + m * C, (uint32_t)((dc + 3) & ~3) * 4u, &full[s]);
        }
      }
      __syncwarp();
    };
    for (int k = 0; k < nt; k++) issue(k, k, true, nullptr);
    const int pre = min(nt, stages);  // the second sweep's first tiles load across the barrier
    if (!resident)
      for (int k = 0; k < pre; k++) issue(nt + k, nt - 1 - k, true, nullptr);
    grid.sync();
    if (!resident)
      for (int k = pre; k < nt; k++) issue(nt + k, nt - 1 - k, true, nullptr);
    grid.sync();
    bar_all();  // s_slow
    const bool slow = s_slow != 0;
    if (!resident)
      for (int k = 0; k < nt; k++) issue(2 * nt + k, k, slow, slow || !xf ? nullptr : dh);
    if (slow) {
      grid.sync();
      bar_all();  // s_n2
    }
    if (blockIdx.x == 0 && lane == 0) gm_update(gs, jj, s_h1, s_h2, s_n2);
    if (lane == 0)
      for (int c = max(0, end - stages); c < end; c++)
        mbar_wait_bounded(&full[c % stages], (c / stages) & 1, kWaitLimit);
    return;
  }

  // ---- consumers
  bool bad = false;  // this lane gave up on a tile; lane 0 frees only while it saw all land
  auto acquire = [&](int c) -> float* {
    const int s = c % stages;
    if (!mbar_wait_bounded(&full[s], (c / stages) & 1, limit)) {
      atomicAdd(&gs->timeouts, 1ull);
      bad = true;
    }
    return s_ring + (size_t)s * stage_f;
  };
  auto release = [&](int c) {
    __syncwarp();
    if (lane == 0 && !bad) mbar_arrive(&empty[c % stages]);
  };
  // dots of the staged w with nd vectors (number nv: w itself): warp -> vector
  // and, with fewer vectors than warps, element range
  FF acc[kArnRounds];
  int dots_n = 0, dots_p = 1, dots_g = 1;
  auto dots_begin = [&](int nd) {
    dots_n = nd;
    dots_p = 1;
    while (dots_p < nd && dots_p < kArnWarps) dots_p *= 2;
    dots_g = kArnWarps / dots_p;  // element ranges per vector
#pragma unroll
    for (int r = 0; r < kArnRounds; r++) acc[r] = FF{0.f, 0.f};
  };
  // (w at wt, its chunks wstride apart)
  auto dots = [&](const float* st, const float* wt, int wstride, int count) {
    const int g = wid / dots_p;
#pragma unroll
    for (int r = 0; r < kArnRounds; r++) {
      const int i = wid % dots_p + kArnWarps * r;
      if (i >= dots_n) continue;
      for (int m = 0; m < M; m++) {
        const float* wm = wt + m * wstride;
        const float* v = i < nv ? st + m * chunk_f + 2 * i * C : wm;
        const int cm = min(C, count - m * C);
#pragma unroll 2
        for (int e = g * 32 + lane; e < cm; e += 32 * dots_g) ff_dot_acc(acc[r], v[e], v[C + e], wm[e], wm[C + e]);
      }
    }
  };
  // block sums to part[i * nblk + blk]; all blocks' sums after the barrier
  auto dots_end = [&](float2* __restrict__ out) {
#pragma unroll
    for (int r = 0; r < kArnRounds; r++) {
      const FF t = ff_norm(ff_warp_sum(acc[r]));
      if (lane == 0) s_red[wid][r] = make_float2(t.s, t.q);
    }
    bar_consumers();
    if (tid < dots_n) {
      const int r = tid / kArnWarps, wi = tid % kArnWarps;
      FF t{0.f, 0.f};
      for (int g = 0; g < dots_g; g++) {
        const float2 q = s_red[wi % dots_p + g * dots_p][r];
        ff_acc(t, q.x, q.y);
      }
      t = ff_norm(t);
      out[(size_t)tid * nblk + blockIdx.x] = make_float2(t.s, t.q);
    }
  };
  auto grid_sums = [&](const float2* __restrict__ in, int nd, double* __restrict__ h) {
    for (int i = wid; i < nd; i += kArnWarps) {
      FF t{0.f, 0.f};
      for (int b = lane; b < nblk; b += 32) {
        const float2 q = __ldcg(in + (size_t)i * nblk + b);
        ff_acc(t, q.x, q.y);
      }
      t = ff_norm(ff_warp_sum(t));
      if (lane == 0) {
        s_f[i] = make_float2(t.s, t.q);
        if (i < nv) h[i] = (double)t.s + (double)t.q;
        else s_n2 = (double)t.s + (double)t.q;
      }
    }
    bar_consumers();
  };
  // sum_i V_i f_i of the staged tile at this thread's M elements (G = 2: its
  // share of the vectors; half 1 leaves its own in s_part); pass: the tile's
  // number in the sweep
  const int e0 = tid & (C - 1), half = tid / C;
  auto share = [&](const float* st, bool pairs, int pass, FF (&p)[M]) {
#pragma unroll
    for (int m = 0; m < M; m++) p[m] = FF{0.f, 0.f};
    if (pairs) {
#pragma unroll 2
      for (int i = half; i < nv; i += G) {
        const float* v = st + 2 * i * C + e0;
        const float2 f = s_f[i];
#pragma unroll
        for (int m = 0; m < M; m++) {
          const FF u = ff_mul(v[m * chunk_f], v[m * chunk_f + C], f.x, f.y);
          ff_acc(p[m], u.s, u.q);
        }
      }
    } else {
#pragma unroll 4
      for (int i = half; i < nv; i += G) {
        const float* v = st + i * C + e0;
        const float f = s_f[i].x;
#pragma unroll
        for (int m = 0; m < M; m++) p[m].s = fmaf(v[m * chunk_f], f, p[m].s);
      }
    }
    if (G == 2) {
      if (half) s_part[(pass & 1) * T + e0] = make_float2(p[0].s, p[0].q);
      bar_consumers();
    }
  };
  // w - V f at this thread's element of a chunk (half 0; p: its own share)
  auto minus = [&](const float* wm, int pass, const FF& p) {
    FF t{wm[e0], wm[C + e0]};
    ff_acc(t, -p.s, -p.q);
    if (G == 2) {
      const float2 o = s_part[(pass & 1) * T + e0];
      ff_acc(t, -o.x, -o.y);
    }
    return ff_norm(t);
  };

  // sweep 1: h1 = V^T w
  dots_begin(nv);
  for (int k = 0; k < nt; k++) {
    const float* st = acquire(k);
    dots(st, st + 2 * nv * C, chunk_f, count_of(k));
    if (!resident) release(k);
  }
  dots_end(part);
  grid.sync();
  grid_sums(part, nv, s_h1);
  // sweep 2: w' = w - V h1; h2 = V^T w', ||w'||^2.  w' stays out of the ring's
  // w rows (the copies of later tiles write there) unless the tiles stay.
  float2* part2 = part + (size_t)kArnDots * nblk;
  dots_begin(nv + 1);
  for (int q = 0; q < nt; q++) {
    const int k = nt - 1 - q, c = resident ? k : nt + q;
    float* st = resident ? s_ring + (size_t)(k % stages) * stage_f : acquire(c);
    float* wt = st + 2 * nv * C;
    float* wn = resident ? wt : s_w + (q & 1) * 2 * T;
    const int wstride = resident ? chunk_f : 2 * C;
    const int count = count_of(k);
    FF p[M];
    share(st, true, q, p);
    if (!half) {
#pragma unroll
      for (int m = 0; m < M; m++) {
        const int e = e0 + C * m;
        const FF t = minus(wt + m * chunk_f, q, p[m]);
        wn[m * wstride + e0] = t.s;
        wn[m * wstride + C + e0] = t.q;
        if (!resident && e < count) {
          const long long g = tile_of(k) * T + e;
          w[g] = t.s;
          w[ld + g] = t.q;
        }
      }
    }
    bar_consumers();
    dots(st, wn, wstride, count);
    if (!resident) release(c);
  }
  if (!resident) fence_proxy_async();  // the third sweep's copies read the w' written here
  dots_end(part2);
  grid.sync();
  grid_sums(part2, nv + 1, s_h2);
  if (wid == 0) {
    double t = lane < nv ? s_h2[lane] * s_h2[lane] : 0.0;
    t = warp_sum(t);
    if (lane == 0) {
      const double w2 = s_n2, n2 = w2 - t;
      s_slow = !(t <= kArnSmallH2 * w2) || !(n2 > 0.0);
      s_n2 = n2;
      s_inv = n2 > 0.0 ? 1.0 / sqrt(n2) : 0.0;
    }
  }
  bar_all();
  const bool slow = s_slow != 0;
  // V_nv = (w' - V h2) / ||w''||, and the next operator's FP32 input fp32(D V_nv)
  auto put = [&](long long g, const FF& t, float ih, float il, float d) {
    const FF u = ff_norm(ff_mul(t.s, t.q, ih, il));
    vnext[g] = u.s;
    vnext[ld + g] = u.q;
    if (xf) xf[g] = u.s * d;
  };
  const bool scaled = xf && dh;
  // resident tiles still hold V's pairs
  const bool pairs3 = slow || resident;
  const float ih = (float)s_inv, il = (float)(s_inv - (double)ih);
  FF nacc{0.f, 0.f};
  for (int k = 0; k < nt; k++) {
    const int c = 2 * nt + k, count = count_of(k);
    const float* st = resident ? s_ring + (size_t)(k % stages) * stage_f : acquire(c);
    float dv[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
      const int e = e0 + C * m;
      dv[m] = 1.f;
      if (!half && scaled && !slow && e < count)
        dv[m] = resident ? dh[tile_of(k) * T + e] : st[m * chunk_f + nv * C + e0];
    }
    FF p[M];
    share(st, pairs3, k, p);
    if (!half) {
#pragma unroll
      for (int m = 0; m < M; m++) {
        const int e = e0 + C * m;
        const FF t = minus(st + 2 * nv * C + m * chunk_f, k, p[m]);
        if (e < count) {
          const long long g = tile_of(k) * T + e;
          if (slow) {
            w[g] = t.s;
            w[ld + g] = t.q;
            ff_dot_acc(nacc, t.s, t.q, t.s, t.q);
          } else {
            put(g, t, ih, il, dv[m]);
          }
        }
      }
    }
    if (!resident) release(c);
  }
  if (!slow) return;
  // the second projection counts: the norm from the remainder's sum itself
  float2* part3 = part2 + (size_t)kArnDots * nblk;
  dots_n = 1;
  dots_p = 1;
  dots_g = kArnWarps;
#pragma unroll
  for (int r = 0; r < kArnRounds; r++) acc[r] = r == 0 ? nacc : FF{0.f, 0.f};
  dots_end(part3);
  grid.sync();
  if (wid == 0) {
    FF t{0.f, 0.f};
    for (int b = lane; b < nblk; b += 32) {
      const float2 q = __ldcg(part3 + b);
      ff_acc(t, q.x, q.y);
    }
    t = ff_norm(ff_warp_sum(t));
    if (lane == 0) {
      s_n2 = (double)t.s + (double)t.q;
      s_inv = s_n2 > 0.0 ? 1.0 / sqrt(s_n2) : 0.0;
    }
  }
  bar_all();
  if (half) return;
  const float jh = (float)s_inv, jl = (float)(s_inv - (double)jh);
  for (int k = 0; k < nt; k++)
    for (int m = 0; m < M; m++) {
      const int e = e0 + C * m;
      const long long g = tile_of(k) * T + e;
      if (e < count_of(k)) put(g, FF{w[g], w[ld + g]}, jh, jl, scaled ? dh[g] : 1.f);
    }
}

// pair stream length of an n-element Krylov vector
__host__ __device__ __forceinline__ long long ff_ld(long long n) { return (n + 3) & ~3LL; }

// rows x cols FP32 array with `pitch` floats between rows, copied in boxes of
// all rows x `width` columns
bool arn_map(CUtensorMap* m, const float* base, long long cols, long long pitch, int rows, int width) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return false;
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  }
  const cuuint64_t dim[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, stride[1] = {(cuuint64_t)pitch * sizeof(float)};
  const cuuint32_t box[2] = {(cuuint32_t)width, (cuuint32_t)rows}, one[2] = {1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dim, stride, box, one,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int T>
cudaError_t launch_arnoldi_t(cudaStream_t s, int ctas, long long n, const float* V, float* w, int nv,
                             float* vnext, double* d_arn, GmState* gs, int jj, float* xf, const float* dh,
                             uint32_t limit) {
  static unsigned long long ready = 0;             // per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!((ready >> dev) & 1ull)) {
    int per = 0;
    cudaError_t e = cudaFuncSetAttribute(k_arnoldi_tile<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kArnSmem);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_arnoldi_tile<T>, kArnBlock, kArnSmem);
    if (e != cudaSuccess) return e;
    if (per < 2) return cudaErrorLaunchOutOfResources;
    ready |= 1ull << dev;
  }
  const long long tiles = (n + T - 1) / T;
  const unsigned g = (unsigned)std::max<long long>(1, std::min<long long>(ctas, tiles));
  const size_t stage = sizeof(float) * 2 * T * (size_t)(nv + 1);
  const long long most = (tiles + g - 1) / g;  // tiles of a CTA
  int stages = (int)std::min<long long>({(long long)kArnMaxStages, (long long)(arn_ring(T) / stage), most});
  long long ld = ff_ld(n);
  float2* part = reinterpret_cast<float2*>(d_arn);
  ArnMaps maps;
  const int width = std::min(T, kArnCons);
  if (!arn_map(&maps.v, V, ld, ld, 2 * nv, width) || !arn_map(&maps.h, V, ld, 2 * ld, nv, width) ||
      !arn_map(&maps.w, w, ld, ld, 2, width))
    return cudaErrorInvalidValue;
  void* args[] = {&maps, &n, &ld, &w, &nv, &vnext, &part, &gs, &jj, &xf, &dh, &stages, &limit};
  return cudaLaunchCooperativeKernel((const void*)k_arnoldi_tile<T>, dim3(g), dim3(kArnBlock), args,
                                     stage * stages + arn_extra(T), s);
}

// Tile length: the longest of 1024, 512, 256, 128 elements at which a CTA's ring
// holds kArnMinStages tiles and, above 128, every CTA gets 4 (a tile costs a
// barrier or two and the warps' latency: short bases need long tiles, short
// vectors need tiles for every SM).  tile, ctas: force a length, bound the grid
// (0: by the rules).
constexpr int kArnMinStages = 2;
bool arn_fits(int T, int nv) {
  return nv + 1 <= kArnDots && kArnMinStages * sizeof(float) * 2 * T * (size_t)(nv + 1) <= arn_ring(T);
}
cudaError_t launch_arnoldi(cudaStream_t s, long long n, const float* V, float* w, int nv, float* vnext,
                           double* d_arn, GmState* gs, int jj, float* xf, const float* dh,
                           uint32_t limit, int tile = 0, int ctas = 0) {
  static int sms[64] = {0};  // per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (sms[dev] == 0) {
    int v = 0;
    cudaError_t e = cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    sms[dev] = std::min(v, kArnMaxGrid / 2);
  }
  if (nv + 1 > kArnDots) return cudaErrorInvalidValue;
  auto takes = [&](int T) {
    return tile ? tile == T : T == 128 || (arn_fits(T, nv) && n >= 8LL * sms[dev] * T);
  };
  const int g = ctas > 0 ? std::min(ctas, 2 * sms[dev]) : 2 * sms[dev];
  if (takes(1024)) return launch_arnoldi_t<1024>(s, g, n, V, w, nv, vnext, d_arn, gs, jj, xf, dh, limit);
  if (takes(512)) return launch_arnoldi_t<512>(s, g, n, V, w, nv, vnext, d_arn, gs, jj, xf, dh, limit);
  if (takes(256)) return launch_arnoldi_t<256>(s, g, n, V, w, nv, vnext, d_arn, gs, jj, xf, dh, limit);
  return launch_arnoldi_t<128>(s, g, n, V, w, nv, vnext, d_arn, gs, jj, xf, dh, limit);
}

// V0 = r / ||r|| as a pair vector (nrm2: ||r||^2)
__global__ void __launch_bounds__(256) k_start_ff(long long n, const double* __restrict__ r,
                                                  const double* __restrict__ nrm2, float* __restrict__ v,
                                                  float* __restrict__ xf, const float* __restrict__ dh) {
  pdl_wait();
  pdl_next();
  const double sc = *nrm2 > 0.0 ? 1.0 / sqrt(*nrm2) : 0.0;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const double x = r[t] * sc;
    const float h = (float)x;
    v[t] = h;
    v[ff_ld(n) + t] = (float)(x - (double)h);
    if (xf) xf[t] = dh ? h * dh[t] : h;  // the first operator's FP32 input
  }
}

// double vector <-> pair vector
__global__ void __launch_bounds__(256) k_to_ff(long long n, const double* __restrict__ x, float* __restrict__ v) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    const double a = x[t];
    const float h = (float)a;
    v[t] = h;
    v[ff_ld(n) + t] = (float)(a - (double)h);
  }
}
__global__ void __launch_bounds__(256) k_from_ff(long long n, const float* __restrict__ v, double* __restrict__ x) {
  pdl_wait();
  pdl_next();
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    x[t] = (double)v[t] + (double)v[ff_ld(n) + t];
}

// x += D sum_i y_i V_i with y of the least-squares state, V pair vectors, D as pairs (or
// none); at most NVM vectors (the loads of all of them are issued before the pair
// sums).  Every CTA solves for y itself (a launch less); xs (optional): the new x as
// pairs, the input of the residual's operator; eo (optional): en + x, E^{n+theta}.
template <int NVM>
__global__ void __launch_bounds__(256) k_combine_ff(long long n, const float* __restrict__ V,
                                                    const GmState* __restrict__ S,
                                                    const float* __restrict__ dff, double* __restrict__ x,
                                                    float* __restrict__ xs, const double* __restrict__ en,
                                                    double* __restrict__ eo) {
  pdl_wait();
  pdl_next();
  __shared__ float s_y[kMaxV][2];
  __shared__ double s_yd[kMaxV];
  const long long ld = ff_ld(n);
  const int nv = min(S->jj, NVM);
  gm_solve(S, s_yd);
  if (threadIdx.x < kMaxV) {
    const double v = threadIdx.x < nv ? s_yd[threadIdx.x] : 0.0;
    s_y[threadIdx.x][0] = (float)v;
    s_y[threadIdx.x][1] = (float)(v - (double)s_y[threadIdx.x][0]);
  }
  __syncthreads();
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x) {
    float vh[NVM], vl[NVM];
#pragma unroll
    for (int i = 0; i < NVM; i++)
      if (i < nv) {
        vh[i] = V[2 * (size_t)i * ld + t];
        vl[i] = V[2 * (size_t)i * ld + ld + t];
      }
    FF a{0.f, 0.f};
#pragma unroll
    for (int i = 0; i < NVM; i++)
      if (i < nv) {
        const FF u = ff_mul(vh[i], vl[i], s_y[i][0], s_y[i][1]);
        ff_acc(a, u.s, u.q);
      }
    a = ff_norm(a);
    if (dff) a = ff_mul(a.s, a.q, dff[t], dff[n + t]);
    const double v = x[t] + ff_value(a);
    x[t] = v;
    if (eo) eo[t] = en[t] + v;
    if (xs) {
      const float h = (float)v;
      xs[t] = h;
      xs[n + t] = (float)(v - (double)h);
    }
  }
}

void launch_combine_ff(cudaStream_t s, unsigned gr, long long n, const float* V, const GmState* S, int nv_host,
                       const float* dff, double* x, float* xs, const double* en, double* eo) {
  if (nv_host <= 4)
    launch_pdl(k_combine_ff<4>, dim3(gr), dim3(256), 0, s, n, V, S, dff, x, xs, en, eo);
  else if (nv_host <= 8)
    launch_pdl(k_combine_ff<8>, dim3(gr), dim3(256), 0, s, n, V, S, dff, x, xs, en, eo);
  else if (nv_host <= 16)
    launch_pdl(k_combine_ff<16>, dim3(gr), dim3(256), 0, s, n, V, S, dff, x, xs, en, eo);
  else
    launch_pdl(k_combine_ff<32>, dim3(gr), dim3(256), 0, s, n, V, S, dff, x, xs, en, eo);
}

// xf = fp32(D v)
__global__ void __launch_bounds__(256) k_in_f32(long long n, OpIn in, float* __restrict__ xf) {
  pdl_wait();
  pdl_next();
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    xf[t] = in.vd ? (float)in.vd[t] : (in.dh ? in.vh[t] * in.dh[t] : in.vh[t]);
}

// w = A (D v) with the identity part in pairs and the rest (curl-curl and
// mass-matrix terms, a small fraction of A on ECSIM time steps) in FP32
// arithmetic: the inner operator of the refined GMRES, which never decides
// convergence.  xf = fp32(D v).
__global__ void __launch_bounds__(32 * kOpGroups) k_matvec32_ff(long long ncor, const int* __restrict__ nbr,
                                                                  const float* __restrict__ M,
                                                                  const float* __restrict__ xf, OpIn in,
                                                                  float* __restrict__ wh, float* __restrict__ wl,
                                                                  const __grid_constant__ TapsF T) {
  pdl_wait();
  pdl_next();
  __shared__ float s_row[3][kOpGroups][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const long long c = (long long)blockIdx.x * 32 + lane;
  int b, i, j, k;
  corner_ijk(c, b, i, j, k);
  for (int g = wid; g < kOpGroups; g += warps) {
    float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll 4
    for (int s = g; s < 27; s += kOpGroups) {
      int di, dj, dk;
      slot_offset(s, di, dj, dk);
      const int nb = local_id(nbr, b, i + di, j + dj, k + dk);
      float x[3], m[9];
#pragma unroll
      for (int q = 0; q < 3; q++) x[q] = xf[q * ncor + nb];
#pragma unroll
      for (int e = 0; e < 9; e++) m[e] = M[(size_t)(9 * s + e) * ncor + c];
#pragma unroll
      for (int p = 0; p < 3; p++)
#pragma unroll
        for (int q = 0; q < 3; q++) acc[p] = fmaf(fmaf(T.f, m[3 * p + q], T.K[p][q][s]), x[q], acc[p]);
    }
#pragma unroll
    for (int p = 0; p < 3; p++) s_row[p][g][lane] = acc[p];
  }
  __syncthreads();
  for (int p = wid; p < 3; p += warps) {
    float a = 0.f;
#pragma unroll
    for (int g = 0; g < kOpGroups; g++) a += s_row[p][g][lane];
    const long long t = p * ncor + c;
    FF y = opin_value(in, t);
    ff_acc(y, a, 0.f);
    y = ff_norm(y);
    wh[t] = y.s;
    wl[t] = y.q;
  }
}

// ---- field updates -----------------------------------------------------------
__global__ void __launch_bounds__(256) k_update_b(long long ncor, const int* __restrict__ nbr,
                                                  const double* __restrict__ Eh,
                                                  const double* __restrict__ Bn,
                                                  double* __restrict__ Bnew, double c4x,
                                                  double c4y, double c4z, double* __restrict__ energy) {
  pdl_wait();
  pdl_next();
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c == 0) *energy = 0.0;  // for k_c2n_update_e
  if (c >= ncor) return;
  int b, i, j, k;
  corner_ijk(c, b, i, j, k);
  double Ex[2][2][2], Ey[2][2][2], Ez[2][2][2];
#pragma unroll
  for (int kk = 0; kk < 2; kk++)
#pragma unroll
    for (int jj = 0; jj < 2; jj++)
#pragma unroll
      for (int ii = 0; ii < 2; ii++) {
        const int id = local_id(nbr, b, i + ii, j + jj, k + kk);
        Ex[ii][jj][kk] = Eh[id];
        Ey[ii][jj][kk] = Eh[ncor + id];
        Ez[ii][jj][kk] = Eh[2 * ncor + id];
      }
  double t0 = 0.0, t1 = 0.0, t2 = 0.0;
#pragma unroll
  for (int ii = 0; ii < 2; ii++)
#pragma unroll
    for (int jj = 0; jj < 2; jj++) {
      t0 += -c4y * (Ez[ii][1][jj] - Ez[ii][0][jj]) + c4z * (Ey[ii][jj][1] - Ey[ii][jj][0]);
      t1 += -c4z * (Ex[ii][jj][1] - Ex[ii][jj][0]) + c4x * (Ez[1][ii][jj] - Ez[0][ii][jj]);
      t2 += -c4x * (Ey[1][ii][jj] - Ey[0][ii][jj]) + c4y * (Ex[ii][1][jj] - Ex[ii][0][jj]);
    }
  Bnew[c] = Bn[c] + t0;
  Bnew[ncor + c] = Bn[ncor + c] + t1;
  Bnew[2 * ncor + c] = Bn[2 * ncor + c] + t2;
}

// Corner B^{n+1} from the 8 cells of a corner, E^{n+1} and the wave energy: one thread
// per corner and cell (one launch: each of the two took 5 us on a small mesh, most of
// it its own start)
__global__ void __launch_bounds__(256) k_c2n_update_e(long long ncor, const int* __restrict__ nbr,
                                                      const double* __restrict__ Bc,
                                                      double* __restrict__ Bcor,
                                                      const double* __restrict__ Eh, double* __restrict__ En,
                                                      double theta, double vol_over_8pi,
                                                      double* __restrict__ energy) {
  pdl_wait();
  pdl_next();
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double en = 0.0;
  if (c < ncor) {
    int b, i, j, k;
    corner_ijk(c, b, i, j, k);
    double t[3] = {0.0, 0.0, 0.0}, b2 = 0.0, e2 = 0.0;
#pragma unroll
    for (int kk = -1; kk <= 0; kk++)
#pragma unroll
      for (int jj = -1; jj <= 0; jj++)
#pragma unroll
        for (int ii = -1; ii <= 0; ii++) {
          const int id = local_id(nbr, b, i + ii, j + jj, k + kk);
#pragma unroll
          for (int d = 0; d < 3; d++) {
            const double v = Bc[d * ncor + id];
            t[d] += v;
            if (ii == 0 && jj == 0 && kk == 0) b2 += v * v;  // cell c itself
          }
        }
#pragma unroll
    for (int d = 0; d < 3; d++) {
      Bcor[d * ncor + c] = t[d] * 0.125;
      const double e = (Eh[d * ncor + c] - (1.0 - theta) * En[d * ncor + c]) / theta;
      En[d * ncor + c] = e;
      e2 += e * e;
    }
    en = (e2 + b2) * vol_over_8pi;
  }
  __shared__ double s[8];
  en = warp_sum(en);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = en;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += s[w];
    atomicAdd(energy, t);
  }
}

__global__ void __launch_bounds__(256) k_add(long long n, const double* __restrict__ a,
                                             const double* __restrict__ b, double* __restrict__ o) {
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n;
       t += (long long)gridDim.x * blockDim.x)
    o[t] = a[t] + b[t];
}

unsigned grid1(long long n) { return (unsigned)((n + 255) / 256); }
// sweep/reduction grid: at least ept elements per thread, at most cap CTAs
unsigned gridr(long long n, int cap = kRedBlocks, int ept = 4) {
  long long g = (n + 256LL * ept - 1) / (256LL * ept);
  if (g > cap) g = cap;
  return (unsigned)(g < 1 ? 1 : g);
}

}  // namespace

// ============================================================================
// FP32 pair split of an operator input into the context's scratch.  d_xs is also where k_start_ff / k_arnoldi_tile
// leave the FP32 input of the next Krylov vector's operator application: this
// split, k_rhs and the AMR operators overwrite it, so none of them may run
// between an Arnoldi step and the operator application that follows it.
static cudaError_t split_input(amps_gpu_ctx* c, const double* x, const double* dinv) {
  const long long n = 3 * c->nvc;
  if (!c->d_xs) {
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&c->d_xs), sizeof(float) * 2 * n);
    if (e != cudaSuccess) return e;
  }
  launch_pdl(k_split, dim3(gridr(n)), dim3(256), 0, c->stream, n, x, dinv, c->d_xs, c->d_xs + n);
  return cudaGetLastError();
}

cudaError_t launch_matvec(amps_gpu_ctx* c, const double* x, const double* dinv, double* y, bool pairs) {
  if (c->amr) return launch_amr_matvec(c, x, dinv, y, pairs);
  const TapsFF T = taps_ff(make_taps(c->cfg, true));
  TimedLaunch t(c, "matvec", pairs ? 1 : 2);
  cudaError_t e = pairs ? cudaSuccess : split_input(c, x, dinv);
  if (e != cudaSuccess) return e;
  const long long n = 3 * c->ncor;
  launch_pdl(k_matvec, dim3((unsigned)(c->ncor / 32)), dim3(c->tune_tb), 0, c->stream, c->ncor, c->d_nbr,
             c->d_M, c->d_xs, c->d_xs + n, y, T);
  return cudaGetLastError();
}

cudaError_t launch_in_f32(amps_gpu_ctx* c, const OpIn& in, float* xf) {
  const long long n = 3 * c->nvc;
  launch_pdl(k_in_f32, dim3(gridr(n)), dim3(256), 0, c->stream, n, in, xf);
  return cudaGetLastError();
}

cudaError_t launch_matvec32_ff(amps_gpu_ctx* c, const OpIn& in, float* wh, float* wl) {
  if (c->amr) return launch_amr_matvec32_ff(c, in, wh, wl);
  const long long n = 3 * c->ncor;
  if (!c->d_xs) {
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&c->d_xs), sizeof(float) * 2 * n);
    if (e != cudaSuccess) return e;
  }
  const TapsF T = taps_f32(make_taps(c->cfg, false));
  TimedLaunch t(c, "matvec32", in.xf_ready ? 1 : 2);
  cudaError_t e = in.xf_ready ? cudaSuccess : launch_in_f32(c, in, c->d_xs);
  if (e != cudaSuccess) return e;
  launch_pdl(k_matvec32_ff, dim3((unsigned)(c->ncor / 32)), dim3(c->tune_tb), 0, c->stream, c->ncor,
             c->d_nbr, c->d_M, c->d_xs, in, wh, wl, T);
  return cudaGetLastError();
}

cudaError_t launch_rhs(amps_gpu_ctx* c, bool diag) {
  if (c->amr) return launch_amr_rhs(c, diag);
  const TapsFF T = taps_ff(make_taps(c->cfg, false));
  double c4[3];
  for (int d = 0; d < 3; d++) c4[d] = 0.25 * (c->cfg.dt / c->cfg.dx[d] * c->cfg.theta);
  TimedLaunch t(c, "rhs", 2);
  cudaError_t e = split_input(c, c->d_En, nullptr);
  if (e != cudaSuccess) return e;
  const long long n = 3 * c->ncor;
  launch_pdl(k_rhs, dim3((unsigned)(c->ncor / 32)), dim3(c->tune_tb), 0, c->stream, c->ncor, c->d_nbr,
             c->d_M, c->d_xs, c->d_xs + n, c->d_Bc, c->d_J, c->d_rhs, T, c4[0], c4[1], c4[2]);
  return cudaGetLastError();
}

cudaError_t launch_jacobi_diag(amps_gpu_ctx* c) {
  if (c->amr) return launch_amr_jacobi(c);
  Taps T = make_taps(c->cfg, true);
  TimedLaunch t(c, "jacobi");
  k_jacobi<<<grid1(c->ncor), 256, 0, c->stream>>>(c->ncor, c->d_M, c->d_dinv, c->d_dff, T.K[0][0][0],
                                                   T.K[1][1][0], T.K[2][2][0], T.f);
  return cudaGetLastError();
}

cudaError_t launch_update_b(amps_gpu_ctx* c) {
  if (c->amr) return launch_amr_update_b(c);
  double c4[3];
  for (int d = 0; d < 3; d++) c4[d] = 0.25 * (c->cfg.dt / c->cfg.dx[d]);
  TimedLaunch t(c, "update_b");
  launch_pdl(k_update_b, dim3(grid1(c->ncor)), dim3(256), 0, c->stream, c->ncor, c->d_nbr, c->d_Eh, c->d_Bc,
             c->d_Bc2, c4[0], c4[1], c4[2], c->d_energy + 1);
  return cudaGetLastError();
}

// after launch_update_b, which clears the wave energy
cudaError_t launch_c2n_update_e(amps_gpu_ctx* c, const double* Bcen, double* Bcor) {
  if (c->amr) {
    const cudaError_t e = launch_amr_c2n(c, Bcen, Bcor);
    return e == cudaSuccess ? launch_amr_update_e(c) : e;
  }
  const double vol = c->cfg.dx[0] * c->cfg.dx[1] * c->cfg.dx[2];
  TimedLaunch t(c, "update_e");  // C2N with it
  launch_pdl(k_c2n_update_e, dim3(grid1(c->ncor)), dim3(256), 0, c->stream, c->ncor, c->d_nbr, Bcen, Bcor,
             c->d_Eh, c->d_En, c->cfg.theta, vol / (8.0 * kPi), c->d_energy + 1);
  return cudaGetLastError();
}

// GMRES(m) with right preconditioning, CGS2 Arnoldi, Givens rotations on the
// device, and iterative refinement across restarts: every cycle starts from
// the true FP64 residual r = b - A x, its Arnoldi steps apply the operator with
// its identity part in FP64 and the rest in FP32 (c->inner_fp32), and the solve
// ends when the FP64 residual satisfies ||b - A x|| <= tol ||b||.  The
// preconditioner is none (precond 0), Jacobi (1, z = D v) or the learned block
// network (2, z = D v + N(D v); flexible form: the directions z_j are kept).
// Each Arnoldi step is the operator plus one cooperative kernel (k_arnoldi_tile:
// CGS2, normalisation and the Givens update).  The host does not wait for each
// step: it queues as many Arnoldi steps as the last cycle took before it first
// reads the device's convergence flag, then one step per read; steps queued
// past convergence leave the least-squares state untouched (gm_update is
// frozen), so they cost time but not accuracy.
// Device scratch layout of d_red: [0, kRedBlocks*kMaxV) partials, ||r||^2, GmState at
// kGmOffset, the tolerance at kTolOffset.
amps_gpu_status gmres_solve(amps_gpu_ctx* c, double tol, int maxit, int precond,
                            amps_gpu_solve_stats* st, bool* eh_done) {
  const long long n = 3 * c->nvc;
  const int m = std::min(c->restart, kMaxV);
  double* partial = c->d_red;
  double* d_n2 = c->d_red + kRedBlocks * kMaxV;
  GmState* gs = reinterpret_cast<GmState*>(c->d_red + kGmOffset);
  const unsigned gr = gridr(n, c->tune_red, c->tune_ept);
  cudaStream_t s = c->stream;
  cudaError_t e;
#define CK(x)                                                   \
  do {                                                          \
    e = (x);                                                    \
    if (e != cudaSuccess) return cuda_check(c, e, #x);          \
  } while (0)

  if (!c->d_arn)
    CK(cudaMalloc(reinterpret_cast<void**>(&c->d_arn), sizeof(double) * 3 * kArnMaxGrid * kMaxV));
  const double* dinv = precond >= 1 ? c->d_dinv : nullptr;
  const bool flexible = precond == 2;
  if (flexible && !c->d_Z)
    return set_err(c, AMPS_GPU_INVALID_ARG, "learned preconditioner: no network loaded");
  // Krylov vectors V_j and the operator output w are FP32 pair vectors (the
  // bytes of d_V / d_w); the Jacobi scaling is used as pairs
  float* Vf = reinterpret_cast<float*>(c->d_V);
  float* wf = reinterpret_cast<float*>(c->d_w);
  const long long ld = ff_ld(n);
  auto vf = [&](int j) { return Vf + 2 * (size_t)j * ld; };
  const float* dh = nullptr;
  const float* dl = nullptr;
  if (dinv) {
    if (!c->d_dff) CK(cudaMalloc(reinterpret_cast<void**>(&c->d_dff), sizeof(float) * 2 * n));
    dh = c->d_dff;
    dl = c->d_dff + n;
  }
  const bool harvest = precond == 1 && c->pn;
  if ((flexible || harvest || !c->inner_fp32) && !c->d_tmpv)
    CK(cudaMalloc(reinterpret_cast<void**>(&c->d_tmpv), sizeof(double) * 2 * n));
  // w = A (D v_j), or A z_j for the flexible directions, as pairs
  // the FP32 operator input of the next Krylov vector is written by the step
  // that makes the vector (k_start_ff, k_arnoldi_tile) when the operator takes V
  // directly (no learned directions, FP32 inner operator)
  // (nothing that writes d_xs -- split_input, k_rhs, the AMR operators -- runs
  // between a step that writes it and the inner_matvec that reads it)
  const bool pre_xf = !flexible && c->inner_fp32;
  if (!c->d_xs) CK(cudaMalloc(reinterpret_cast<void**>(&c->d_xs), sizeof(float) * 2 * n));
  float* xf_next = pre_xf ? c->d_xs : nullptr;
  auto inner_matvec = [&](int jj, const double* zj, bool zf) -> cudaError_t {
    if (c->inner_fp32) {
      OpIn in{};
      if (zj) {
        in.vd = zj;
        in.xf_ready = zf;  // the network left fp32(z) in d_xs
      } else {
        in.vh = vf(jj);
        in.vl = vf(jj) + ld;
        in.dh = dh;
        in.dl = dl;
        in.xf_ready = pre_xf;
      }
      return launch_matvec32_ff(c, in, wf, wf + ld);
    }
    // FP64 inner operator, through FP64 copies
    const double* x = zj;
    if (!zj) {
      launch_pdl(k_from_ff, dim3(gr), dim3(256), 0, s, n, vf(jj), c->d_tmpv);
      x = c->d_tmpv;
    }
    cudaError_t ee = launch_matvec(c, x, zj ? nullptr : dinv, c->d_tmpv + n);
    if (ee != cudaSuccess) return ee;
    k_to_ff<<<gr, 256, 0, s>>>(n, c->d_tmpv + n, wf);
    return cudaGetLastError();
  };
  double* w = c->d_w;  // between cycles: the FP64 residual
  // the Jacobi scaling, x0 = 0, r0 = b, ||b|| and the first cycle's state
  auto prologue = [&]() -> cudaError_t {
    if (dinv) {
      cudaError_t ee = launch_jacobi_diag(c);
      if (ee != cudaSuccess) return ee;
    }
    launch_pdl(k_first, dim3(gr), dim3(256), 0, s, n, c->d_rhs, w, c->d_x, partial, d_n2, gs,
               c->d_red + kTolOffset);
    return cudaGetLastError();
  };
  // Arnoldi step jj: the operator (after the network for flexible directions),
  // then the cooperative CGS2 + normalisation + Givens step
  auto arnoldi_step = [&](int jj) -> cudaError_t {
    const int nv = jj + 1;
    cudaError_t ee;
    if (flexible) {
      double* zj = c->d_Z + (size_t)jj * n;
      launch_pdl(k_from_ff, dim3(gr), dim3(256), 0, s, n, vf(jj), c->d_tmpv);  // v_j in FP64 for the network
      bool zf = false;
      if ((ee = launch_precond_net(c, c->d_tmpv, zj, c->d_xs, &zf)) != cudaSuccess) return ee;
      if ((ee = inner_matvec(jj, zj, zf)) != cudaSuccess) return ee;
    } else {
      if ((ee = inner_matvec(jj, nullptr, false)) != cudaSuccess) return ee;
      // training pairs for the learned preconditioner: (A D v_j, D v_j)
      if (harvest) {
        launch_pdl(k_from_ff, dim3(gr), dim3(256), 0, s, n, wf, c->d_tmpv);
        launch_pdl(k_from_ff, dim3(gr), dim3(256), 0, s, n, vf(jj), c->d_tmpv + n);
        if ((ee = precond_harvest_pairs(c, c->d_tmpv, c->d_tmpv + n, 1)) != cudaSuccess) return ee;
      }
    }
    TimedLaunch t(c, "gmres_orth");
    return launch_arnoldi(s, n, Vf, wf, nv, vf(nv), c->d_arn, gs, jj, xf_next, dh, c->wait_limit);
  };
  // end of a cycle of at most nv_max steps: least squares, x += (D) V y (with its pairs
  // in d_xs and E^{n+theta} = E^n + x), the true FP64 residual into w and its squared
  // norm into d_n2
  auto cycle_end = [&](int nv_max) -> cudaError_t {
    if (flexible) {
      k_gm_solve<<<1, 256, 0, s>>>(gs);
      k_combine<<<gr, 256, 0, s>>>(n, c->d_Z, gs->y, kMaxV, &gs->jj, nullptr, c->d_x);
    } else {
      launch_combine_ff(s, gr, n, Vf, gs, nv_max, dinv ? c->d_dff : nullptr, c->d_x, c->d_xs, c->d_En, c->d_Eh);
    }
    cudaError_t ee = cudaGetLastError();
    if (ee == cudaSuccess) ee = launch_matvec(c, c->d_x, nullptr, w, !flexible);
    if (ee != cudaSuccess) return ee;
    launch_pdl(k_residual, dim3(gr), dim3(256), 0, s, n, c->d_rhs, w, partial, d_n2, gs);
    return cudaGetLastError();
  };

  const GmStatus& stat = *reinterpret_cast<const GmStatus*>(c->h_red);  // after its copy
  // every read of the step count carries the steps' timeouts
  auto gave_up = [&]() {
    return set_err(c, AMPS_GPU_DEVICE_TIMEOUT,
                   "field solve: " + std::to_string(stat.timeouts) + " bounded waits of the Arnoldi step ran out");
  };
  if (c->red_tol != tol) {  // zero at creation, when no solve's tolerance is
    CK(cudaMemcpyAsync(c->d_red + kTolOffset, &tol, sizeof(double), cudaMemcpyHostToDevice, s));
    c->red_tol = tol;
  }
  int it = 0, cycles = 0;
  bool conv = false;
  double rel = 0.0, bnorm = 0.0, beta = 0.0;
  // The first cycle as one CUDA graph when the previous solve with this
  // preconditioner tells how many Arnoldi steps to queue (K): prologue, ||b||
  // and the cycle start on the device, K steps, the cycle end, one read of
  // (steps used, converged, ||b||^2, ||r||^2).  Steps past convergence are
  // frozen; a cycle that needed more than K steps ends as a restart.  Later
  // cycles run as below.
  const int K = std::max(1, std::min({c->gm_guess[precond], m, maxit}));
  const bool graph = c->use_graphs && !c->timing && !flexible && !harvest && c->inner_fp32 &&
                     c->gm_guess[precond] > 0 && !c->solve_graphs_off;
  bool graph_done = false;
  if (graph) {
    cudaGraphExec_t exec = nullptr;
    for (auto& g : c->solve_graphs)
      if (g.precond == precond && g.steps == K && g.tb == c->tune_tb && g.red == c->tune_red &&
          g.ept == c->tune_ept)
        exec = g.exec;
    if (!exec) {
      cudaGraph_t gr_cap = nullptr;
      cudaError_t ee = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
      if (ee == cudaSuccess) {
        cudaError_t e1 = prologue();
        if (e1 == cudaSuccess) {
          launch_pdl(k_start_ff, dim3(gr), dim3(256), 0, s, n, w, d_n2, vf(0), xf_next, dh);
          for (int jj = 0; jj < K && e1 == cudaSuccess; jj++) e1 = arnoldi_step(jj);
        }
        if (e1 == cudaSuccess) e1 = cycle_end(K);
        if (e1 == cudaSuccess)
          e1 = cudaMemcpyAsync(c->h_red, &gs->jj, sizeof(GmStatus), cudaMemcpyDeviceToHost, s);
        ee = cudaStreamEndCapture(s, &gr_cap);
        if (ee == cudaSuccess && e1 == cudaSuccess)
          ee = cudaGraphInstantiate(&exec, gr_cap, 0);
        else if (ee == cudaSuccess)
          ee = e1;
        if (gr_cap) cudaGraphDestroy(gr_cap);
      }
      if (ee != cudaSuccess || !exec) {
        // not capturable here: clear the error state of the capture, solve eagerly
        cudaGetLastError();
        c->solve_graphs_off = true;
        exec = nullptr;
      } else {
        if (c->solve_graphs.size() >= 8) {
          cudaGraphExecDestroy(c->solve_graphs.front().exec);
          c->solve_graphs.erase(c->solve_graphs.begin());
        }
        c->solve_graphs.push_back({precond, K, c->tune_tb, c->tune_red, c->tune_ept, exec});
      }
    }
    if (exec) {
      CK(cudaGraphLaunch(exec, s));
      CK(cudaStreamSynchronize(s));
      it = stat.jj;
      cycles = 1;
      bnorm = std::sqrt(stat.bn2);
      beta = std::sqrt(std::max(0.0, stat.rn2));
      if (stat.timeouts) return gave_up();
      graph_done = true;
    }
  }
  if (!graph_done) {
    CK(prologue());
    CK(cudaMemcpyAsync(c->h_red, d_n2, sizeof(double), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    beta = bnorm = std::sqrt(c->h_red[0]);
  }
  while (true) {
    rel = bnorm > 0.0 ? beta / bnorm : 0.0;
    if (rel <= tol) {
      conv = true;
      break;
    }
    if (it >= maxit) break;
    cycles++;
    // the FP32 operators keep the identity part in FP64 accuracy (their noise
    // is ~1e-7 of the off-identity terms), so a cycle runs to the tolerance; a
    // later cycle only corrects what that noise left
    const double target = tol * bnorm;
    // V0 = r / ||r|| (d_n2 holds ||r||^2)
    k_gm_start<<<1, 32, 0, s>>>(gs, d_n2, target);
    launch_pdl(k_start_ff, dim3(gr), dim3(256), 0, s, n, w, d_n2, vf(0), xf_next, dh);
    int launched = 0, used = 0;
    bool done = false;
    const int first_read = cycles == 1 ? std::max(1, std::min(c->gm_guess[precond], m)) : 1;
    while (!done && launched < m && it + launched < maxit) {
      CK(arnoldi_step(launched++));
      CK(cudaGetLastError());
      if (launched >= first_read || launched == m || it + launched >= maxit) {
        CK(cudaMemcpyAsync(c->h_red, &gs->jj, sizeof(GmStatus), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        if (stat.timeouts) return gave_up();
        used = stat.jj;
        done = stat.done != 0;
      }
    }
    it += used;
    CK(cycle_end(used));
    CK(cudaMemcpyAsync(c->h_red, d_n2, sizeof(double), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    beta = std::sqrt(c->h_red[0]);
  }
  *eh_done = cycles > 0 && !flexible;  // cycle_end left E^n + x in d_Eh
  // the next solve's first cycle queues as many steps as this solve took
  if (conv) c->gm_guess[precond] = std::max(1, std::min(it, m));
  // the solve's own pair (b, x)
  if (conv && precond == 1 && c->pn) CK(precond_harvest_pairs(c, c->d_rhs, c->d_x, 0));
#undef CK
  if (st) {
    st->iterations = it;
    st->converged = conv ? 1 : 0;
    st->rel_residual = rel;
  }
  return conv ? AMPS_GPU_OK : AMPS_GPU_GMRES_NOT_CONVERGED;
}

// Autotuner: candidate launch shapes timed with CUDA events on the context
// stream, on scratch vectors (the operator and the sweeps have no side effects
// outside them).  ms[0..2]: operator with 64/128/256 threads per CTA;
// ms[3..5]: one 8-vector combination sweep with 76/152/304 CTAs (4 elements per thread).
amps_gpu_status field_autotune(amps_gpu_ctx* c, double* ms) {
  const long long n = 3 * c->nvc;
  cudaStream_t s = c->stream;
  cudaError_t e;
  cudaEvent_t a, b;
  if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess)
    return set_err(c, AMPS_GPU_CUDA_ERROR, "autotune: events");
  const bool timing = c->timing;
  c->timing = false;
  amps_gpu_status st = AMPS_GPU_OK;
  auto fail = [&](cudaError_t err, const char* what) {
    st = cuda_check(c, err, what);
    return st;
  };
  double* x = c->d_x;
  float* yf = reinterpret_cast<float*>(c->d_w);
  OpIn in{};
  in.vd = x;
  if ((e = cudaMemsetAsync(x, 0, sizeof(double) * n, s)) != cudaSuccess) fail(e, "autotune");
  if ((e = cudaMemsetAsync(c->d_V, 0, sizeof(double) * n * 10, s)) != cudaSuccess) fail(e, "autotune");
  const int tbs[3] = {64, 128, 256};
  double best = 1e30;
  int best_tb = c->tune_tb;
  for (int q = 0; q < 3 && !st; q++) {
    c->tune_tb = tbs[q];
    for (int w = 0; w < 2 && !st; w++)
      if ((e = launch_matvec32_ff(c, in, yf, yf + ff_ld(n))) != cudaSuccess) fail(e, "autotune matvec");
    cudaEventRecord(a, s);
    for (int r = 0; r < 5 && !st; r++)
      if ((e = launch_matvec32_ff(c, in, yf, yf + ff_ld(n))) != cudaSuccess) fail(e, "autotune matvec");
    cudaEventRecord(b, s);
    cudaEventSynchronize(b);
    float t = 0.f;
    cudaEventElapsedTime(&t, a, b);
    if (ms) ms[q] = t / 5.0;
    if (t < best) { best = t; best_tb = tbs[q]; }
  }
  c->tune_tb = best_tb;
  const int caps[3] = {76, 152, 304};
  // the sweep: x += sum of 8 pair vectors times coefficients (k_combine_ff),
  // the shape of the solve's grid-stride vector passes
  GmState* gs = reinterpret_cast<GmState*>(c->d_red + kGmOffset);
  const int eight = 8;
  if ((e = cudaMemsetAsync(gs, 0, sizeof(GmState), s)) != cudaSuccess) fail(e, "autotune");
  if ((e = cudaMemcpyAsync(&gs->jj, &eight, sizeof(int), cudaMemcpyHostToDevice, s)) != cudaSuccess)
    fail(e, "autotune");
  const float* Vf = reinterpret_cast<const float*>(c->d_V);
  best = 1e30;
  int best_cap = c->tune_red;
  for (int q = 0; q < 3 && !st; q++) {
    const unsigned gr = gridr(n, caps[q], 4);
    launch_combine_ff(s, gr, n, Vf, gs, 8, nullptr, x, nullptr, nullptr, nullptr);
    cudaEventRecord(a, s);
    for (int r = 0; r < 5; r++) launch_combine_ff(s, gr, n, Vf, gs, 8, nullptr, x, nullptr, nullptr, nullptr);
    cudaEventRecord(b, s);
    if ((e = cudaEventSynchronize(b)) != cudaSuccess) fail(e, "autotune sweep");
    float t = 0.f;
    cudaEventElapsedTime(&t, a, b);
    if (ms) ms[3 + q] = t / 5.0;
    if (t < best) { best = t; best_cap = caps[q]; }
  }
  c->tune_red = best_cap;
  c->tune_ept = 4;
  c->timing = timing;
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (!st) st = cuda_check(c, cudaGetLastError(), "autotune");
  return st;
}

cudaError_t launch_add(amps_gpu_ctx* c, const double* a, const double* b, double* o, long long n) {
  k_add<<<gridr(n), 256, 0, c->stream>>>(n, a, b, o);
  return cudaGetLastError();
}

// One Arnoldi step on host vectors (as many elements as a tile copy's 32-bit
// coordinate reaches), for checks of k_arnoldi_tile by itself: pairs
// of V and w, a least-squares state whose rotations are the identity (so that its
// column is h and the norm), the step, and everything back.
extern "C" amps_gpu_status amps_gpu_arnoldi_step(int device, long long n, int nv, const double* V, const double* w,
                                                 const double* d, int tile, int ctas, double* h, double* norm,
                                                 double* vnext, float* xf) {
  if (n < kArnCons || n > (1LL << 31) - 2048 || nv < 1 || nv + 1 > kArnDots || !V || !w || !h || !norm || !vnext || !xf || ctas < 0)
    return AMPS_GPU_INVALID_ARG;
  if (tile != 0 && ((tile != 128 && tile != 256 && tile != 512 && tile != 1024) || !arn_fits(tile, nv)))
    return AMPS_GPU_INVALID_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return AMPS_GPU_NO_DEVICE;
  if (device < 0 || device >= ndev) return AMPS_GPU_INVALID_ARG;
  cudaSetDevice(device);
  const long long ld = ff_ld(n);
  const size_t vec = 2 * (size_t)ld * sizeof(float);  // bytes of a pair vector
  cudaStream_t s = nullptr;
  char* mem = nullptr;
  // the basis and V_nv, w, D as a pair vector, one FP64 vector, xf, then the step's scratch
  const size_t arn = sizeof(double) * 3 * kArnMaxGrid * kMaxV, state = (sizeof(GmState) + 63) & ~(size_t)63;
  const size_t bytes = vec * (nv + 5) + arn + state;
  cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&mem), bytes);
  float* dV = reinterpret_cast<float*>(mem);
  float* dvn = dV + 2 * (size_t)nv * ld;
  float* dw = dvn + 2 * ld;
  float* dd = dw + 2 * ld;
  double* d64 = reinterpret_cast<double*>(dd + 2 * ld);
  float* dxf = reinterpret_cast<float*>(d64 + ld);
  double* darn = reinterpret_cast<double*>(mem + vec * (nv + 5));
  GmState* gs = reinterpret_cast<GmState*>(reinterpret_cast<char*>(darn) + arn);
  if (e == cudaSuccess) e = cudaMemsetAsync(mem, 0, bytes, s);
  auto up = [&](const double* src, float* dst) {
    if (e == cudaSuccess) e = cudaMemcpyAsync(d64, src, sizeof(double) * n, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return;
    k_to_ff<<<gridr(n), 256, 0, s>>>(n, d64, dst);
    e = cudaGetLastError();
  };
  for (int i = 0; i < nv; i++) up(V + (size_t)i * n, dV + 2 * (size_t)i * ld);
  up(w, dw);
  if (d) up(d, dd);
  std::vector<GmState> S(1);
  std::fill_n(S[0].cs, kMaxV, 1.0);
  if (e == cudaSuccess) e = cudaMemcpyAsync(gs, S.data(), sizeof(GmState), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = launch_arnoldi(s, n, dV, dw, nv, dvn, darn, gs, nv - 1, dxf, d ? dd : nullptr, kWaitLimit, tile, ctas);
  if (e == cudaSuccess) {
    launch_pdl(k_from_ff, dim3(gridr(n)), dim3(256), 0, s, n, dvn, d64);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(vnext, d64, sizeof(double) * n, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(xf, dxf, sizeof(float) * n, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(S.data(), gs, sizeof(GmState), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(mem);
  if (s) cudaStreamDestroy(s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return AMPS_GPU_CUDA_ERROR;
  }
  const int jj = nv - 1;
  for (int i = 0; i < jj; i++) h[i] = S[0].H[i * kMaxV + jj];
  h[jj] = S[0].H[jj * kMaxV + jj] * S[0].cs[jj];
  *norm = S[0].H[jj * kMaxV + jj] * S[0].sn[jj];
  return S[0].timeouts ? AMPS_GPU_DEVICE_TIMEOUT : AMPS_GPU_OK;
}
