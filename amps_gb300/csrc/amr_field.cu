// ECSIM field kernels on block-structured AMR meshes (FP64), and the AMR
// variants of the particle import/export and stencil packing.
//
// The operator is assembled per cell in weak form (each term times the cell
// volume V): identity/8, (theta c dt)^2 C^T C with C the face-average curl of
// UpdateB (pic_field_solver_ecsim.cpp:5160-5711) whose transpose is the curl B
// of the RHS supports (src/pic/ecsim/get_stencil.cpp:1500-1599), and
// 4 pi theta dt M from the per-cell mass-matrix partials of ProcessCell
// (:1882-2438).  Corners of fine blocks that lie on a coarser block's face or
// edge off its corner lattice are hanging: they take the interpolation of the
// coarse corners (P), contributions to them are scattered to the parents (P^T),
// and their rows read x_h - (P x)_h = 0.  On a uniform mesh this is the
// reference operator times V.  Tiles of cells, atomics for the scatter to the (up
// to 8) cells sharing a corner.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "deposit_core.cuh"

namespace {

constexpr double kPi = 3.14159265358979323846264338327950288;
// offset bit d of corner c of a cell, in the order (x, y) = (0,0) (1,0) (1,1) (0,1)
// on the lower face, then on the upper
__host__ __device__ constexpr int off_bit(int c, int d) {
  return d == 0 ? (((c + 1) >> 1) & 1) : (d == 1 ? ((c >> 1) & 1) : (c >> 2));
}

struct Hang {
  const int* hs;
  const int* hp;
  const double* hw;
  const float* hwh;  // hw as FP32 pairs
  const float* hwl;
  // boundary rows of meshes with open axes (bflag null: none): row b reads
  // x_b - sum_{t in [bs[b], bs[b+1])} bw[t] x_{bc[t]}
  const int* bflag;
  const int* bs;
  const int* bc;
  const double* bw;
  const float* bwh;
  const float* bwl;
};
__device__ __forceinline__ bool is_bnd(const Hang& h, long long c) { return h.bflag && h.bflag[c]; }

// value of corner c of a component-major field (component d), P applied,
// optionally scaled by a diagonal (right preconditioner)
__device__ __forceinline__ double cval(const double* __restrict__ F, const double* __restrict__ dinv,
                                       long long nvc, int c, int d, const Hang& h) {
  const int s = h.hs[c], e = h.hs[c + 1];
  if (s == e) return dinv ? dinv[d * nvc + c] * F[d * nvc + c] : F[d * nvc + c];
  double v = 0.0;
  for (int t = s; t < e; t++) {
    const int p = h.hp[t];
    v += h.hw[t] * (dinv ? dinv[d * nvc + p] * F[d * nvc + p] : F[d * nvc + p]);
  }
  return v;
}

template <typename T>
__device__ __forceinline__ void cell_curl(const T e[8][3], T q, T cu[3]) {
  T a = 0, b = 0, c = 0, d = 0, f = 0, g = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const bool px = k == 1 || k == 2 || k == 5 || k == 6;
    const bool py = k == 2 || k == 3 || k == 6 || k == 7;
    const bool pz = k >= 4;
    a += py ? e[k][2] : -e[k][2];
    b += pz ? e[k][1] : -e[k][1];
    c += pz ? e[k][0] : -e[k][0];
    d += px ? e[k][2] : -e[k][2];
    f += px ? e[k][1] : -e[k][1];
    g += py ? e[k][0] : -e[k][0];
  }
  cu[0] = q * (a - b);
  cu[1] = q * (c - d);
  cu[2] = q * (f - g);
}

// out[k] += component p of s C^T y on the 8 corners
template <typename T>
__device__ __forceinline__ void cell_curl_t_row(const T y[3], T s, int p, T out[8]) {
  const T a0 = s * y[0], a1 = s * y[1], a2 = s * y[2];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const bool px = k == 1 || k == 2 || k == 5 || k == 6;
    const bool py = k == 2 || k == 3 || k == 6 || k == 7;
    const bool pz = k >= 4;
    if (p == 0) out[k] += (pz ? a1 : -a1) - (py ? a2 : -a2);
    else if (p == 1) out[k] += (px ? a2 : -a2) - (pz ? a0 : -a0);
    else out[k] += (py ? a0 : -a0) - (px ? a1 : -a1);
  }
}

// per cell size (index log2 of the block's cell size in finest cells): the
// operator's scale factors as FP32 pairs (the FP32 inner operator takes the hi
// halves)
struct LevelK {
  float curl[2], cc[2], id[2], m[2], bb[2];  // 0.25/dx, th2dt2 V 0.25/dx, V/8, f V, thdt V 0.25/dx
  float dg;                                  // V (1/8 + th2dt2 / (8 dx^2)), of the Jacobi diagonal
};
constexpr int kMaxScale = 8;

struct ApplyArgs {
  long long ncell, nvc;
  const int* ctabh;     // block corner -> corner, hanging ones as ~id
  Hang h;
  const int* bscale;
  LevelK lk[kMaxScale];
  float fj[2];          // f as a pair (the current term of the RHS)
  const float* xh;      // ACC 1/2 input as FP32 pairs (the scaling applied)
  const float* xl;
  const float* cellM;
  const float* cellJ;
  const float* xf;      // the same in FP32 (the FP32 inner operator)
  const double* Bcen;   // RHS: centre B (component-major over cells)
  unsigned long long* flags;  // [2]: bounded-wait timeouts
  double* diag;               // RHS: += the Jacobi diagonal of free corners (null: not wanted)
  int* next;                  // tiles handed out beyond the first two per CTA
};

// ---------------------------------------------------------------------------
// The operator per cell (weak form, see above), y += its contributions, on
// tiles of 32 cells (an 8 x 4 x 1 slab of a block: 9 x 5 x 2 corners, 31,104
// contiguous bytes of partials) with 3 threads per cell: warp p takes the 32
// cells' output component p and reads the rows 3p..3p+2 of each cell's 27
// monomial blocks from shared memory (stride 243 words between the lanes'
// cells: conflict-free).
constexpr int kTileCells = 32;
constexpr int kTileThreads = 3 * kTileCells;
constexpr uint32_t kTileBytes = kTileCells * AMPS_CELLM * 4;  // 31,104
constexpr int kTC = 90;  // tile corners, (i, j, k) at i + 9 (j + 5 k)
constexpr int kT32Threads = 2 * kTileThreads;

// The FP32 inner operator (curl-curl + mass; identity added in pairs by
// k_amr_finish_ff).  Bound: reading the partials (478 MB at 491,520 cells).
// Persistent CTAs, three per SM with two tile buffers each.  Three producer warps
// gather a tile's 90 corner values (once each; the corner table carries hanging
// corners as ~id, so the common corner needs no look at the constraint rows) and
// start the bulk copy of its partials as soon as a buffer is free; three consumer
// warps, one output component each, wait for nothing but the buffer.  (With the
// gather in the computing warps and two CTA barriers per tile: 94 us; one tile per
// CTA, which held its buffer through the whole chain of dependent loads: 132; tiles
// of 16 cells, six CTAs per SM: 106, as a tile's chain does not shrink with it.)  The
// cells' contributions to a corner are added by shuffles along x and y, and go out as
// one global reduction per tile corner and component (P^T for hanging ones).
// 491,520 cells: 84 us (5.9 TB/s).
__global__ void __launch_bounds__(kT32Threads) k_amr_tile32(ApplyArgs a, int tiles, float* __restrict__ y32) {
  extern __shared__ __align__(16) float s_m[];  // two tiles of partials
  // tx: a tile's partials have landed; val: its corners are stored (3 warps); empty:
  // the 3 consumer warps have read both
  __shared__ __align__(8) uint64_t tx[2], val[2], empty[2];
  __shared__ float s_x[2][3][kTC];
  __shared__ int s_id[2][kTC];
  const int tid = threadIdx.x, p = tid / 32 % 3, lane = tid & 31;
  const int step = gridDim.x;
  if (tid == 0) {
    for (int q = 0; q < 2; q++) {
      mbar_init(&tx[q], 1);
      mbar_init(&val[q], 3);
      mbar_init(&empty[q], 3);
    }
    fence_mbar_init();
  }
  __syncthreads();
  auto arrive = [&](uint64_t* bar) {
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
  };
  // a wait that runs out is counted, and the warp leaves its loop
  auto wait = [&](uint64_t* bar, int phase) {
    const bool ok = __all_sync(0xffffffffu, mbar_wait_bounded(bar, phase, kWaitLimit)) != 0;
    if (!ok && lane == 0) atomicAdd(a.flags + 2, 1ull);
    return ok;
  };
  if (tid >= kTileThreads) {
    // ---- producers: warp p brings 30 of a tile's 90 corners, the first the partials
    const int t = 30 * p + lane, ti = t % 9, tj = (t / 9) % 5, tk = t / 45;
    const bool act = lane < 30;
    auto corner_id = [&](int tile) {
      if (tile >= tiles || !act) return 0;
      const int b = tile >> 4, l = (tile & 15) * kTileCells;  // 16 tiles per block
      return __ldg(a.ctabh + b * 729 + ti + 9 * (((l >> 3) & 7) + tj + 9 * ((l >> 6) + tk)));
    };
    float x[3] = {0.f, 0.f, 0.f};
    auto corner_values = [&](int id) {
      if (!act) return;
      if (id >= 0) {
#pragma unroll
        for (int d = 0; d < 3; d++) x[d] = a.xf[d * a.nvc + id];
      } else {
        const int h = ~id, s = a.h.hs[h], e = a.h.hs[h + 1];
#pragma unroll
        for (int d = 0; d < 3; d++) x[d] = 0.f;
        for (int r = s; r < e; r++) {
          const float w = a.h.hwh[r];
          const int q = a.h.hp[r];
#pragma unroll
          for (int d = 0; d < 3; d++) x[d] = fmaf(w, a.xf[d * a.nvc + q], x[d]);
        }
      }
    };
    auto copy = [&](int tile, int buf) {
      if (p != 0 || lane != 0) return;
      mbar_arrive_expect_tx(&tx[buf], kTileBytes);
      bulk_copy_g2s(s_m + (size_t)buf * (kTileBytes / 4), a.cellM + (size_t)tile * kTileCells * AMPS_CELLM,
                    kTileBytes, &tx[buf]);
    };
    // the partials don't change within a solve: the first two tiles' before the wait
    for (int q = 0; q < 2; q++)
      if ((int)blockIdx.x + q * step < tiles) copy(blockIdx.x + q * step, q);
    int id = corner_id(blockIdx.x), n = 0;
    pdl_wait();
    pdl_next();
    corner_values(id);
    bool ok = true;
    for (int tile = blockIdx.x; tile < tiles; tile += step, n++) {
      const int buf = n & 1;
      const int idn = corner_id(tile + step);
      if (n >= 2) {
        ok = wait(&empty[buf], ((n >> 1) - 1) & 1);
        if (!ok) break;
        copy(tile, buf);
      }
      if (act) {
        s_id[buf][t] = id;
#pragma unroll
        for (int d = 0; d < 3; d++) s_x[buf][d][t] = x[d];
      }
      arrive(&val[buf]);
      id = idn;
      if (tile + step < tiles) corner_values(id);
    }
    // the last copies land before the CTA's shared memory goes, whoever gave up (n is
    // 0, or the two last copies are of tiles n - 2 and n - 1)
    if (p == 0)
      for (int q = max(0, n - 2); q < n; q++) mbar_wait_bounded(&tx[q & 1], (q >> 1) & 1, kWaitLimit);
    return;
  }
  // ---- consumers: warp p takes component p
  pdl_wait();
  int n = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += step, n++) {
    const int buf = n & 1;
    if (!wait(&val[buf], (n >> 1) & 1) || !wait(&tx[buf], (n >> 1) & 1)) return;
    const LevelK& K = a.lk[min(__ffs(__ldg(a.bscale + (tile >> 4))) - 1, kMaxScale - 1)];
    const int i = lane & 7, j = lane >> 3;
    float e[8][3], out[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
      out[c] = 0.f;
      const int tc = (i + off_bit(c, 0)) + 9 * ((j + off_bit(c, 1)) + 5 * off_bit(c, 2));
#pragma unroll
      for (int d = 0; d < 3; d++) e[c][d] = s_x[buf][d][tc];
    }
    // mass term, monomial by monomial: the ordered corner pairs that share it
    const float* mm = s_m + (size_t)buf * (kTileBytes / 4) + lane * AMPS_CELLM + 3 * p;
#pragma unroll
    for (int mono = 0; mono < 27; mono++) {
      const float m0 = mm[9 * mono], m1 = mm[9 * mono + 1], m2 = mm[9 * mono + 2];
#pragma unroll
      for (int c1 = 0; c1 < 8; c1++)
#pragma unroll
        for (int c2 = 0; c2 < 8; c2++)
          if (pair_monomial(c1, c2) == mono) out[c1] = fmaf(m0, e[c2][0], fmaf(m1, e[c2][1], fmaf(m2, e[c2][2], out[c1])));
    }
    float cu[3];
    cell_curl<float>(e, K.curl[0], cu);
    const float fv = K.m[0];
#pragma unroll
    for (int c = 0; c < 8; c++) out[c] *= fv;
    if (p == 0) cell_curl_t_row<float>(cu, K.cc[0], 0, out);
    else if (p == 1) cell_curl_t_row<float>(cu, K.cc[0], 1, out);
    else cell_curl_t_row<float>(cu, K.cc[0], 2, out);
    // out[c] in the table order (0,0) (1,0) (1,1) (0,1), z: add along x and y
    auto put = [&](int tc, float v) {
      const int q = s_id[buf][tc];
      if (q >= 0) {
        atomicAdd(y32 + p * a.nvc + q, v);
      } else {
        const int h = ~q;
        for (int t = a.h.hs[h]; t < a.h.hs[h + 1]; t++) atomicAdd(y32 + p * a.nvc + a.h.hp[t], a.h.hwh[t] * v);
      }
    };
#pragma unroll
    for (int z = 0; z < 2; z++) {
      const float r0 = __shfl_up_sync(0xffffffffu, out[4 * z + 1], 1);
      const float r1 = __shfl_up_sync(0xffffffffu, out[4 * z + 2], 1);
      const float c0 = out[4 * z] + (i > 0 ? r0 : 0.f);      // corner (i, j)
      const float c1 = out[4 * z + 3] + (i > 0 ? r1 : 0.f);  // corner (i, j + 1)
      const float e0 = out[4 * z + 1], e1 = out[4 * z + 2];  // lanes i = 7: corners (8, j), (8, j + 1)
      const float d0 = __shfl_up_sync(0xffffffffu, c1, 8), d1 = __shfl_up_sync(0xffffffffu, e1, 8);
      put(i + 9 * (j + 5 * z), c0 + (j > 0 ? d0 : 0.f));
      if (i == 7) put(8 + 9 * (j + 5 * z), e0 + (j > 0 ? d1 : 0.f));
      if (j == 3) put(i + 9 * (4 + 5 * z), c1);
      if (i == 7 && j == 3) put(8 + 9 * (4 + 5 * z), e1);
    }
    arrive(&empty[buf]);
  }
}

// Two FP32 pairs side by side (FF in each half of the registers): packed
// instructions halve the issue slots of the error-free sums.
struct FF2 {
  unsigned long long s, q;
};
__device__ __forceinline__ unsigned long long pk(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 upk(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// a += m (xh + xl) in both halves, m exact in FP32, nm = -m: the steps of ff_add
__device__ __forceinline__ void ff2_add(FF2& a, unsigned long long m, unsigned long long nm,
                                        unsigned long long xh, unsigned long long xl) {
  const unsigned long long ph = mul2(m, xh);
  const unsigned long long npl = fma2(nm, xl, fma2(nm, xh, ph));
  const unsigned long long t = add2(a.s, ph);
  const unsigned long long bp = sub2(t, a.s);
  const unsigned long long err = add2(sub2(a.s, sub2(t, bp)), sub2(ph, bp));
  a.s = t;
  a.q = add2(a.q, sub2(err, npl));
}

// The operator (ACC 1) and the RHS (ACC 2) to FP64 accuracy in FP32 pairs (FF,
// common.cuh): FP64 arithmetic is a small fraction of the FP32 rate on this part;
// the pairs carry FP64 accuracy.  Bound: issue and the FP32 pipe (192 error-free
// products of 11 operations per cell and component).  Persistent CTAs as in
// k_amr_tile32 (the next tile's partials, for the RHS also its currents, and its
// corner values are in flight while one is computed), on tiles of 16 cells (8 x 2
// x 1, 9 x 3 x 2 corners): six small CTAs per SM hide each other's barriers, which
// cost three of twice the size half their time.  Tiles are claimed one by one: those
// with hanging corners take longer, and a fixed share per CTA left a fifth of the
// warps idle towards the end (216 us; k_amr_tile32, which waits for memory anyway,
// gains nothing by it); the kernel launched after this one clears the counter.  A
// warp takes one component, a lane one cell's corners of y = 0 or of y = 1; two
// z-neighbours of a corner column share packed instructions: with M_a the monomial
// block of z-sum a, both sums take e(z=0) times (M_0, M_1) and e(z=1) times (M_1,
// M_2).  The cells' sums for a corner are added in pairs by shuffles, and one FP64
// reduction per tile corner and component goes out (from shared memory: in full
// warps, as the conversion is FP64 too).  The RHS also sums the Jacobi diagonal,
// whose entries lie in the staged partials (24 us more; a kernel of its own read half
// of the partials again: 84).  491,520 cells: 191 us (32-cell tiles 230;
// one tile per CTA, scalar pairs and values gathered per cell: 345).
constexpr int kFFCells = 16;
constexpr int kFFCorners = 54;                            // (i, j, k) at i + 9 (j + 3 k)
constexpr uint32_t kFFBytes = kFFCells * AMPS_CELLM * 4;  // 15,552
constexpr uint32_t kFFJBytes = kFFCells * 24 * 4;
template <int ACC>
constexpr uint32_t tile_ff_bytes() { return kFFBytes + (ACC == 2 ? kFFJBytes : 0); }
template <int ACC>
__global__ void __launch_bounds__(kTileThreads, ACC == 2 ? 5 : 6) k_amr_tile_ff(ApplyArgs a, int tiles, double* __restrict__ y64) {
  pdl_wait();
  pdl_next();
  extern __shared__ __align__(16) float s_m[];  // two tiles of partials (and currents)
  constexpr uint32_t kBytes = tile_ff_bytes<ACC>();
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ float4 s_x[3][kFFCorners];  // corner values as pairs (h, h, l, l)
  __shared__ float2 s_cu[3][kFFCells];   // the cell's curl and centre B, a component per warp
  __shared__ float2 s_b[ACC == 2 ? 3 : 1][kFFCells];
  __shared__ float2 s_out[3][kFFCorners];
  __shared__ float2 s_dg[ACC == 2 ? 3 : 1][kFFCorners];
  const int tid = threadIdx.x, p = tid / 32, lane = tid & 31;
  const int set = lane / kFFCells, lc = lane % kFFCells;
  // tiles of this CTA: the first two fixed, then as they are asked for
  __shared__ int s_next;
  auto claim = [&] { return 2 * (int)gridDim.x + atomicAdd(a.next, 1); };
  if (tid == 0) {
    s_next = claim();
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  auto copy = [&](int tile, int buf) {
    mbar_arrive_expect_tx(&bar[buf], kBytes);
    float* dst = s_m + (size_t)buf * (kBytes / 4);
    bulk_copy_g2s(dst, a.cellM + (size_t)tile * kFFCells * AMPS_CELLM, kFFBytes, &bar[buf]);
    if (ACC == 2) bulk_copy_g2s(dst + kFFBytes / 4, a.cellJ + (size_t)tile * kFFCells * 24, kFFJBytes, &bar[buf]);
  };
  // thread t < 54 owns tile corner t
  const int ti = tid % 9, tj = (tid / 9) % 3, tk = tid / 27;
  auto corner_id = [&](int tile) {
    if (tile >= tiles || tid >= kFFCorners) return 0;
    const int b = tile >> 5, l = (tile & 31) * kFFCells;  // 32 tiles per block
    return __ldg(a.ctabh + b * 729 + ti + 9 * (((l >> 3) & 7) + tj + 9 * ((l >> 6) + tk)));
  };
  auto corner_values = [&](int id, FF (&x)[3]) {
    if (id >= 0) {
#pragma unroll
      for (int d = 0; d < 3; d++) x[d] = FF{a.xh[d * a.nvc + id], a.xl[d * a.nvc + id]};
    } else {
      const int h = ~id, s = a.h.hs[h], e = a.h.hs[h + 1];
      FF v[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
      for (int t = s; t < e; t++) {
        const float wh = a.h.hwh[t], wl = a.h.hwl[t];
        const int q = a.h.hp[t];
#pragma unroll
        for (int d = 0; d < 3; d++) ff_add2(v[d], wh, wl, a.xh[d * a.nvc + q], a.xl[d * a.nvc + q]);
      }
#pragma unroll
      for (int d = 0; d < 3; d++) x[d] = ff_norm(v[d]);
    }
  };
  auto centre = [&](int tile) { return a.Bcen[p * a.ncell + (long long)tile * kFFCells + lc]; };
  const float sg = ACC == 2 ? -1.f : 1.f;
  int tile = blockIdx.x, t1 = tile + gridDim.x, t2 = s_next;  // grid <= tiles
  if (tid == 0) copy(tile, 0);
  int id = corner_id(tile), id1 = corner_id(t1);
  FF x[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  if (tid < kFFCorners) corner_values(id, x);
  double bc = ACC == 2 && set == 0 ? centre(tile) : 0.0;
  int n = 0;  // tiles done
  while (tile < tiles) {
    const int buf = n & 1;
    const bool more = t1 < tiles;
    if (tid == 0 && more) copy(t1, buf ^ 1);
    const int t3 = tid == 0 && more ? claim() : tiles;
    if (tid < kFFCorners) {
#pragma unroll
      for (int d = 0; d < 3; d++) s_x[d][tid] = make_float4(x[d].s, x[d].s, x[d].q, x[d].q);
    }
    if (ACC == 2 && set == 0) {
      const float bh = (float)bc;
      s_b[p][lc] = make_float2(bh, (float)(bc - (double)bh));
      if (more) bc = centre(t1);
    }
    // in flight over this tile's arithmetic
    const int id2 = corner_id(t2);
    if (tid < kFFCorners && more) corner_values(id1, x);
    const int idc = id;  // this tile's
    id = id1;
    id1 = id2;
    // CTA-uniform: every thread leaves together on a timeout
    const bool ok = __syncthreads_and(mbar_wait_bounded(&bar[buf], (n >> 1) & 1, kWaitLimit)) != 0;
    if (!ok) {
      if (tid == 0) atomicAdd(a.flags + 2, 1ull);
      // let the copies land before exiting
      mbar_wait_bounded(&bar[buf], (n >> 1) & 1, kWaitLimit);
      if (more) mbar_wait_bounded(&bar[buf ^ 1], ((n + 1) >> 1) & 1, kWaitLimit);
      return;
    }
    const LevelK& K = a.lk[min(__ffs(__ldg(a.bscale + (tile >> 5))) - 1, kMaxScale - 1)];
    const int i = lc & 7, j = lc >> 3;
    auto tc = [&](int xx, int yy, int zz) { return i + xx + 9 * (j + yy + 3 * zz); };
    // the curl's component p: cu_p = 0.25/dx (sum +-E_qa - sum +-E_qb), a sum per set:
    // cu0 = (dEz/dy - dEy/dz), cu1 = (dEx/dz - dEz/dx), cu2 = (dEy/dx - dEx/dy)
    {
      const int q = (p + 2 - set) % 3;   // qa = p + 2, qb = p + 1
      const int ax = (p + 1 + set) % 3;  // the axis of the difference
      FF d{0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 8; c++) {
        const float4 v = s_x[q][tc(c & 1, (c >> 1) & 1, c >> 2)];
        const bool plus = (((c >> ax) & 1) != 0) == (set == 0);
        ff_acc(d, plus ? v.x : -v.x, plus ? v.z : -v.z);
      }
      const float ds = __shfl_xor_sync(0xffffffffu, d.s, kFFCells), dq = __shfl_xor_sync(0xffffffffu, d.q, kFFCells);
      ff_acc(d, ds, dq);
      d = ff_norm(d);
      const FF cu = ff_norm(ff_mul(d.s, d.q, K.curl[0], K.curl[1]));
      if (set == 0) s_cu[p][lc] = make_float2(cu.s, cu.q);
    }
    // mass term: sum over pairs of m (FP32 partial) x e, in FP32 pairs; acc[x] holds
    // the corners x, y = set of the cell's lower (z = 0) and upper face.  Row p of the
    // monomial blocks, from y-sum `set` on.
    const float* tm = s_m + (size_t)buf * (kBytes / 4);
    const float* mm = tm + lc * AMPS_CELLM + 27 * set + 3 * p;
    FF2 acc[2] = {{0ull, 0ull}, {0ull, 0ull}};
#pragma unroll 1
    for (int q = 0; q < 3; q++) {
#pragma unroll
      for (int y2 = 0; y2 < 2; y2++) {
        ulonglong2 e[2][2];  // [x][z], (h, h) and (l, l)
#pragma unroll
        for (int x2 = 0; x2 < 2; x2++)
#pragma unroll
          for (int z2 = 0; z2 < 2; z2++) e[x2][z2] = *reinterpret_cast<const ulonglong2*>(&s_x[q][tc(x2, y2, z2)]);
#pragma unroll
        for (int ax = 0; ax < 3; ax++) {
          const float* m = mm + 9 * (ax + 3 * y2) + q;
          const float m0 = m[0], m1 = m[81], m2 = m[162];
          const unsigned long long mA = pk(m0, m1), mB = pk(m1, m2), nA = pk(-m0, -m1), nB = pk(-m1, -m2);
#pragma unroll
          for (int x1 = 0; x1 < 2; x1++) {
            const int x2 = ax - x1;
            if (x2 < 0 || x2 > 1) continue;
            ff2_add(acc[x1], mA, nA, e[x2][0].x, e[x2][0].y);
            ff2_add(acc[x1], mB, nB, e[x2][1].x, e[x2][1].y);
          }
        }
      }
    }
    FF out[2][2];  // [z][x]
#pragma unroll
    for (int z = 0; z < 2; z++)
#pragma unroll
      for (int xx = 0; xx < 2; xx++) {
        const float2 as = upk(acc[xx].s), aq = upk(acc[xx].q);
        const FF t = ff_norm(FF{z ? as.y : as.x, z ? aq.y : aq.x});
        out[z][xx] = ff_mul(t.s, t.q, sg * K.m[0], sg * K.m[1]);
        if (ACC == 1) {
          const float4 v = s_x[p][tc(xx, set, z)];
          ff_add2(out[z][xx], K.id[0], K.id[1], v.x, v.z);
        } else {
          // corner (x, y) in the table order (0,0) (1,0) (1,1) (0,1)
          const int c = 4 * z + (set ? 3 - xx : xx);
          ff_add2(out[z][xx], -a.fj[0], -a.fj[1], tm[kFFBytes / 4 + lc * 24 + 3 * c + p], 0.f);
        }
      }
    __syncthreads();  // s_cu complete; s_x is not read again
    // out += s (sig1 y[q1] - sig2 y[q2]) for y = the curl (s = sg th2dt2 V 0.25/dx)
    // and, for the RHS, y = centre B (s = thdt V 0.25/dx): C^T y, component p
    const int q1 = (p + 1) % 3, q2 = (p + 2) % 3;
    auto curl_t = [&](const float2 (*y)[kFFCells], float sh, float sl) {
      const float2 y1 = y[q1][lc], y2 = y[q2][lc];
      FF tpp{y1.x, y1.y}, tpm{y1.x, y1.y};
      ff_acc(tpp, -y2.x, -y2.y);  // y1 - y2
      ff_acc(tpm, y2.x, y2.y);    // y1 + y2
      tpp = ff_norm(tpp);
      tpm = ff_norm(tpm);
      const FF upp = ff_mul(tpp.s, tpp.q, sh, sl), upm = ff_mul(tpm.s, tpm.q, sh, sl);
#pragma unroll
      for (int z = 0; z < 2; z++)
#pragma unroll
        for (int xx = 0; xx < 2; xx++) {
          const bool s1 = p == 0 ? z : (p == 1 ? xx : set);
          const bool s2 = p == 0 ? set : (p == 1 ? z : xx);
          // s1 y1 - s2 y2: (+,+) y1 - y2, (+,-) y1 + y2, (-,+) -(y1 + y2), (-,-) -(y1 - y2)
          const float us = s1 == s2 ? upp.s : upm.s, uq = s1 == s2 ? upp.q : upm.q;
          ff_acc(out[z][xx], s1 ? us : -us, s1 ? uq : -uq);
        }
    };
    curl_t(s_cu, sg * K.cc[0], sg * K.cc[1]);
    if (ACC == 2) curl_t(s_b, K.bb[0], K.bb[1]);
    // row j + set: the cell's corner and its left neighbour's; row 1 is of both sets
    auto row = [&](float2 (*dst)[kFFCorners], int xx, int z, FF v) {
      const float rs = __shfl_down_sync(0xffffffffu, v.s, 8), rq = __shfl_down_sync(0xffffffffu, v.q, 8);
      const bool both = set == 0 && j == 1;  // lanes 8 .. 15; lanes 16 .. 23 hold the rest
      ff_acc(v, both ? rs : 0.f, both ? rq : 0.f);
      const FF o = ff_norm(v);
      if ((xx == 0 || i == 7) && (set == 0 || j == 1)) dst[p][tc(xx, set, z)] = make_float2(o.s, o.q);
    };
    auto corners = [&](float2 (*dst)[kFFCorners], FF (&v)[2][2]) {
#pragma unroll
      for (int z = 0; z < 2; z++) {
        const float rs = __shfl_up_sync(0xffffffffu, v[z][1].s, 1), rq = __shfl_up_sync(0xffffffffu, v[z][1].q, 1);
        ff_acc(v[z][0], i > 0 ? rs : 0.f, i > 0 ? rq : 0.f);
        row(dst, 0, z, v[z][0]);
        row(dst, 1, z, v[z][1]);
      }
    };
    corners(s_out, out);
    if (ACC == 2 && a.diag) {
      // the cell's diagonal (a preconditioner: FP32 per cell is enough): monomial of a
      // corner with itself, entry (p, p)
      FF dg[2][2];
#pragma unroll
      for (int z = 0; z < 2; z++)
#pragma unroll
        for (int xx = 0; xx < 2; xx++)
          dg[z][xx] = FF{fmaf(K.m[0], tm[lc * AMPS_CELLM + 9 * (2 * xx + 6 * set + 18 * z) + 4 * p], K.dg), 0.f};
      corners(s_dg, dg);
    }
    if (tid == 0) s_next = t3;
    __syncthreads();  // s_out, s_next complete; this buffer is not read again
    // scatter with P^T: one FP64 reduction per tile corner and component
    if (tid < kFFCorners) {
      if (ACC == 2 && a.diag && idc >= 0) {
#pragma unroll
        for (int d = 0; d < 3; d++)
          atomicAdd(a.diag + d * a.nvc + idc, (double)s_dg[d][tid].x + (double)s_dg[d][tid].y);
      }
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const FF o{s_out[d][tid].x, s_out[d][tid].y};
        if (idc >= 0) {
          atomicAdd(y64 + d * a.nvc + idc, ff_value(o));
        } else {
          for (int t = a.h.hs[~idc]; t < a.h.hs[~idc + 1]; t++)
            atomicAdd(y64 + d * a.nvc + a.h.hp[t], ff_value(ff_mul(o.s, o.q, a.h.hwh[t], a.h.hwl[t])));
        }
      }
    }
    tile = t1;
    t1 = t2;
    t2 = s_next;
    n++;
  }
}

// x (times dinv) as FP32 pairs: the input of the pair-arithmetic operator
__global__ void __launch_bounds__(256) k_amr_split(long long n, const double* __restrict__ x,
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

// w = A (D v) from y32 as FP32 pairs (Krylov vectors): free rows S (D v) + y32
// in pairs, hanging rows (D v)_h - (P D v)_h; y32 cleared for the next
// application.  Almost every row of S is its diagonal alone (diag, a pair; 0: any
// other row): a thread takes two corners, whose loads depend on nothing (a CTA's
// life is one memory latency: more loads per thread, fewer CTAs).
// The other rows are listed; the CTAs past the first `plain` take them, 8 lanes
// per row over its entries: one thread walking a row of up to 27 entries, two
// dependent loads each, set the time of the whole kernel
// (500,832 corners: 14 us, before 21; clearing y32 before the operator took 4 more).
constexpr int kRowLanes = 8;
constexpr int kFinPer = 2;
__global__ void __launch_bounds__(256) k_amr_finish_ff(long long nvc, Hang h, unsigned plain,
                                                       int nrows, const int* __restrict__ rows,
                                                       const int* __restrict__ ss,
                                                       const int* __restrict__ sc,
                                                       const float* __restrict__ svh,
                                                       const float* __restrict__ svl,
                                                       const float2* __restrict__ diag,
                                                       float* __restrict__ y32, OpIn in,
                                                       float* __restrict__ wh, float* __restrict__ wl) {
  if (blockIdx.x < plain) {
    // kFinPer corners per thread, all their loads in flight together
    const long long c0 = (long long)blockIdx.x * (256 * kFinPer) + threadIdx.x;
    float2 dg[kFinPer];
    float y[kFinPer][3];
    FF v[kFinPer][3];
#pragma unroll
    for (int k = 0; k < kFinPer; k++) {
      const long long c = min(c0 + 256 * k, nvc - 1);
      dg[k] = diag[c];
#pragma unroll
      for (int d = 0; d < 3; d++) v[k][d] = opin_value(in, d * nvc + c);
    }
    pdl_wait();  // the tiles' sums
#pragma unroll
    for (int k = 0; k < kFinPer; k++)
#pragma unroll
      for (int d = 0; d < 3; d++) y[k][d] = y32[d * nvc + min(c0 + 256 * k, nvc - 1)];
#pragma unroll
    for (int k = 0; k < kFinPer; k++) {
      const long long c = c0 + 256 * k;
      if (c >= nvc || dg[k].x == 0.f) continue;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        FF acc{y[k][d], 0.f};
        ff_add2(acc, dg[k].x, dg[k].y, v[k][d].s, v[k][d].q);
        acc = ff_norm(acc);
        wh[d * nvc + c] = acc.s;
        wl[d * nvc + c] = acc.q;
        y32[d * nvc + c] = 0.f;
      }
    }
    return;
  }
  const int r = (int)(blockIdx.x - plain) * (int)(blockDim.x / kRowLanes) + (int)(threadIdx.x / kRowLanes);
  const int lane = threadIdx.x % kRowLanes;
  const bool act = r < nrows;
  const int c = act ? rows[r] : 0;
  int s = 0, e = 0;
  const int* col = h.hp;
  const float* cwh = h.hwh;
  const float* cwl = h.hwl;
  float sign = -1.f;
  bool con = true;
  if (act) {
    s = h.hs[c];
    e = h.hs[c + 1];
    if (s == e && is_bnd(h, c)) {  // boundary rows (donors)
      s = h.bs[c];
      e = h.bs[c + 1];
      col = h.bc;
      cwh = h.bwh;
      cwl = h.bwl;
    } else if (s == e) {  // free rows with other entries of S
      con = false;
      s = ss[c];
      e = ss[c + 1];
      col = sc;
      cwh = svh;
      cwl = svl;
      sign = 1.f;
    }
  }
  FF acc[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  for (int t = s + lane; t < e; t += kRowLanes) {
    const int q = col[t];
    const float mh = sign * cwh[t], ml = sign * cwl[t];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const FF u = opin_value(in, d * nvc + q);
      ff_add2(acc[d], mh, ml, u.s, u.q);
    }
  }
#pragma unroll
  for (int k = kRowLanes / 2; k > 0; k >>= 1)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float bs = __shfl_xor_sync(0xffffffffu, acc[d].s, k), bq = __shfl_xor_sync(0xffffffffu, acc[d].q, k);
      ff_acc(acc[d], bs, bq);
    }
  pdl_wait();
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (!act || lane != d) continue;
    const long long o = d * nvc + c;
    const FF v = opin_value(in, o);
    FF w = acc[d];
    ff_acc(w, con ? v.s : y32[o], con ? v.q : 0.f);
    w = ff_norm(w);
    wh[o] = w.s;
    wl[o] = w.q;
    y32[o] = 0.f;
  }
}

// constraint rows (hanging, boundary; rows lists them among others):
// y_h = x_h - (P x)_h (operator) or 0 (rhs)
__global__ void __launch_bounds__(256) k_amr_constraint(int nrows, const int* __restrict__ rows, long long nvc,
                                                        Hang h, const double* __restrict__ x,
                                                        const double* __restrict__ dinv,
                                                        double* __restrict__ y, int rhs_mode,
                                                        int* __restrict__ next) {
  pdl_wait();
  pdl_next();
  if (blockIdx.x == 0 && threadIdx.x == 0) *next = 0;  // for the next tile kernel
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (t0 >= nrows) return;
  const int c = rows[t0];
  int s = h.hs[c], e = h.hs[c + 1];
  const int* col = h.hp;
  const double* w = h.hw;
  if (s == e) {
    // boundary rows (open axes): the same form with the donor list
    if (!is_bnd(h, c)) return;
    s = h.bs[c];
    e = h.bs[c + 1];
    col = h.bc;
    w = h.bw;
  }
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (rhs_mode) {
      y[d * nvc + c] = 0.0;
    } else {
      double pv = 0.0;
      for (int t = s; t < e; t++) {
        const int p = col[t];
        pv += w[t] * (dinv ? dinv[d * nvc + p] : 1.0) * x[d * nvc + p];
      }
      y[d * nvc + c] = (dinv ? dinv[d * nvc + c] : 1.0) * x[d * nvc + c] - pv;
    }
  }
}

// 1 / the Jacobi diagonal that the RHS kernel summed
__global__ void __launch_bounds__(256) k_amr_invert_diag(long long nvc, Hang h, const double* __restrict__ diag,
                                                         double* __restrict__ dinv, float* __restrict__ dff) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nvc) return;
  const bool hang = h.hs[c + 1] > h.hs[c] || is_bnd(h, c);  // constraint rows: scaling 1
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const float v = (float)diag[d * nvc + c];  // a preconditioner: FP32 reciprocal
    const float r = (hang || v == 0.f) ? 1.f : 1.0f / v;
    dinv[d * nvc + c] = (double)r;
    dff[d * nvc + c] = r;  // as pairs: FP32 values
    dff[3 * nvc + d * nvc + c] = 0.f;
  }
}

// B^{n+1} = B^n - dt curl E^{n+theta}, one CTA per block: each corner value is
// gathered once into shared memory (hanging ones interpolated there), and the face
// sums of the curl share their partial sums along the third axis: 24 FP64 additions
// per cell instead of 42.  FP64 (a 64th of the FP32 rate) and the gathers' latency
// bound it.  491,520 cells: 49 us (one thread per cell gathering its 8 corners: 85).
__global__ void __launch_bounds__(256) k_amr_update_b(long long ncell, long long nvc,
                                                      const int* __restrict__ ctabh, Hang h,
                                                      const double* __restrict__ bdx,
                                                      const double* __restrict__ Eh,
                                                      const double* __restrict__ Bn,
                                                      double* __restrict__ Bnew, double dt,
                                                      double* __restrict__ energy) {
  pdl_wait();
  pdl_next();
  __shared__ double s_e[3][729];
  const int b = blockIdx.x;
  if (b == 0 && threadIdx.x == 0) *energy = 0.0;  // for k_amr_update_e
  for (int q = threadIdx.x; q < 729; q += 256) {
    const int id = ctabh[b * 729 + q];
#pragma unroll
    for (int d = 0; d < 3; d++) s_e[d][q] = id >= 0 ? Eh[d * nvc + id] : cval(Eh, nullptr, nvc, ~id, d, h);
  }
  const long long cell0 = (long long)b * AMPS_CPB + threadIdx.x;
  double B[2][3];
#pragma unroll
  for (int k = 0; k < 2; k++)
#pragma unroll
    for (int d = 0; d < 3; d++) B[k][d] = Bn[d * ncell + cell0 + 256 * k];
  const double f = dt * 0.25 / bdx[b];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int l = threadIdx.x + 256 * k;
    const int c0 = (l & 7) + 9 * (((l >> 3) & 7) + 9 * (l >> 6));
    // diff[d][e]: 4 dx times the mean difference of component d along axis e
    auto diffs = [&](int d, int sa, int sb, int sc, double& da, double& db) {
      // sums along the stride sc, then differences along sa and sb
      const double* e = s_e[d] + c0;
      const double s00 = e[0] + e[sc], s10 = e[sa] + e[sa + sc];
      const double s01 = e[sb] + e[sb + sc], s11 = e[sa + sb] + e[sa + sb + sc];
      const double t1 = s11 - s00, t2 = s10 - s01;
      da = t1 + t2;
      db = t1 - t2;
    };
    double xy, xz, yx, yz, zx, zy;  // xy: of E_x along y
    diffs(0, 9, 81, 1, xy, xz);
    diffs(1, 1, 81, 9, yx, yz);
    diffs(2, 1, 9, 81, zx, zy);
    Bnew[cell0 + 256 * k] = B[k][0] - f * (zy - yz);
    Bnew[ncell + cell0 + 256 * k] = B[k][1] - f * (xz - zx);
    Bnew[2 * ncell + cell0 + 256 * k] = B[k][2] - f * (yx - xy);
  }
}

// UpdateB's boundary branch on meshes with open axes
// (pic_field_solver_ecsim.cpp:5274-5600): a cell with a face on an open domain
// face keeps B^n (Dirichlet, pass 0) or takes the mean of B^{n+1} of its
// face-normal inward neighbours, one per such face, in the same block
// (Neumann, pass p = number of such faces: faces, then edges, then corners, so
// every donor is final when read).  A cell on a Neumann face (bit 2d + high of
// neumann) is Neumann, whatever its other faces.
__global__ void __launch_bounds__(256) k_amr_bnd_b(long long ncell, const int* __restrict__ borg,
                                                   const int* __restrict__ bscale, int nf0, int nf1, int nf2,
                                                   int open, int neumann, int pass, const double* __restrict__ Bn,
                                                   double* __restrict__ Bnew) {
  const long long cell = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (cell >= ncell) return;
  const int b = (int)(cell >> 9), l = (int)(cell & 511);
  const int idx[3] = {l & 7, (l >> 3) & 7, l >> 6};
  const int st = bscale[b], nf[3] = {nf0, nf1, nf2};
  int side[3] = {0, 0, 0}, nface = 0;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (!((open >> d) & 1)) continue;
    const int lo = borg[3 * b + d] + idx[d] * st;
    if (lo == 0) side[d] = -1;
    else if (lo + st == nf[d]) side[d] = 1;
    nface += side[d] != 0;
  }
  if (!nface) return;
  bool neu = false;
#pragma unroll
  for (int d = 0; d < 3; d++)
    if (side[d]) neu |= (neumann >> (2 * d + (side[d] > 0))) & 1;
  if (!neu) {
    if (pass == 0)
#pragma unroll
      for (int q = 0; q < 3; q++) Bnew[q * ncell + cell] = Bn[q * ncell + cell];
    return;
  }
  if (nface != pass) return;
  double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (!side[d]) continue;
    int j[3] = {idx[0], idx[1], idx[2]};
    j[d] -= side[d];
    const long long dn = (long long)b * 512 + j[0] + 8 * (j[1] + 8 * j[2]);
#pragma unroll
    for (int q = 0; q < 3; q++) acc[q] += Bnew[q * ncell + dn];
  }
#pragma unroll
  for (int q = 0; q < 3; q++) Bnew[q * ncell + cell] = acc[q] / nface;
}

// C2N, corner B = sum of V B over the corner's cells / sum of V (cinv, the mesh's
// own), one CTA per block: the block's cells are summed onto its 729 corners axis by
// axis in shared memory (11 FP64 additions per cell), corners inside the block are
// written, those on its faces added to the other blocks' shares.  Hanging corners
// are interpolated afterwards.  491,520 cells: 33 us with the hanging corners (8
// reductions per cell and component, and the volumes summed again each time: 70).
__global__ void __launch_bounds__(256) k_amr_c2n(long long ncell, long long nvc,
                                                 const int* __restrict__ ctab,
                                                 const double* __restrict__ bdx,
                                                 const double* __restrict__ cinv,
                                                 const double* __restrict__ Bcen, double* __restrict__ acc) {
  pdl_wait();
  pdl_next();
  __shared__ double s_c[512], s_x[576], s_y[648];
  const int b = blockIdx.x, tid = threadIdx.x;
  const double dx = bdx[b], V = dx * dx * dx;
  int cc[3];
  double w[3];
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const int q = tid + 256 * r;
    cc[r] = q < 729 ? ctab[b * 729 + q] : 0;
    w[r] = V * cinv[cc[r]];
  }
  for (int d = 0; d < 3; d++) {
#pragma unroll
    for (int k = 0; k < 2; k++) s_c[tid + 256 * k] = Bcen[d * ncell + (long long)b * AMPS_CPB + tid + 256 * k];
    __syncthreads();
    for (int q = tid; q < 576; q += 256) {
      const int i = q % 9, r = q / 9;  // corner i of row r
      s_x[q] = (i > 0 ? s_c[8 * r + i - 1] : 0.0) + (i < 8 ? s_c[8 * r + i] : 0.0);
    }
    __syncthreads();
    for (int q = tid; q < 648; q += 256) {
      const int i = q % 9, j = q / 9 % 9, k = q / 81;
      s_y[q] = (j > 0 ? s_x[i + 9 * (j - 1 + 8 * k)] : 0.0) + (j < 8 ? s_x[i + 9 * (j + 8 * k)] : 0.0);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const int q = tid + 256 * r;
      if (q >= 729) break;
      const int i = q % 9, j = q / 9 % 9, k = q / 81;
      const double v = w[r] * ((k > 0 ? s_y[q - 81] : 0.0) + (k < 8 ? s_y[q] : 0.0));
      double* o = acc + d * nvc + cc[r];
      if (i > 0 && i < 8 && j > 0 && j < 8 && k > 0 && k < 8) *o = v;
      else atomicAdd(o, v);
    }
  }
}

// sum of en over the grid into *energy (256 threads per CTA)
__device__ __forceinline__ void add_energy(double en, double* energy) {
  __shared__ double s[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) en += __shfl_xor_sync(0xffffffffu, en, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = en;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += s[w];
    atomicAdd(energy, t);
  }
}

// hanging corners of a field take the interpolation of their (free) parents; rows
// lists them among others.  cvol (optional): their share of the wave energy.
__global__ void __launch_bounds__(256) k_amr_fix_hanging(int nrows, const int* __restrict__ rows, long long nvc,
                                                         Hang h, double* F, const double* __restrict__ cvol,
                                                         double* energy) {
  pdl_wait();
  pdl_next();
  const int t0 = blockIdx.x * blockDim.x + threadIdx.x;
  double en = 0.0;
  if (t0 < nrows) {
    const int c = rows[t0], s = h.hs[c], e = h.hs[c + 1];
    if (s < e) {
      double v[3] = {0.0, 0.0, 0.0};
      for (int t = s; t < e; t++) {
        const double w = h.hw[t];
        const int p = h.hp[t];
#pragma unroll
        for (int d = 0; d < 3; d++) v[d] += w * F[d * nvc + p];
      }
#pragma unroll
      for (int d = 0; d < 3; d++) F[d * nvc + c] = v[d];
      if (cvol) en = -cvol[c] * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) * 0.015625 / kPi;
    }
  }
  if (cvol) add_energy(en, energy);
}

// E^{n+1} = ri E^{n+theta} - r1 E^n, and the wave energy sum_cells V (sum_corners
// |E|^2/8 + |B|^2) / (8 pi) per corner with the volume of its cells (cvol; hanging
// corners carry it negative: their E and its energy follow in k_amr_fix_hanging).
// The FP64 pipe bounds it.  491,520 cells: 42 us with k_amr_fix_hanging (a pass over
// the cells' 8 corners each, and all corners looked at for hanging ones: 85).
__global__ void __launch_bounds__(256) k_amr_update_e(long long ncell, long long nvc,
                                                      const double* __restrict__ Eh, double* __restrict__ En,
                                                      double ri, double r1, const double* __restrict__ cvol,
                                                      const double* __restrict__ bdx,
                                                      const double* __restrict__ Bcen, double* energy) {
  pdl_wait();
  pdl_next();
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  double ee = 0.0, eb = 0.0;
  for (long long c = t0; c < nvc; c += step) {
    double e2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double v = ri * Eh[d * nvc + c] - r1 * En[d * nvc + c];
      En[d * nvc + c] = v;
      e2 += v * v;
    }
    const double w = cvol[c];
    ee += w > 0.0 ? w * e2 : 0.0;
  }
  for (long long cell = t0; cell < ncell; cell += step) {
    const double dx = bdx[cell >> 9];
    double b2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double v = Bcen[d * ncell + cell];
      b2 += v * v;
    }
    eb += dx * dx * dx * b2;
  }
  add_energy((0.125 * ee + eb) * 0.125 / kPi, energy);
}

// three CTAs per block, a corner per thread (ctabh: hanging corners as ~id); 960 blocks:
// 33 us (one CTA per block and two looks at the constraint rows per value: 41)
__global__ void __launch_bounds__(256) k_amr_pack(long long nvc, const int* __restrict__ ctabh, Hang h,
                                                  const double* __restrict__ Eh, const double* __restrict__ Bprev,
                                                  const double* __restrict__ Bcur, float* __restrict__ sp,
                                                  float* __restrict__ sd) {
  pdl_wait();
  pdl_next();
  const int b = blockIdx.x, s = blockIdx.y * 256 + threadIdx.x;
  if (s >= AMPS_SC) return;
  const int id = ctabh[b * 729 + s];
  auto val = [&](const double* F, int d) {
    return (float)(id >= 0 ? F[d * nvc + id] : cval(F, nullptr, nvc, ~id, d, h));
  };
  float4* op = reinterpret_cast<float4*>(sp + ((size_t)b * AMPS_SC + s) * AMPS_PUSH_STRIDE);
  op[0] = make_float4(val(Eh, 0), val(Eh, 1), val(Eh, 2), val(Bprev, 0));
  op[1] = make_float4(val(Bprev, 1), val(Bprev, 2), 0.f, 0.f);
  reinterpret_cast<float4*>(sd)[(size_t)b * AMPS_SC + s] =
      make_float4(val(Bcur, 0), val(Bcur, 1), val(Bcur, 2), 0.f);
}

Hang hang_of(const amps_gpu_ctx* c) {
  return Hang{c->d_hs, c->d_hp, c->d_hw, c->d_hwh, c->d_hwl,
              c->d_bflag, c->d_bs, c->d_bc, c->d_bw, c->d_bwh, c->d_bwl};
}
unsigned g1(long long n) { return (unsigned)((n + 255) / 256); }

}  // namespace

// ============================================================================
cudaError_t launch_amr_pack(amps_gpu_ctx* c, const double* Eh, const double* Bprev,
                            const double* Bcur) {
  TimedLaunch t(c, "pack_stencils");
  launch_pdl(k_amr_pack, dim3(c->nb, 3), dim3(256), 0, c->stream, c->nvc, c->d_ctabh, hang_of(c), Eh, Bprev,
             Bcur, c->d_stencil_push, c->d_stencil_dep);
  return cudaGetLastError();
}

static ApplyArgs apply_args(amps_gpu_ctx* c) {
  ApplyArgs a{};
  a.ncell = c->ncor;
  a.nvc = c->nvc;
  a.ctabh = c->d_ctabh;
  a.h = hang_of(c);
  a.cellM = c->d_cellM;
  a.cellJ = c->d_cellJ;
  const double th = c->cfg.theta, dt = c->cfg.dt;
  const double th2dt2 = th * th * dt * dt, f = 4.0 * kPi * dt * th, thdt = th * dt;
  a.flags = c->d_flags;
  a.next = c->d_next;
  a.bscale = c->d_bscale;
  auto split = [](double v, float* o) {
    o[0] = (float)v;
    o[1] = (float)(v - (double)o[0]);
  };
  for (int sc = 0; sc < kMaxScale; sc++) {
    const double dx = c->dxf * (double)(1 << sc), V = dx * dx * dx;
    LevelK& K = a.lk[sc];
    split(0.25 / dx, K.curl);
    split(th2dt2 * V * 0.25 / dx, K.cc);
    split(0.125 * V, K.id);
    split(f * V, K.m);
    split(thdt * V * 0.25 / dx, K.bb);
    K.dg = (float)(V * (0.125 + th2dt2 / (8.0 * dx * dx)));
  }
  split(f, a.fj);
  return a;
}

// x (times dinv) as FP32 pairs in the context's scratch (2 x 3 nvc floats)
static cudaError_t split_input(amps_gpu_ctx* c, const double* x, const double* dinv, ApplyArgs& a) {
  const long long n = 3 * c->nvc;
  cudaError_t e = cudaSuccess;
  if (!c->d_xs && (e = cudaMalloc(reinterpret_cast<void**>(&c->d_xs), sizeof(float) * 2 * n)) != cudaSuccess)
    return e;
  a.xh = c->d_xs;
  a.xl = c->d_xs + n;
  launch_pdl(k_amr_split, dim3((unsigned)(std::min<long long>((n + 255) / 256, 152LL * 16))), dim3(256), 0,
             c->stream, n, x, dinv, c->d_xs, c->d_xs + n);
  return cudaGetLastError();
}

// CTAs of a persistent tile kernel that the device holds at a time (asked once per
// device and kernel)
template <typename Kernel>
static cudaError_t tile_grid(Kernel kernel, int threads, uint32_t smem, int (&grid)[64], int& n) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (grid[dev] == 0) {
    int sms = 0, per = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    grid[dev] = sms * std::max(per, 1);
  }
  n = grid[dev];
  return cudaSuccess;
}

// y64 += the operator (ACC 1) or the RHS (ACC 2) in FP32 pairs
template <int ACC>
static cudaError_t launch_tile(amps_gpu_ctx* c, const ApplyArgs& a, double* y64) {
  static int grid[64] = {0};
  int n = 0;
  cudaError_t e = tile_grid(k_amr_tile_ff<ACC>, kTileThreads, 2 * tile_ff_bytes<ACC>(), grid, n);
  if (e != cudaSuccess) return e;
  // AMR meshes hold whole 512-cell blocks: ncell is a multiple of the tile
  const int tiles = (int)(c->ncor / kFFCells);
  launch_pdl(k_amr_tile_ff<ACC>, dim3(std::min(n, tiles)), dim3(kTileThreads), 2 * tile_ff_bytes<ACC>(),
             c->stream, a, tiles, y64);
  return cudaGetLastError();
}

// y32 += the FP32 operator on a.xf
static cudaError_t launch_tile32(amps_gpu_ctx* c, const ApplyArgs& a, float* y32) {
  static int grid[64] = {0};
  int n = 0;
  cudaError_t e = tile_grid(k_amr_tile32, kT32Threads, 2 * kTileBytes, grid, n);
  if (e != cudaSuccess) return e;
  const int tiles = (int)(c->ncor / kTileCells);
  launch_pdl(k_amr_tile32, dim3(std::min(n, tiles)), dim3(kT32Threads), 2 * kTileBytes, c->stream, a, tiles,
             y32);
  return cudaGetLastError();
}

cudaError_t launch_amr_matvec(amps_gpu_ctx* c, const double* x, const double* dinv, double* y, bool pairs) {
  cudaError_t e = cudaMemsetAsync(y, 0, sizeof(double) * 3 * c->nvc, c->stream);
  if (e != cudaSuccess) return e;
  ApplyArgs a = apply_args(c);
  TimedLaunch t(c, "matvec", pairs ? 2 : 3);
  if (pairs) {
    a.xh = c->d_xs;
    a.xl = c->d_xs + 3 * c->nvc;
  } else if ((e = split_input(c, x, dinv, a)) != cudaSuccess) {
    return e;
  }
  if ((e = launch_tile<1>(c, a, y)) != cudaSuccess) return e;
  launch_pdl(k_amr_constraint, dim3(g1(std::max(c->nsrows, 1))), dim3(256), 0, c->stream, c->nsrows,
             c->d_srows, c->nvc, a.h, x, dinv, y, 0, c->d_next);
  return cudaGetLastError();
}

// (d_y32 is zero between applications: the finish kernel clears what it reads)
cudaError_t launch_amr_matvec32_ff(amps_gpu_ctx* c, const OpIn& in, float* wh, float* wl) {
  cudaError_t e = cudaSuccess;
  ApplyArgs a = apply_args(c);
  const long long n = 3 * c->nvc;
  if (!c->d_xs && (e = cudaMalloc(reinterpret_cast<void**>(&c->d_xs), sizeof(float) * 2 * n)) != cudaSuccess)
    return e;
  a.xf = c->d_xs;
  TimedLaunch t(c, "matvec32", in.xf_ready ? 2 : 3);
  if (!in.xf_ready && (e = launch_in_f32(c, in, c->d_xs)) != cudaSuccess) return e;
  if ((e = launch_tile32(c, a, c->d_y32)) != cudaSuccess) return e;
  const unsigned plain = (unsigned)((c->nvc + 256 * kFinPer - 1) / (256 * kFinPer));
  const int per = 256 / kRowLanes;
  launch_pdl(k_amr_finish_ff, dim3(plain + (unsigned)((c->nsrows + per - 1) / per)), dim3(256), 0,
             c->stream, c->nvc, a.h, plain, c->nsrows, c->d_srows, c->d_ss, c->d_sc, c->d_svh, c->d_svl,
             c->d_sdiag, c->d_y32, in, wh, wl);
  return cudaGetLastError();
}

// diag: also sum the Jacobi diagonal, for launch_amr_jacobi
cudaError_t launch_amr_rhs(amps_gpu_ctx* c, bool diag) {
  cudaError_t e = cudaMemsetAsync(c->d_rhs, 0, sizeof(double) * 3 * c->nvc, c->stream);
  if (e == cudaSuccess && diag) e = cudaMemsetAsync(c->d_diag, 0, sizeof(double) * 3 * c->nvc, c->stream);
  if (e != cudaSuccess) return e;
  ApplyArgs a = apply_args(c);
  a.diag = diag ? c->d_diag : nullptr;
  a.Bcen = c->d_Bc;
  TimedLaunch t(c, "rhs", 3);
  if ((e = split_input(c, c->d_En, nullptr, a)) != cudaSuccess) return e;
  if ((e = launch_tile<2>(c, a, c->d_rhs)) != cudaSuccess) return e;
  launch_pdl(k_amr_constraint, dim3(g1(std::max(c->nsrows, 1))), dim3(256), 0, c->stream, c->nsrows,
             c->d_srows, c->nvc, a.h, nullptr, nullptr, c->d_rhs, 1, c->d_next);
  return cudaGetLastError();
}

cudaError_t launch_amr_jacobi(amps_gpu_ctx* c) {
  TimedLaunch t(c, "jacobi");
  k_amr_invert_diag<<<g1(c->nvc), 256, 0, c->stream>>>(c->nvc, hang_of(c), c->d_diag, c->d_dinv, c->d_dff);
  return cudaGetLastError();
}

cudaError_t launch_amr_update_b(amps_gpu_ctx* c) {
  TimedLaunch t(c, "update_b");
  launch_pdl(k_amr_update_b, dim3(c->nb), dim3(256), 0, c->stream, c->ncor, c->nvc, c->d_ctabh, hang_of(c),
             c->d_bdx, c->d_Eh, c->d_Bc, c->d_Bc2, c->cfg.dt, c->d_energy + 1);
  if (c->mesh_open) {
    const int* nf = c->amrdev.nfine;
    for (int pass = 0; pass <= (c->neumann ? 3 : 0); pass++)
      k_amr_bnd_b<<<g1(c->ncor), 256, 0, c->stream>>>(c->ncor, c->d_borg, c->d_bscale, nf[0], nf[1], nf[2],
                                                       c->mesh_open, c->neumann, pass, c->d_Bc, c->d_Bc2);
  }
  return cudaGetLastError();
}

// hanging corners of F, optionally with their wave energy
static cudaError_t fix_hanging(amps_gpu_ctx* c, double* F, const double* cvol, double* energy) {
  if (c->nsrows == 0) return cudaSuccess;
  launch_pdl(k_amr_fix_hanging, dim3(g1(c->nsrows)), dim3(256), 0, c->stream, c->nsrows, c->d_srows, c->nvc,
             hang_of(c), F, cvol, energy);
  return cudaGetLastError();
}

cudaError_t launch_amr_c2n(amps_gpu_ctx* c, const double* Bcen, double* Bcor) {
  cudaError_t e = cudaMemsetAsync(Bcor, 0, sizeof(double) * 3 * c->nvc, c->stream);
  if (e != cudaSuccess) return e;
  TimedLaunch t(c, "c2n", 2);
  launch_pdl(k_amr_c2n, dim3(c->nb), dim3(256), 0, c->stream, c->ncor, c->nvc, c->d_ctab, c->d_bdx,
             c->d_cinv, Bcen, Bcor);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return fix_hanging(c, Bcor, nullptr, nullptr);
}

cudaError_t launch_amr_update_e(amps_gpu_ctx* c) {
  cudaError_t e;
  TimedLaunch t(c, "update_e", 2);
  const double th = c->cfg.theta;
  const unsigned grid = (unsigned)std::min<long long>((std::max(c->nvc, c->ncor) + 255) / 256, 152LL * 8);
  launch_pdl(k_amr_update_e, grid, dim3(256), 0, c->stream, c->ncor, c->nvc, c->d_Eh, c->d_En, 1.0 / th,
             (1.0 - th) / th, c->d_cvol, c->d_bdx, c->d_Bc, c->d_energy + 1);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return fix_hanging(c, c->d_En, c->d_cvol, c->d_energy + 1);
}
