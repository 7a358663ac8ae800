// BF16 tensor-core inference of the learned preconditioner on sm_103a:
// tcgen05.mma with FP32 accumulators in tensor memory, two CTAs per mesh block.
//
// Each 3x3x3 convolution over the region R of 10^3 voxels is an implicit GEMM.
// An x-plane of R is one tile of 128 accumulator rows: voxel (i, j, k) is row
// j + 11 k of plane i, so a tap (dy, dz) is a shift of dy + 11 dz rows (the zero
// rows j = 10 and 110 .. 127 are the ring; a plane's lower ring is the end of the
// plane before it).  Activations live in shared memory as BF16 planes of 8
// channels, 16 bytes per row, so the A operand of a tap is the same buffer read
// from a shifted row: a K-major, non-swizzled operand whose 8x16-byte core matrices
// are 8 consecutive rows (stride-dimension offset 128 B) and whose next 8 channels
// are the next channel plane (leading-dimension offset = its size).  A tap's dx
// moves the output by whole tiles: the three dx of one (dy, dz) are side by side in
// the B operand, [dx = +1 | 0 | -1], and one MMA adds input plane x to the
// accumulators of planes x-1, x and x+1, which are neighbours in tensor memory.
// The first (dy, dz) and K chunk goes by single planes, the centre one first and
// without accumulation, as it starts the sums.
//
// A cluster of two CTAs serves one mesh block; each computes 5 output planes from
// 6 input planes, counted from the block's outside: u = 0 .. 4 its own, 5 the
// peer's nearest.  One thread issues the MMAs of 128 x N x 16 (N = 32 a plane, 16
// in the 3-channel output layer), those of u < 4 first; each half is committed to
// its own mbarrier.  Warps 0-3 read planes 0-2 back (tcgen05.ld, 32 lanes a warp)
// and write the next layer's rows while the second half runs, warps 4-7 planes 3-4.
// Once the peer's MMAs have read their plane 5 (a split cluster barrier), plane 4
// is written there too (distributed shared memory); the first half of the next
// layer doesn't need it and is issued before.  The last layer writes the owned
// voxels' FP32 output.
//
// What bounds it: an MMA of M = 128 and K = 16 takes 40 cycles at N = 16 and 32
// alike (its A rows come from shared memory) and 64 at N = 96, so three dx per MMA
// count (294 MMAs per CTA instead of 810), and an issue loop in uniform control flow
// (one elected thread, descriptors in uniform registers; a loop under tid == 0 issues
// one MMA in 74 cycles); these are 15,000 of the kernel's 25,000 cycles (13 us, warm),
// the chain gather - read-back - exchange the rest.  64 blocks of a mesh: 27 us between
// events around an application in a solve (launch, events and cold inputs included);
// with an MMA per tap, 4 warps and one commit a layer 60.
// Shared memory per CTA: 4 channel planes (82,944 B) + the three layers'
// BF16 weight images (110,592 B, one bulk copy); tensor memory: 256 columns.
// Every mbarrier wait is bounded; a timeout is counted in flags[2] and the CTA
// still takes part in every cluster barrier, so its peer never waits on it.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "precond.cuh"
#include "ptx.cuh"

namespace {

constexpr int kLead = 16;                   // zero rows before plane 0 (a tap reaches 12 back)
constexpr int kRows = kLead + 10 * 128;     // ten x-planes of 128 rows
constexpr int kPlane = kRows * 16;          // bytes per 8-channel BF16 plane
constexpr int kActBytes = 4 * kPlane;       // 82,944
constexpr int kSplit = 2;                   // CTAs (cluster) per mesh block
constexpr int kMine = 5;                    // output planes per CTA
constexpr int kFirst = 3;                   // of these read back by warps 0-3
constexpr int kW1 = 27 * 2 * 4 * 128;       // K 16 (3 used), N 32
constexpr int kW2 = 27 * 4 * 4 * 128;       // K 32, N 32
constexpr int kW3 = 27 * 4 * 2 * 128;       // K 32, N 16 (3 used)
constexpr int kWBytes = kW1 + kW2 + kW3;    // 110,592
constexpr int kSmem = kActBytes + kWBytes + 64;
constexpr int kThreads = 256;
constexpr int kTmemCols = 256;              // kMine x 32 columns, a power of two
constexpr uint32_t kWait = 1u << 24;

// shared-memory matrix descriptor: no swizzle, K-major
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of tcgen05
  return d;
}

// instruction descriptor, kind::f16: BF16 A and B (K-major), FP32 D, M = 128
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t ad, uint64_t bd, uint32_t idesc,
                                         uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(ad), "l"(bd), "r"(idesc), "r"(accum)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void fence_async_cluster() {
  asm volatile("fence.proxy.async;" ::: "memory");
}

// 16 consecutive accumulator columns of this warp's 32 lanes; the registers are
// valid only after tmem_wait() and reg_fence16()
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t r[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// orders every use of r after the preceding tmem_wait()
__device__ __forceinline__ void reg_fence16(uint32_t r[16]) {
  asm volatile(""
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                 "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]));
}

// shared::cluster address of the same offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_addr(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w)
               : "memory");
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_sync() {
  cluster_arrive();
  cluster_wait();
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ int act_row(int i, int j, int k) { return kLead + 128 * i + 11 * k + j; }

__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.b32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p != 0;
}

// The MMAs of one half of layer L (0: input planes u < 4, and the first of every
// sum; 1: u = 4, 5).  Called by a converged warp.
template <int L>
__device__ __forceinline__ void issue_half(int half, int rank, uint32_t act_s, uint32_t w_s, uint32_t tmem,
                                           uint64_t* bar) {
  constexpr int N1 = L < 2 ? 32 : 16;   // accumulator columns per plane
  constexpr int G1 = N1 / 8;
  constexpr int KS = L == 0 ? 1 : 2;    // K steps of 16 channels
  const bool el = elect_one();
  const int p0 = rank * kMine;
  // 18 bits of the shared address: in a cluster the rest holds the CTA's rank
  const uint32_t act = act_s & 0x3FFFFu;
  const uint32_t wb = (w_s & 0x3FFFFu) + (L == 0 ? 0 : (L == 1 ? kW1 : kW1 + kW2));
  const uint64_t adesc0 = sdesc(0, kPlane, 128), bdesc0 = sdesc(0, 3 * G1 * 128, 128);
  // input plane x of (dy, dz) t and K step ks into the cnt output planes from lo on
  auto mma = [&](int t, int ks, int x, int lo, int cnt, bool acc) {
    const int off = t % 3 - 1 + 11 * (t / 3 - 1);
    const uint32_t a = act + (uint32_t)(2 * ks * kPlane + (kLead + 128 * x + off) * 16);
    const uint32_t b = wb + (uint32_t)(((t * 2 * KS + 2 * ks) * 3 + lo - (x - 1)) * G1 * 128);
    if (el)
      mma_bf16(tmem + (uint32_t)((lo - p0) * N1), adesc0 | (uint64_t)(a >> 4), bdesc0 | (uint64_t)(b >> 4),
               idesc_bf16(cnt * N1), acc);
  };
  const int u0 = half ? 4 : 0, u1 = half ? 6 : 4;
  if (!half) {
#pragma unroll
    for (int u = 0; u < kMine; u++) {
      const int x = rank ? 9 - u : u;
      mma(0, 0, x, x, 1, false);
    }
  }
#pragma unroll
  for (int u = u0; u < u1; u++) {
    const int x = rank ? 9 - u : u;
    if (x - 1 >= p0 && x - 1 < p0 + kMine) mma(0, 0, x, x - 1, 1, true);
    if (x + 1 >= p0 && x + 1 < p0 + kMine) mma(0, 0, x, x + 1, 1, true);
  }
#pragma unroll 3
  for (int t = 0; t < 9; t++)
#pragma unroll
    for (int ks = 0; ks < KS; ks++) {
      if (t == 0 && ks == 0) continue;
#pragma unroll
      for (int u = u0; u < u1; u++) {
        const int x = rank ? 9 - u : u;
        const int lo = max(x - 1, p0);
        const int cnt = u == 0 || u == 4 ? 2 : (u == 5 ? 1 : 3);
        mma(t, ks, x, lo, cnt, true);
      }
    }
  if (el) mma_commit(bar);
}

// Inputs/outputs: samples mode (x[S][1000][3] -> y[S][1000][3], owned voxels)
// or mesh mode (mesh.v != null: x = dinv .* v gathered around mesh block s
// through in_map, z = x + y written to the FP64 corners of out_map, with the
// weight set set[s] of the block, or set 0 when set is null).
struct MeshIO {
  const double* v;
  const double* dinv;
  const int* in_map;
  const int* hs;  // hanging-corner CSR (AMR), for pc_input
  const int* hp;
  const double* hw;
  const int* out_map;
  const int* set;
  long long nvc;
  double* z;
  float* xf;  // z in FP32, the operator's input
};

__global__ void __cluster_dims__(kSplit, 1, 1) __launch_bounds__(kThreads, 1)
    k_precond_tc(const float* __restrict__ x, float* __restrict__ y,
                 const uint16_t* __restrict__ wimg, unsigned long long* __restrict__ flags,
                 MeshIO mesh) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* act = smem;
  uint8_t* wsm = smem + kActBytes;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + kActBytes + kWBytes);  // [0], [1] MMA halves, [2] weights
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 3);
  const int s = blockIdx.x / kSplit;
  const int rank = (int)(blockIdx.x % kSplit);  // the rank in the cluster
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform, as the issue loop wants it

  if (tid == 0) {
    for (int q = 0; q < 3; q++) mbar_init(&bar[q], 1);
    fence_mbar_init();
    const int wset = (mesh.v && mesh.set) ? mesh.set[s] : 0;
    mbar_arrive_expect_tx(&bar[2], kWBytes);
    bulk_copy_g2s(wsm, wimg + (size_t)wset * (kWBytes / 2), kWBytes, &bar[2]);
  }
  // zero the channel planes of the first layer, and of the others the rows before
  // planes 0 and 4, the lowest of the two CTAs (the lower ring); the rest is written
  // before it is read for a voxel of R
  for (int q = tid; q < 2 * kRows; q += kThreads)
    reinterpret_cast<uint4*>(act)[q] = make_uint4(0u, 0u, 0u, 0u);
  if (tid < 4 * kLead)
    reinterpret_cast<uint4*>(act)[(2 + tid / kLead % 2) * kRows + tid / (2 * kLead) * 4 * 128 + tid % kLead] =
        make_uint4(0u, 0u, 0u, 0u);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tslot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // everything up to here overlaps the end of the kernel before
  pdl_wait();
  pdl_next();
  // layer-1 input, channels 0..2 of channel plane 0
  constexpr int kPer = (1000 + kThreads - 1) / kThreads;
  const float* xs = x + (size_t)s * 1000 * 3;
  float xv[kPer][3];
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const int v = tid + q * kThreads;
#pragma unroll
    for (int ch = 0; ch < 3; ch++) xv[q][ch] = 0.f;
    if (v < 1000) {
      if (mesh.v) {
        const int id = mesh.in_map[(size_t)s * 1000 + v];
#pragma unroll
        for (int ch = 0; ch < 3; ch++)
          xv[q][ch] = (float)pc_input(id, ch, mesh.nvc, mesh.v, mesh.dinv, mesh.hs, mesh.hp, mesh.hw);
      } else {
#pragma unroll
        for (int ch = 0; ch < 3; ch++) xv[q][ch] = __ldg(xs + 3 * v + ch);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; q++) {
    const int v = tid + q * kThreads;
    if (v < 1000)
      *reinterpret_cast<uint4*>(act + (size_t)act_row(v % 10, (v / 10) % 10, v / 100) * 16) =
          make_uint4(pack_bf16(xv[q][0], xv[q][1]), pack_bf16(xv[q][2], 0.f), 0u, 0u);
  }
  fence_async_smem();
  // CTA-uniform status: the warp-collective tcgen05 calls below need it
  bool ok = __syncthreads_and(mbar_wait_bounded(&bar[2], 0, kWait)) != 0;
  const uint32_t tmem = *tslot;
  const uint32_t act_s = smem_u32(act), w_s = smem_u32(wsm);
  const uint32_t act_peer = peer_addr(act_s, (uint32_t)rank ^ 1u);
  // rows of this thread: row o of the planes u = u0 .. u0 + nu - 1
  const int half = warp >> 2, u0 = half ? kFirst : 0, nu = half ? kMine - kFirst : kFirst;
  const int o = (warp & 3) * 32 + lane, k = o / 11, j = o % 11;
  const bool in = o < 110 && j < 10;
  uint4 keep[4];
  int issued = -1;  // the last layer with MMAs on their way

  for (int L = 0; L < 3; L++) {
    tc_fence_after();
    if (warp == 0 && ok) {
      if (L == 0) issue_half<0>(0, rank, act_s, w_s, tmem, &bar[0]);
      if (L == 1) issue_half<1>(0, rank, act_s, w_s, tmem, &bar[0]);
      if (L == 2) issue_half<2>(0, rank, act_s, w_s, tmem, &bar[0]);
    }
    uint32_t r[kFirst][2][16];
    if (L > 0) {
      // the peer's MMAs of the layer before have read its plane u = 5: this CTA's
      // plane u = 4 goes there
      cluster_wait();
      if (half && ok) {
        const uint32_t dst = act_peer + (uint32_t)act_row(rank ? 5 : 4, 0, 0) * 16u + (uint32_t)o * 16u;
#pragma unroll
        for (int q = 0; q < 4; q++)
          st_cluster_v4(dst + (uint32_t)q * kPlane, keep[q]);
      }
      fence_async_cluster();
      cluster_sync();
    }
    if (warp == 0 && ok) {
      fence_async_smem();
      if (L == 0) issue_half<0>(1, rank, act_s, w_s, tmem, &bar[1]);
      if (L == 1) issue_half<1>(1, rank, act_s, w_s, tmem, &bar[1]);
      if (L == 2) issue_half<2>(1, rank, act_s, w_s, tmem, &bar[1]);
    }
    __syncwarp();
    if (ok) issued = L;
    // the accumulators (warp-uniform: tcgen05.ld is a warp's)
    bool mine = false;
    if (ok) mine = __all_sync(0xffffffffu, mbar_wait_bounded(&bar[half], L & 1, kWait)) != 0;
    tc_fence_after();
    if (mine) {
#pragma unroll
      for (int g = 0; g < kFirst; g++) {
        if (g >= nu) break;
        const int N1 = L < 2 ? 32 : 16;
        const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) +
                            (uint32_t)((rank ? kMine - 1 - (u0 + g) : u0 + g) * N1);
        tmem_ld16(ta, r[g][0]);
        if (L < 2) tmem_ld16(ta + 16, r[g][1]);
      }
      tmem_wait();
#pragma unroll
      for (int g = 0; g < kFirst; g++) {
        reg_fence16(r[g][0]);
        reg_fence16(r[g][1]);
      }
      tc_fence_before();
#pragma unroll
      for (int g = 0; g < kFirst; g++) {
        if (g >= nu) break;
        const int i = rank ? 9 - (u0 + g) : u0 + g;
        if (L < 2) {
          // the second half reads no row of planes u < 3 that this changes
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const uint32_t* src = r[g][q >> 1] + 8 * (q & 1);
            uint4 w4 = make_uint4(0u, 0u, 0u, 0u);
            if (in) {
              w4.x = pack_bf16(__uint_as_float(src[0]), __uint_as_float(src[1]));
              w4.y = pack_bf16(__uint_as_float(src[2]), __uint_as_float(src[3]));
              w4.z = pack_bf16(__uint_as_float(src[4]), __uint_as_float(src[5]));
              w4.w = pack_bf16(__uint_as_float(src[6]), __uint_as_float(src[7]));
            }
            if (g == kMine - 1 - kFirst) keep[q] = w4;  // plane u = 4 of warps 4-7
            *reinterpret_cast<uint4*>(act + (uint32_t)q * kPlane + (uint32_t)(act_row(i, 0, 0) + o) * 16u) = w4;
          }
        } else if (in && i >= 1 && i <= 8 && j >= 1 && j <= 8 && k >= 1 && k <= 8) {
          if (mesh.v) {
            // z = D v (FP64) + N(D v) on the block's corner (i-1, j-1, k-1)
            const long long id = mesh.out_map[(size_t)s * 512 + (i - 1) + 8 * ((j - 1) + 8 * (k - 1))];
            if (id >= 0) {
#pragma unroll
              for (int ch = 0; ch < 3; ch++) {
                const double z = mesh.dinv[ch * mesh.nvc + id] * mesh.v[ch * mesh.nvc + id] +
                                 (double)__uint_as_float(r[g][0][ch]);
                mesh.z[ch * mesh.nvc + id] = z;
                mesh.xf[ch * mesh.nvc + id] = (float)z;
              }
            }
          } else {
            float* dst = y + ((size_t)s * 1000 + (k * 10 + j) * 10 + i) * 3;
            dst[0] = __uint_as_float(r[g][0][0]);
            dst[1] = __uint_as_float(r[g][0][1]);
            dst[2] = __uint_as_float(r[g][0][2]);
          }
        }
      }
    }
    if (L == 2) {
      if (!mine) ok = false;
      break;
    }
    // the rows of the next layer are written, this layer's MMAs have read theirs
    fence_async_smem();
    if (ok) ok = __syncthreads_and(mine) != 0;
    cluster_arrive();
  }
  ok = __syncthreads_and(ok) != 0;
  if (!ok) {
    if (tid == 0) atomicAdd(flags + 2, 1ull);
    // let outstanding MMAs and the weight copy finish before releasing memory
    if (issued >= 0)
      for (int g = 0; g < 2; g++) mbar_wait_bounded(&bar[g], issued & 1, kWait);
    mbar_wait_bounded(&bar[2], 0, kWait);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols)
                 : "memory");
  }
}

// BF16 operand images of the FP32 weights: layer, (dy, dz), K chunk q, dx (+1, 0,
// -1), N group g: core matrix of 8 rows (n = 8g + r) x 8 K elements (k = 8q + e),
// 128 bytes.
__global__ void k_pack_wtc(const float* __restrict__ w1, const float* __restrict__ w2,
                           const float* __restrict__ w3, uint16_t* __restrict__ img) {
  const int total = kWBytes / 2;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < total; q += gridDim.x * blockDim.x) {
    int byte = q * 2, cin, cout, NQ, NG;
    const float* W;
    if (byte < kW1) {
      W = w1; cin = 3; cout = 32; NQ = 2; NG = 4;
    } else if (byte < kW1 + kW2) {
      W = w2; cin = 32; cout = 32; NQ = 4; NG = 4; byte -= kW1;
    } else {
      W = w3; cin = 32; cout = 3; NQ = 4; NG = 2; byte -= kW1 + kW2;
    }
    const int core = byte / 128, within = byte % 128;
    const int r = within / 16, e = (within % 16) / 2;
    const int g = core % NG, sl = core / NG % 3, tq = core / (3 * NG), qq = tq % NQ;
    const int t = tq / NQ * 3 + 2 - sl;  // taps count dx fastest
    const int n = 8 * g + r, k = 8 * qq + e;
    const float v = (k < cin && n < cout) ? W[((size_t)t * cin + k) * cout + n] : 0.f;
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    img[q] = *reinterpret_cast<const uint16_t*>(&h);
  }
}

}  // namespace

cudaError_t precond_prepare_tc(PrecondState* P, cudaStream_t st) {
  P->tc_ready = false;
  if (!P->wtc) {
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&P->wtc), (size_t)kWBytes * P->nsets);
    if (e != cudaSuccess) return e;
  }
  k_pack_wtc<<<108, 256, 0, st>>>(P->w[0], P->w[1], P->w[2],
                                  P->wtc + (size_t)P->active * (kWBytes / 2));
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) P->tc_ready = true;
  return e;
}

static cudaError_t set_tc_attr() {
  static unsigned long long attr_set = 0;  // per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!((attr_set >> dev) & 1ull)) {
    cudaError_t e = cudaFuncSetAttribute(k_precond_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return e;
    attr_set |= 1ull << dev;
  }
  return cudaSuccess;
}

cudaError_t precond_forward_tc(PrecondState* P, cudaStream_t st, int S, const float* x, float* y) {
  if (!P->tc_ready || !P->flags) return cudaErrorInvalidValue;
  cudaError_t e = set_tc_attr();
  if (e != cudaSuccess) return e;
  MeshIO none{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, nullptr, nullptr};
  k_precond_tc<<<S * kSplit, kThreads, kSmem, st>>>(x, y, P->wtc + (size_t)P->active * (kWBytes / 2),
                                                    P->flags, none);
  return cudaGetLastError();
}

cudaError_t precond_apply_tc_mesh(PrecondState* P, cudaStream_t st, int nb, const int* in_map,
                                  const int* hs, const int* hp, const double* hw,
                                  const int* out_map, const int* set, long long nvc,
                                  const double* v, const double* dinv, double* z, float* xf) {
  if (!P->tc_ready || !P->flags) return cudaErrorInvalidValue;
  cudaError_t e = set_tc_attr();
  if (e != cudaSuccess) return e;
  MeshIO io{v, dinv, in_map, hs, hp, hw, out_map, set, nvc, z, xf};
  // (the weights were packed long before: only the input is of the kernel before)
  return launch_pdl(k_precond_tc, dim3(nb * kSplit), dim3(kThreads), kSmem, st, nullptr, nullptr, P->wtc,
                    P->flags, io);
}
