// Corner assembly shared by the uniform context deposit (particles.cu) and the
// no-allocation entry point (noalloc.cu): per-cell partial sums (27 weight
// monomials x 9, 8 corners x 3) -> the 243-term mass matrix M and current J of
// the corners (ProcessCell's flush, pic_field_solver_ecsim.cpp:2362-2426, with
// the shared corners summed).
//
// Slot (dx, dy, dz) of corner c sums, over the cells in which both c and its
// partner at offset (dx, dy, dz) are corners, the cell's block of the pair's
// weight monomial: per axis, with l the corner's offset bit in the cell, offset
// 0 takes the cells l = 0 and 1, -1 the cell l = 1, +1 the cell l = 0, and the
// monomial digit is 2 l + d.
//
// A CTA takes 32 corners (8 x 4 x 1 of a block) and stages the 9 x 5 x 2 cells
// around them, 87.5 KB, in shared memory by asynchronous copies (16 bytes at a
// time for the ten rows of 8 cells of one block, 4 for the ten cells left of
// them).  Read straight from global memory, the 64 blocks of 36 bytes that a
// corner needs touch one cache line per lane and load, and that line rate
// bounds the kernel; the staged copy is read at a cell stride of 243 words (19
// banks) and a row stride of 24 banks, conflict-free within the rows.  The 64
// entries of a corner split evenly over the 8 warps: slot 0 (8 cells), the 6
// face slots (4 each) on three warps, the 12 edge slots (2 each) on three, the 8
// vertex slots on one.  Every slot adds its cells in the order of the corner's
// offset bits, x fastest.
#pragma once

#include "common.cuh"
#include "ptx.cuh"

namespace {

constexpr int kAsmCorners = 32;              // 8 x 4 x 1 corners of a block per CTA
constexpr int kAsmPerBlock = AMPS_CPB / kAsmCorners;
constexpr int kAsmRows = 10;                 // rows of 8 cells: 5 in y, 2 in z
constexpr int kAsmRowF = 8 * AMPS_CELLM;     // floats of a row
constexpr int kAsmThreads = 256;
constexpr size_t kAsmSmem = sizeof(float) * (kAsmRows * kAsmRowF + kAsmRows * AMPS_CELLM);

// slots by the number of entries: warp w of 8 takes s_asm_slot[first[w] .. first[w+1])
__constant__ unsigned char c_asm_slot[27] = {0,  1,  2,  3,  6,  9,  18, 4,  5,  7,  8,  10, 11, 19,
                                             20, 12, 15, 21, 24, 13, 14, 16, 17, 22, 23, 25, 26};
__constant__ unsigned char c_asm_first[9] = {0, 1, 3, 5, 7, 11, 15, 19, 27};

// Stage the cells around the corners (0..7, j0..j0+3, k0) of a block; cell_id(i,
// j, k) maps block-local cell indices in [-1, 8) to a cell.
template <class CellId>
__device__ __forceinline__ void asm_stage(float* s_c, const float* __restrict__ cellM, int j0, int k0,
                                          const CellId& cell_id) {
  __shared__ long long s_id[2 * kAsmRows];  // per row: its first cell, the cell left of it
  if (threadIdx.x < 2 * kAsmRows) {
    const int r = threadIdx.x >> 1;
    s_id[threadIdx.x] = cell_id(-(int)(threadIdx.x & 1), j0 - 1 + r % 5, k0 - 1 + r / 5) * AMPS_CELLM;
  }
  __syncthreads();
#pragma unroll 4
  for (int t = threadIdx.x; t < kAsmRows * (kAsmRowF / 4); t += kAsmThreads) {
    const int r = t / (kAsmRowF / 4), q = t - r * (kAsmRowF / 4);
    cp_async16(s_c + 4 * t, cellM + s_id[2 * r] + 4 * q);
  }
#pragma unroll 2
  for (int t = threadIdx.x; t < kAsmRows * AMPS_CELLM; t += kAsmThreads) {
    const int r = t / AMPS_CELLM, q = t - r * AMPS_CELLM;
    cp_async4(s_c + kAsmRows * kAsmRowF + t, cellM + s_id[2 * r + 1] + q);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// slot of corner `lane` of the tile: acc[9]
__device__ __forceinline__ void asm_slot(const float* __restrict__ s_c, int slot, int lane, float (&acc)[9]) {
  const int i = lane & 7, j = lane >> 3;
  int d[3] = {slot % 3, (slot / 3) % 3, slot / 9};
  int lo[3], hi[3];  // the corner's offset bits in the slot's cells
#pragma unroll
  for (int a = 0; a < 3; a++) {
    d[a] = d[a] == 0 ? 0 : (d[a] == 1 ? -1 : 1);
    lo[a] = d[a] < 0 ? 1 : 0;
    hi[a] = d[a] > 0 ? 0 : 1;
  }
#pragma unroll
  for (int e = 0; e < 9; e++) acc[e] = 0.f;
  for (int lz = lo[2]; lz <= hi[2]; lz++)
    for (int ly = lo[1]; ly <= hi[1]; ly++)
      for (int lx = lo[0]; lx <= hi[0]; lx++) {
        const int mono = (2 * lx + d[0]) + 3 * (2 * ly + d[1]) + 9 * (2 * lz + d[2]);
        const int row = (j - ly + 1) + 5 * (1 - lz), ii = i - lx;
        const float* src = (ii >= 0 ? s_c + row * kAsmRowF + ii * AMPS_CELLM
                                    : s_c + kAsmRows * kAsmRowF + row * AMPS_CELLM) +
                           mono * 9;
#pragma unroll
        for (int e = 0; e < 9; e++) acc[e] += src[e];
      }
}

// The warp's slots of corner `lane` of the tile: out(slot, acc[9])
template <class Out>
__device__ __forceinline__ void asm_slots(const float* __restrict__ s_c, int wid, int lane, const Out& out) {
  for (int q = c_asm_first[wid]; q < c_asm_first[wid + 1]; q++) {
    const int slot = c_asm_slot[q];
    float acc[9];
    asm_slot(s_c, slot, lane, acc);
    out(slot, acc);
  }
}
constexpr int kAsmMaxSlots = 8;  // of a warp

// component d of corner (i, j, k)'s current: the sum over its 8 cells
template <class CellId>
__device__ __forceinline__ float asm_current(const float* __restrict__ cellJ, int i, int j, int k, int d,
                                             const CellId& cell_id) {
  float s = 0.f;
#pragma unroll
  for (int co = 0; co < 8; co++) {
    const long long c = cell_id(i - (co & 1), j - ((co >> 1) & 1), k - (co >> 2));
    s += cellJ[c * 24 + (co ^ ((co >> 1) & 1)) * 3 + d];  // the table order of the corners
  }
  return s;
}

}  // namespace
