// march.cuh -- warps that march along j: FP32 stencils without shared memory.
//
// A shared-memory tile kernel pays for every intermediate with index arithmetic, a store, a
// barrier and its neighbours' loads; in FP32 those instructions and waits, not the memory, bound
// the stencils.  Here a warp owns a strip of columns (lane = i) and a chunk of rows, and marches
// along j: what a row needs from the rows before it stays in registers, what it needs from the
// neighbouring columns comes from the neighbouring lanes (shuffles, one instruction a value) or,
// for raw inputs, from L1.  Nothing waits on a barrier, and the next row's loads are in flight
// while a row is computed.  A strip's outer lanes hold the apron the shuffles consume.
//
// Addresses: a field is read at a 64-bit byte offset from its interior origin, a kernel
// parameter, so that an access costs one 64-bit addition and its pointer holds no registers
// between rows (a pointer a field, kept or recomputed, was measured to take more instructions
// than the arithmetic of fvtp2d).
#pragma once

#include <cuda_runtime.h>

#include "precision.cuh"
#include "stencil_util.cuh"

namespace oeb {

constexpr unsigned kWarpMask = 0xFFFFFFFFu;

// The value of lane - D (the lane's own where there is none) and of lane + D.
template <int D>
__device__ __forceinline__ float lane_below(float x) {
  return __shfl_up_sync(kWarpMask, x, D);
}
template <int D>
__device__ __forceinline__ float lane_above(float x) {
  return __shfl_down_sync(kWarpMask, x, D);
}
// Whether this lane or the one below it is set.
__device__ __forceinline__ bool here_or_below(bool c) {
  const unsigned m = __ballot_sync(kWarpMask, c);
  return ((m | (m << 1)) >> threadIdx.x) & 1u;
}

// The field p at byte offset o.
__device__ __forceinline__ float get(const float* p, int64_t o) {
  return ld(reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + o));
}
__device__ __forceinline__ void put(float* p, int64_t o, float v) {
  *reinterpret_cast<float*>(reinterpret_cast<char*>(p) + o) = v;
}

// Strip and chunk of a marching warp: a CTA's 8 warps are 2^wx_log strips x the rest in chunks of rows.
struct MarchPos {
  int strip, chunk;
};
__device__ __forceinline__ MarchPos march_pos(const uint3& blk, int wx_log) {
  const int w = (int)threadIdx.y;
  return MarchPos{(int)((blk.x << wx_log) + (w & ((1 << wx_log) - 1))),
                  (int)(blk.y * (kTY >> wx_log) + (w >> wx_log))};
}

// How a marching kernel covers nx x ny x nz: rows a chunk, strips a CTA (as a logarithm) and the
// grid (strips, chunks, groups of kb levels).
struct MarchShape {
  int rows, wx_log;
  dim3 grid;
};
// cols: columns a strip writes; apron: rows a chunk marches beyond its own; ctas_per_sm: CTAs the
// kernel's registers allow.
MarchShape march_shape(int nx, int ny, int nz, int kb, int cols, int apron, int ctas_per_sm);
// Levels a chunk for a kernel that marches nz levels with `ctas` CTAs a chunk and forms two levels
// beyond its own.
int march_levels(int ctas, int nz, int ctas_per_sm);

}  // namespace oeb
