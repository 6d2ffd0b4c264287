// k_fvtp2d.cu -- fvtp2d (kernels/fvtp2d.h:4-177, the serial variant) in FP64 and FP32.
//
// FP64: two launches per call, per k-level tiles of 32 x 32 with every PPM intermediate computed
// once per point into shared memory:
//   1. fvtp2d_q:    y-PPM of q -> fy2 (fvtp2d.h:8-37), x-PPM of q -> fx2 (:84-113), then
//                   q_i (:39-51) and q_j (:115-127).  Tiles cover the extended index range
//                   [-3, N+2) of these arrays; each value is written exactly where the
//                   reference writes it (fy2, q_i: i in [-3,N+2); fx2, q_j: j in [-3,N+2)).
//   2. fvtp2d_flux: x-PPM of q_i -> fx1 (:53-82), y-PPM of q_j -> fy1 (:129-158) and the
//                   transport fluxes fx1 = (fx1+fx2)/2 * xfx, fy1 = (fy1+fy2)/2 * yfx (:160-176).
// q_i, q_j, fx2 and fy2 are outputs of the reference signature; launch 2 reads them back
// from global memory (the FP64 pipe, not HBM, bounds this kernel, so storing them costs
// less than recomputing their aprons).  FP32 runs one launch that reads nothing back
// (fvtp2d_march_f32).
//
// Compiled with --fmad=false (see k_pointwise.cu).  In FP32 the monotonicity flag smt5 is decided
// on the exact product (precision.cuh).
#include <type_traits>

#include "oeb_reach.cuh"
#include "precision.cuh"
#include "march.cuh"
#include "stencil_util.cuh"
#include "tangent.cuh"

// Built on its own, this file's bodies and helpers are local to it; the step kernel
// (step.cu) includes it with OEB_BODIES_ONLY and a namespace of its own instead.
#ifndef OEB_BODIES_NS
#define OEB_BODIES_NS
#endif
namespace oeb {
namespace OEB_BODIES_NS {

constexpr int kT = 32;

// PPM edge value al(j) = p1 (q(j-1) + q(j)) + p2 (q(j-2) + q(j+1))   (fvtp2d.h:12)
template <class T>
__device__ __forceinline__ T ppm_al(T p1, T p2, T qm2, T qm1, T q0, T qp1) {
  return (p1 * (qm1 + q0)) + (p2 * (qm2 + qp1));
}

// fvtp2d.h:20-23: almq = al - q, br = al(+1) - q, smt5 = almq*br < 0 (b0 = almq + br is formed
// where it is used: ppm_flux uses one of its two b0 operands, so forming it there is one
// addition a flux point, as storing it was one an aux point, of the same operands)
template <class T>
__device__ __forceinline__ void ppm_aux(T al0, T al1, T q0, T* almq, T* br, unsigned char* smt) {
  const T m = al0 - q0;
  const T r = al1 - q0;
  *almq = m;
  *br = r;
  *smt = Prec<T>::prod_lt0(m, r);
}

// fvtp2d.h:28-34: upwind flux at point j from the aux values at j-1 and j.  The flag sum
// smt5(j-1) + smt5(j)*(smt5(j-1)==0) is exactly 1.0 when either flag is set, else 0.0.
// Branch-free: each lane selects the operands of its upwind side and performs that side's
// FP64 operations, (1 - c)(br - c b0) as 1 + (-c) and br + (-(c b0)) -- the same values, an
// IEEE subtraction being the addition of the negation -- so no warp runs both sides.
template <class T>
__device__ __forceinline__ T ppm_flux(T c, T q_m1, T q_0, T almq_m1, T br_m1, T almq_0, T br_0, unsigned char smt_m1,
                                      unsigned char smt_0) {
  const bool pos = gt0(c);
  const T u = T(1.) + (pos ? -c : c);
  const T b0 = (pos ? almq_m1 : almq_0) + (pos ? br_m1 : br_0);  // fvtp2d.h:22 at the upwind side
  const T p = c * b0;
  const T v = (pos ? br_m1 : almq_0) + (pos ? -p : p);
  return Prec<T>::add_flag(pos ? q_m1 : q_0, u * v, (smt_m1 | smt_0) != 0);
}

// ------------------------------ launch 1 ---------------------------------------------
// The y pass (fy2, fyy, then q_i) and the x pass (fx2, fxx, then q_j) are independent given
// q: each CTA does one of them (blk.z's low bit picks the axis) and holds only the part of
// the q tile and the PPM intermediates that pass reads, with fyy / fxx in the place of al,
// which is dead once the aux values are set (37 KB a CTA in FP64; its 42 registers a thread
// allow five CTAs per SM).
// Tile origin (i0, j0) = (-3 + 32 bx, -3 + 32 by).  Shared layout:
//   y pass: q 32 x 39 (i0+a, j0-3+b); al 32 x 35 (i0+a, j0-1+b), then fyy 32 x 33 (i0+a, j0+b)
//           = yfy * fy2, 0 outside fy2's range; almq/br/smt 32 x 34 (i0+a, j0-1+b)
//   x pass: q 38 x 32 (i0-3+a, j0+b); al 35 x 32 (i0-1+a, j0+b), then fxx 33 x 32 (i0+a, j0+b)
//           = xfx * fx2, 0 outside fx2's range; almq/br/smt 34 x 32 (i0-1+a, j0+b)
template <class T>
struct FvQSmem {
  union {
    struct {
      T q[39][32];
      union {
        T al[35][32];
        T fyy[33][32];
      } e;
      T almq[34][32], br[34][32];
      unsigned char smt[34][32];
    } y;
    struct {
      T q[32][38];
      union {
        T al[32][35];
        T fxx[32][33];
      } e;
      T almq[32][34], br[32][34];
      unsigned char smt[32][34];
    } x;
  } w;
};

template <class T>
struct fvtp2d_q_kernel {
  static constexpr int kStepOp = step_op<T>(kOpFvQ);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, OutPtr<T> q_i, OutPtr<T> q_j,
                                             OutPtr<T> fx2, OutPtr<T> fy2, InPtr<T> q,
                                             InPtr<T> crx, InPtr<T> cry,
                                             InPtr<T> ra_x, InPtr<T> ra_y,
                                             InPtr<T> xfx, InPtr<T> yfx,
                                             InPtr<T> area, T p1, T p2, Dims d, int kb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FvQSmem<T>& s = *reinterpret_cast<FvQSmem<T>*>(smem_raw);
    const int i0 = -3 + (int)blk.x * kT, j0 = -3 + (int)blk.y * kT;
    const int sj = (int)d.sj;
    const int nx = d.nx, ny = d.ny;
    const bool ypass = (blk.z & 1u) == 0;
    const int k0 = (int)(blk.z >> 1) * kb, k1 = min(k0 + kb, d.nz);
    // the cells each phase needs for this tile's outputs (fewer at the output box's far
    // edge: the box is nx+5 wide, so the last tile column holds a few useful columns only)
    auto lim = [](int v, int hi) { return max(0, min(v, hi)); };
    auto qok = [&](int i, int j) { return i >= -3 && i < nx + 3 && j >= -3 && j < ny + 3; };
  #pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int64_t kofs = (int64_t)k * d.sk;
      if (ypass) {
        auto& w = s.w.y;
        const int ax = lim(nx + 2 - i0, 32);   // columns of fy2 and q_i
        const int yfb = lim(ny + 1 - j0, 33);  // rows of fy2 / fyy
        const int qib = lim(ny - j0, 32);      // rows of q_i
        const InPtr<T> late[4] = {cry, yfx, area, ra_y};  // read after the PPM phases
        prefetch_tile<T>(late, kofs, i0, j0, nx, ny, sj);
        // (one row more than the phases read, so that full tiles take the compile-time loop)
        for_region_lim<32, 39>(ax, min(39, max(yfb + 6, qib + 3)), [&](int a, int b) {
          const int i = i0 + a, j = j0 - 3 + b;
          w.q[b][a] = qok(i, j) ? ld(q + kofs + i + j * sj) : T(0);
        });
        __syncthreads();
        for_region_lim<32, 35>(ax, yfb + 2, [&](int a, int b) {
          w.e.al[b][a] = ppm_al(p1, p2, w.q[b][a], w.q[b + 1][a], w.q[b + 2][a], w.q[b + 3][a]);
        });
        __syncthreads();
        for_region_lim<32, 34>(ax, yfb + 1, [&](int a, int b) {
          ppm_aux(w.e.al[b][a], w.e.al[b + 1][a], w.q[b + 2][a], &w.almq[b][a], &w.br[b][a], &w.smt[b][a]);
        });
        __syncthreads();
        for_region_lim<32, 33>(ax, yfb, [&](int a, int b) {
          const int i = i0 + a, j = j0 + b;
          T fyy = T(0);
          if (i >= -3 && i < nx + 2 && j >= 0 && j < ny + 1) {  // fvtp2d.h:26-27
            const int64_t o = kofs + i + j * sj;
            const T f = ppm_flux(ld(cry + o), w.q[b + 2][a], w.q[b + 3][a], w.almq[b][a], w.br[b][a],
                                 w.almq[b + 1][a], w.br[b + 1][a], w.smt[b][a], w.smt[b + 1][a]);
            if (b < kT) fy2[o] = f;
            fyy = ld(yfx + o) * f;  // fvtp2d.h:43
          }
          w.e.fyy[b][a] = fyy;  // al is dead: the aux values are set
        });
        __syncthreads();
        // q_i (fvtp2d.h:48)
        for_region_lim<32, 32>(ax, qib, [&](int a, int b) {
          const int i = i0 + a, j = j0 + b;
          if (i >= -3 && i < nx + 2 && j >= 0 && j < ny) {
            const int64_t o = kofs + i + j * sj;
            q_i[o] = (((w.q[b + 3][a] * ld(area + o)) + w.e.fyy[b][a]) - w.e.fyy[b + 1][a]) / ld(ra_y + o);
          }
        });
        __syncthreads();
      } else {
        auto& w = s.w.x;
        const int xfa = lim(nx + 1 - i0, 33);  // columns of fx2 / fxx
        const int by = lim(ny + 2 - j0, 32);   // rows of fx2 and q_j
        const int qja = lim(nx - i0, 32);      // columns of q_j
        const InPtr<T> late[4] = {crx, xfx, area, ra_x};
        prefetch_tile<T>(late, kofs, i0, j0, nx, ny, sj);
        for_region_lim<38, 32>(min(38, max(xfa + 5, qja + 3)), by, [&](int a, int b) {
          const int i = i0 - 3 + a, j = j0 + b;
          w.q[b][a] = qok(i, j) ? ld(q + kofs + i + j * sj) : T(0);
        });
        __syncthreads();
        for_region_lim<35, 32>(xfa + 2, by, [&](int a, int b) {
          w.e.al[b][a] = ppm_al(p1, p2, w.q[b][a], w.q[b][a + 1], w.q[b][a + 2], w.q[b][a + 3]);
        });
        __syncthreads();
        for_region_lim<34, 32>(xfa + 1, by, [&](int a, int b) {
          ppm_aux(w.e.al[b][a], w.e.al[b][a + 1], w.q[b][a + 2], &w.almq[b][a], &w.br[b][a], &w.smt[b][a]);
        });
        __syncthreads();
        for_region_lim<33, 32>(xfa, by, [&](int a, int b) {
          const int i = i0 + a, j = j0 + b;
          T fxx = T(0);
          if (i >= 0 && i < nx + 1 && j >= -3 && j < ny + 2) {  // fvtp2d.h:102-103
            const int64_t o = kofs + i + j * sj;
            const T f = ppm_flux(ld(crx + o), w.q[b][a + 2], w.q[b][a + 3], w.almq[b][a], w.br[b][a],
                                 w.almq[b][a + 1], w.br[b][a + 1], w.smt[b][a], w.smt[b][a + 1]);
            if (a < kT) fx2[o] = f;
            fxx = ld(xfx + o) * f;  // fvtp2d.h:119
          }
          w.e.fxx[b][a] = fxx;  // al is dead: the aux values are set
        });
        __syncthreads();
        // q_j (fvtp2d.h:124)
        for_region_lim<32, 32>(qja, by, [&](int a, int b) {
          const int i = i0 + a, j = j0 + b;
          if (i >= 0 && i < nx && j >= -3 && j < ny + 2) {
            const int64_t o = kofs + i + j * sj;
            q_j[o] = (((w.q[b][a + 3] * ld(area + o)) + w.e.fxx[b][a]) - w.e.fxx[b][a + 1]) / ld(ra_x + o);
          }
        });
        __syncthreads();
      }
    }
  }
};

// Grid of launch 1: the tiles of the output box [-3, n+2)^2, twice along z (one CTA per axis).
inline dim3 q_grid(const Dims& d, int kb) {
  dim3 g = tile_grid(d.nx + 5, d.ny + 5, d.nz, kT, kT, kb);
  g.z *= 2;
  return g;
}

// ------------------------------ launch 2 ---------------------------------------------
// The x sweep (fx1 from q_i) and the y sweep (fy1 from q_j) are independent: each CTA does
// one of them (blk.z's low bit picks the axis), so a CTA holds one field and one set of PPM
// intermediates (36 KB in FP64: six CTAs per SM) and half the dependent phases.
// Interior tile origin (i0, j0).  Shared layout:
//   x sweep: qi 37 x 32 (i0-3+a, j0+b); al 34 x 32 (i0-1+a, j0+b); almq/br/smt 33 x 32 (i0-1+a, j0+b)
//   y sweep: qj 32 x 37 (i0+a, j0-3+b); al 32 x 34 (i0+a, j0-1+b); almq/br/smt 32 x 33 (i0+a, j0-1+b)
template <class T>
struct FvFluxSmem {
  union {
    struct {
      T qi[32][37];
      T al[32][34];
      T almq[32][33], br[32][33];
      unsigned char smt[32][33];
    } x;
    struct {
      T qj[37][32];
      T al[34][32];
      T almq[33][32], br[33][32];
      unsigned char smt[33][32];
    } y;
  } w;
};

template <class T>
struct fvtp2d_flux_kernel {
  static constexpr int kStepOp = step_op<T>(kOpFvFlux);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, OutPtr<T> fx1, OutPtr<T> fy1,
                                             InPtr<T> q_i, InPtr<T> q_j,
                                             InPtr<T> fx2, InPtr<T> fy2,
                                             InPtr<T> crx, InPtr<T> cry,
                                             InPtr<T> xfx, InPtr<T> yfx, T p1, T p2, Dims d,
                                             int kb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FvFluxSmem<T>& s = *reinterpret_cast<FvFluxSmem<T>*>(smem_raw);
    const int i0 = blk.x * kT, j0 = blk.y * kT;
    const int sj = (int)d.sj;
    const int nx = d.nx, ny = d.ny;
    const bool ysweep = (blk.z & 1u) != 0;
    const int k0 = (int)(blk.z >> 1) * kb, k1 = min(k0 + kb, d.nz);
    // outputs of this tile (fewer at the domain's far edge) and what each phase needs for them
    const int vx = max(0, min(kT, nx - i0)), vy = max(0, min(kT, ny - j0));
  #pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int64_t kofs = (int64_t)k * d.sk;
      if (!ysweep) {
        // ---- x-PPM of q_i -> fx1 and the x transport flux
        const InPtr<T> late[3] = {crx, fx2, xfx};  // read in the last phase only
        prefetch_tile<T>(late, kofs, i0, j0, nx, ny, sj);
        for_region_lim<37, 32>(vx + 5, vy, [&](int a, int b) {
          const int i = i0 - 3 + a, j = j0 + b;
          s.w.x.qi[b][a] = (i < nx + 2 && j < ny) ? ld(q_i + kofs + i + j * sj) : T(0);
        });
        __syncthreads();
        for_region_lim<34, 32>(vx + 2, vy, [&](int a, int b) {
          s.w.x.al[b][a] = ppm_al(p1, p2, s.w.x.qi[b][a], s.w.x.qi[b][a + 1], s.w.x.qi[b][a + 2], s.w.x.qi[b][a + 3]);
        });
        __syncthreads();
        for_region_lim<33, 32>(vx + 1, vy, [&](int a, int b) {
          ppm_aux(s.w.x.al[b][a], s.w.x.al[b][a + 1], s.w.x.qi[b][a + 2], &s.w.x.almq[b][a], &s.w.x.br[b][a],
                &s.w.x.smt[b][a]);
        });
        __syncthreads();
        for_region_lim<32, 32>(vx, vy, [&](int a, int b) {
          const int i = i0 + a, j = j0 + b;
          if (i < nx && j < ny) {
            const int64_t o = kofs + i + j * sj;
            const T f = ppm_flux(ld(crx + o), s.w.x.qi[b][a + 2], s.w.x.qi[b][a + 3], s.w.x.almq[b][a], s.w.x.br[b][a],
                                 s.w.x.almq[b][a + 1], s.w.x.br[b][a + 1], s.w.x.smt[b][a], s.w.x.smt[b][a + 1]);
            fx1[o] = (scale2<-1>(f + ld(fx2 + o)) * ld(xfx + o));  // fvtp2d.h:164
          }
        });
        __syncthreads();
      } else {
        // ---- y-PPM of q_j -> fy1 and the y transport flux
        const InPtr<T> late[3] = {cry, fy2, yfx};
        prefetch_tile<T>(late, kofs, i0, j0, nx, ny, sj);
        for_region_lim<32, 37>(vx, vy + 5, [&](int a, int b) {
          const int i = i0 + a, j = j0 - 3 + b;
          s.w.y.qj[b][a] = (i < nx && j < ny + 2) ? ld(q_j + kofs + i + j * sj) : T(0);
        });
        __syncthreads();
        for_region_lim<32, 34>(vx, vy + 2, [&](int a, int b) {
          s.w.y.al[b][a] = ppm_al(p1, p2, s.w.y.qj[b][a], s.w.y.qj[b + 1][a], s.w.y.qj[b + 2][a], s.w.y.qj[b + 3][a]);
        });
        __syncthreads();
        for_region_lim<32, 33>(vx, vy + 1, [&](int a, int b) {
          ppm_aux(s.w.y.al[b][a], s.w.y.al[b + 1][a], s.w.y.qj[b + 2][a], &s.w.y.almq[b][a], &s.w.y.br[b][a],
                &s.w.y.smt[b][a]);
        });
        __syncthreads();
        for_region_lim<32, 32>(vx, vy, [&](int a, int b) {
          const int i = i0 + a, j = j0 + b;
          if (i < nx && j < ny) {
            const int64_t o = kofs + i + j * sj;
            const T f = ppm_flux(ld(cry + o), s.w.y.qj[b + 2][a], s.w.y.qj[b + 3][a], s.w.y.almq[b][a], s.w.y.br[b][a],
                                 s.w.y.almq[b + 1][a], s.w.y.br[b + 1][a], s.w.y.smt[b][a], s.w.y.smt[b + 1][a]);
            fy1[o] = (scale2<-1>(f + ld(fy2 + o)) * ld(yfx + o));  // fvtp2d.h:173
          }
        });
        __syncthreads();
      }
    }
  }
};

// Grid of launch 2: the tiles of the interior, twice along z (one CTA per axis).
inline dim3 flux_grid(const Dims& d, int kb) {
  dim3 g = tile_grid(d.nx, d.ny, d.nz, kT, kT, kb);
  g.z *= 2;
  return g;
}

// ------------------------------ FP32: one marching launch ----------------------------
// FP32 runs both sweeps of q and the sweeps of q_i and q_j in one launch of marching warps
// (march.cuh): lane = column i0 - 3 + lane, 26 columns a strip (the x sweeps' shuffles consume an
// apron of three lanes below and three above), rows from ja - 3 to jb + 2 of a chunk [ja, jb).
// At iteration s a warp holds q on rows s .. s+3 and computes
//   the y sweep's edge value at s+2, aux values and flux fy2 at s+1, and from it q_i at s;
//   the x sweep of row s: fx2, and q_j at s;
//   the x sweep of q_i's row s: fx1;    the y sweep of q_j: fy1 at row s - 2.
// Every input is read once a warp, and q_i, q_j, fx2 and fy2 are never read back.  Each value is
// written by the one warp that owns it: its own 26 columns and rows, plus the columns (rows)
// before the first strip (chunk) and after the last.  The arithmetic is launch 1's and launch
// 2's on the same operands in the same order: the same bits.
//
// What bounds it: instruction issue (70 % of the slots taken) and the latency of its dependent chains
// (about 280 instructions a row of 26 columns, 110 of them the arithmetic; DRAM moves its inputs and
// outputs once).  80 registers, three CTAs an SM: at 256 x 256 x 80 two CTAs (113 registers)
// measured 106 us, four (64, spilling) 110, three 90; two rows unrolled 91 (83 since the lanes off a
// field divide 1 by 1, numerator() in precision.cuh).  Two levels a warp in
// packed FP32 instructions (f32x2) took a quarter fewer instructions but 128 registers: 98 us.
// The form before it, a 32 x 32 shared-memory tile in nine phases, took 180 us (56 against 25 us
// at 128 x 128 x 80).

// The aux values of one cell of a PPM sweep (fvtp2d.h:20-23).  a b < 0 is decided on the exact
// product: with both factors scaled by 2^100 a nonzero product cannot underflow, one that overflows
// keeps its sign, and 0 times an overflow is a NaN, which compares false as 0 does.
struct PpmCell {
  float m, r, b0;  // almq, br, b0
  bool smt;
};
__device__ __forceinline__ PpmCell ppm_cell(float al0, float al1, float q0) {
  constexpr float s = 1.2676506002282294e30f;
  PpmCell c;
  c.m = al0 - q0;
  c.r = al1 - q0;
  c.b0 = c.m + c.r;
  c.smt = (c.m * s) * (c.r * s) < 0.f;
  return c;
}
// The flux at a face (fvtp2d.h:28-34) from its upwind cell's values: ql, rl, bl of the cell below
// the face, qh, mh, bh of the cell above it.  (1 - c) and (1 + c) are both 1 - |c|, and the
// products with c both -(|c| b0), on the side that takes them.
__device__ __forceinline__ float ppm_face(float c, float ql, float rl, float bl, float qh, float mh, float bh,
                                          bool flag) {
  const bool pos = c > 0.f;
  const float n = neg_abs(c);
  const float v = (pos ? rl : mh) + n * (pos ? bl : bh);
  return fmaf((1.f + n) * v, flag ? 1.f : 0.f, pos ? ql : qh);
}

// The x sweep of one row: f the lane's value, c the Courant number of its low face; the flux there.
// Valid from lane 3 to lane 29 (the edge value at i reads i-2 .. i+1, the flux the aux values at
// i-1 and i).
__device__ __forceinline__ float ppm_row(float p1, float p2, float f, float c) {
  const float fm1 = lane_below<1>(f), fm2 = lane_below<2>(f), fp1 = lane_above<1>(f);
  const float al = ppm_al(p1, p2, fm2, fm1, f, fp1);
  const PpmCell x = ppm_cell(al, lane_above<1>(al), f);
  return ppm_face(c, fm1, lane_below<1>(x.r), lane_below<1>(x.b0), f, x.m, x.b0, here_or_below(x.smt));
}

struct fvtp2d_march_f32 {
  static constexpr bool kAnyGrid = true;
  static constexpr int kStepOp = step_op<float>(kOpFvMarch);  // the step kernel's id
  static constexpr int kCols = 26, kApron = 5, kMinCtas = 3;
  // The inputs of iteration s: q on row s + 3, cry and yfx on row s + 1, the rest on s.
  struct Row {
    float q, cry, yfx, crx, xfx, area, rax, ray;
  };
  static __device__ __forceinline__ void run(const uint3& blk, float* __restrict__ q_i, float* __restrict__ q_j,
                                             float* __restrict__ fx1, float* __restrict__ fx2, float* __restrict__ fy1,
                                             float* __restrict__ fy2, const float* __restrict__ q,
                                             const float* __restrict__ crx, const float* __restrict__ cry,
                                             const float* __restrict__ ra_x, const float* __restrict__ ra_y,
                                             const float* __restrict__ xfx, const float* __restrict__ yfx,
                                             const float* __restrict__ area, float p1, float p2, Dims d, int rows,
                                             int wx_log) {
    const MarchPos pos = march_pos(blk, wx_log);
    const int nx = d.nx, ny = d.ny;
    const int i0 = pos.strip * kCols, ja = pos.chunk * rows, jb = min(ja + rows, ny);
    if (i0 >= nx || ja >= ny) return;
    const int lane = (int)threadIdx.x, i = i0 - 3 + lane;
    const bool first_i = i0 == 0, last_i = i0 + kCols >= nx, first_j = ja == 0, last_j = jb == ny;
    const bool own = lane >= 3 && lane < 3 + kCols;
    // columns this lane writes: fy2 and q_i; fx2; q_j, fx1 and fy1 -- and reads
    const bool st_y = i < nx + 2 && (own || (first_i && lane < 3) || (last_i && lane >= 3));
    const bool st_x = i >= 0 && i < nx + 1 && (own || (last_i && lane >= 3));
    const bool st = own && i < nx;
    const bool in_q = i < nx + 3, in_y = i < nx + 2, in_x = i >= 0 && i < nx + 1, in_r = i >= 0 && i < nx;
    const int64_t sjb = d.sj * 4;
    int64_t o = ((int64_t)blk.z * d.sk + (int64_t)(ja - 3) * d.sj + i) * 4;  // (i, s)
    Row nxt{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 1.f, 1.f};  // off a field's reach nothing is read: 0 (divisors 1)
    // the inputs of iteration s, (i, s) at offset c; ALL: every row of them is this chunk's
    auto fetch = [&](auto all, int s, int64_t c) {
      constexpr bool ALL = decltype(all)::value;
      if (in_q && (ALL || s + 3 <= jb + 2)) nxt.q = get(q, c + 3 * sjb);
      if (in_y && (ALL || (s + 1 >= ja && s < jb))) nxt.cry = get(cry, c + sjb), nxt.yfx = get(yfx, c + sjb);  // fy2's
      if (in_x && (ALL || s <= jb + 1)) nxt.crx = get(crx, c), nxt.xfx = get(xfx, c);                          // fx2's
      if (in_y && (ALL || s <= jb + 1)) nxt.area = get(area, c);
      if (in_r && (ALL || s <= jb + 1)) nxt.rax = get(ra_x, c);
      if (in_y && (ALL || (s >= ja && s < jb))) nxt.ray = get(ra_y, c);  // q_i's
    };
    float q0 = 0.f, q1 = 0.f, q2 = 0.f;  // q on rows s, s+1, s+2
    if (in_q) q0 = get(q, o), q1 = get(q, o + sjb), q2 = get(q, o + 2 * sjb);
    float al_lo = 0.f;                        // the y sweep's edge value at s+1
    PpmCell yc = ppm_cell(0.f, 0.f, 0.f);     // its aux values at s
    float fyy0 = 0.f;                         // yfx fy2 at s
    float j1 = 0.f, j2 = 0.f, j3 = 0.f;       // q_j on rows s-1, s-2, s-3
    float jal = 0.f;                          // the edge value of q_j's y sweep at s-2
    PpmCell jc = ppm_cell(0.f, 0.f, 0.f);     // its aux values at s-3
    float cy0 = 0.f, cy1 = 0.f, cy2 = 0.f;    // cry on rows s, s-1, s-2
    float yf0 = 0.f, yf1 = 0.f, yf2 = 0.f;    // yfx
    float fy0 = 0.f, fyA = 0.f, fyB = 0.f;    // fy2 on rows s, s-1, s-2
    // one iteration; ALL: rows s-2 .. s+1 all lie in the chunk
    auto step_row = [&](auto all, int s) {
      constexpr bool ALL = decltype(all)::value;
      const Row w = nxt;
      fetch(all, s + 1, o + sjb);
      // y sweep of q: fy2 at s+1
      const float al_hi = ppm_al(p1, p2, q0, q1, q2, w.q);  // at s+2
      const PpmCell yn = ppm_cell(al_lo, al_hi, q1);        // at s+1
      const float fyn = ppm_face(w.cry, q0, yc.r, yc.b0, q1, yn.m, yn.b0, yc.smt || yn.smt);
      const float fyy1 = w.yfx * fyn;
      if (st_y && (ALL || (s + 1 >= ja && (s + 1 < jb || (last_j && s + 1 == ny))))) put(fy2, o + sjb, fyn);
      // x sweep of q's row s: fx2, and q_j
      const float fxn = ppm_row(p1, p2, q0, w.crx);
      const float fxx = w.xfx * fxn;
      const float qa = q0 * w.area;
      const float jnum = (qa + fxx) - lane_above<1>(fxx);
      const float jn = numerator(in_r, jnum) / w.rax;
      const bool row_own = ALL || ((s >= ja || first_j) && (s < jb || last_j));
      if (st_x && row_own) put(fx2, o, fxn);
      if (st && row_own) put(q_j, o, jn);
      if (ALL || (s >= ja && s < jb)) {
        // q_i, and its x sweep
        const float inum = (qa + fyy0) - fyy1;
        const float qi = numerator(in_y, inum) / w.ray;
        if (st_y) put(q_i, o, qi);
        const float f = ppm_row(p1, p2, qi, w.crx);
        if (st) put(fx1, o, (0.5f * (f + fxn)) * w.xfx);
      }
      // y sweep of q_j: fy1 at s-2
      const float jah = ppm_al(p1, p2, j3, j2, j1, jn);  // the edge value at s-1
      const PpmCell jd = ppm_cell(jal, jah, j2);         // aux at s-2
      const float f1 = ppm_face(cy2, j3, jc.r, jc.b0, j2, jd.m, jd.b0, jc.smt || jd.smt);
      if (st && (ALL || s - 2 >= ja)) put(fy1, o - 2 * sjb, (0.5f * (f1 + fyB)) * yf2);
      q0 = q1, q1 = q2, q2 = w.q;
      al_lo = al_hi, yc = yn, fyy0 = fyy1;
      j3 = j2, j2 = j1, j1 = jn, jal = jah, jc = jd;
      cy2 = cy1, cy1 = cy0, cy0 = w.cry;
      yf2 = yf1, yf1 = yf0, yf0 = w.yfx;
      fyB = fyA, fyA = fy0, fy0 = fyn;
      o += sjb;
    };
    fetch(std::false_type{}, ja - 3, o);
    int s = ja - 3;
  #pragma unroll 1
    for (; s < min(ja + 2, jb + 2); ++s) step_row(std::false_type{}, s);
  #pragma unroll 1
    for (; s < jb - 1; ++s) step_row(std::true_type{}, s);
  #pragma unroll 1
    for (; s < jb + 2; ++s) step_row(std::false_type{}, s);
  }
};

constexpr int kKB = 1;  // k-levels per CTA by default (the most CTAs hide latency best)

template <class T, class M3>
oeb_status fvtp2d_entry(const M3* q_i, const M3* q_j, const M3* fx1, const M3* fx2, const M3* fy1, const M3* fy2,
                        const M3* q, const M3* crx, const M3* cry, const M3* ra_x, const M3* ra_y, const M3* xfx,
                        const M3* yfx, const M3* area, T p1, T p2, const oeb_domain* dom, void* stream) {
  OEB_TRY(check_domain(dom));
  Grid<T> gqi, gqj, gfx1, gfx2, gfy1, gfy2, gq, gcx, gcy, grx, gry, gxf, gyf, gar;
  const Reach rx_ext = kFvFx2;  // fx2 written, crx and xfx read: i in [0,N], j in [-3,N+1]
  const Reach ry_ext = kFvFy2;  // fy2 written, cry and yfx read: i in [-3,N+1], j in [0,N]
  OEB_TRY((check_field3<T>(q_i, *dom, kFvQi, &gqi)));
  OEB_TRY((check_field3<T>(q_j, *dom, kFvQj, &gqj)));
  OEB_TRY((check_field3<T>(fx1, *dom, kInterior, &gfx1)));
  OEB_TRY((check_field3<T>(fx2, *dom, rx_ext, &gfx2)));
  OEB_TRY((check_field3<T>(fy1, *dom, kInterior, &gfy1)));
  OEB_TRY((check_field3<T>(fy2, *dom, ry_ext, &gfy2)));
  OEB_TRY((check_field3<T>(q, *dom, Reach{3, 3, 3, 3, 0, 0}, &gq)));
  OEB_TRY((check_field3<T>(crx, *dom, rx_ext, &gcx)));
  OEB_TRY((check_field3<T>(cry, *dom, ry_ext, &gcy)));
  OEB_TRY((check_field3<T>(ra_x, *dom, Reach{0, 0, 3, 2, 0, 0}, &grx)));
  OEB_TRY((check_field3<T>(ra_y, *dom, Reach{3, 2, 0, 0, 0, 0}, &gry)));
  OEB_TRY((check_field3<T>(xfx, *dom, rx_ext, &gxf)));
  OEB_TRY((check_field3<T>(yfx, *dom, ry_ext, &gyf)));
  OEB_TRY((check_field3<T>(area, *dom, Reach{3, 2, 3, 2, 0, 0}, &gar)));
  OEB_TRY(check_same_strides<T>({&gqi, &gqj, &gfx1, &gfx2, &gfy1, &gfy2, &gq, &gcx, &gcy, &grx, &gry, &gxf,
                                      &gyf, &gar}));
  OEB_TRY(check_no_alias({gqi.lo, gqi.hi, gqj.lo, gqj.hi, gfx1.lo, gfx1.hi, gfx2.lo, gfx2.hi, gfy1.lo, gfy1.hi,
                          gfy2.lo, gfy2.hi},
                         {gq.lo, gq.hi, gcx.lo, gcx.hi, gcy.lo, gcy.hi, grx.lo, grx.hi, gry.lo, gry.hi, gxf.lo,
                          gxf.hi, gyf.lo, gyf.hi, gar.lo, gar.hi}));
  OEB_RETURN_IF_VALIDATING();
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gq.sj, gq.sk};
  cudaStream_t st = (cudaStream_t)stream;
  if constexpr (std::is_same<T, float>::value) {
    using B = fvtp2d_march_f32;
    const MarchShape m = march_shape(d.nx, d.ny, d.nz, 1, B::kCols, B::kApron, B::kMinCtas);
    return launch<B>(m.grid, 0, st, gqi.origin, gqj.origin, gfx1.origin, gfx2.origin, gfy1.origin, gfy2.origin,
                     gq.origin, gcx.origin, gcy.origin, grx.origin, gry.origin, gxf.origin, gyf.origin, gar.origin, p1,
                     p2, d, m.rows, m.wx_log);
  } else {
    const int kb = tuned_kb(kKB);
    OEB_TRY(launch<fvtp2d_q_kernel<T>>(q_grid(d, kb), sizeof(FvQSmem<T>), st, gqi.origin, gqj.origin, gfx2.origin,
                                       gfy2.origin, gq.origin, gcx.origin, gcy.origin, grx.origin, gry.origin,
                                       gxf.origin, gyf.origin, gar.origin, p1, p2, d, kb));
    return launch<fvtp2d_flux_kernel<T>>(flux_grid(d, kb), sizeof(FvFluxSmem<T>), st, gfx1.origin, gfy1.origin,
                                         gqi.origin, gqj.origin, gfx2.origin, gfy2.origin, gcx.origin, gcy.origin,
                                         gxf.origin, gyf.origin, p1, p2, d, kb);
  }
}

// Tangent-linear fvtp2d with respect to q (the PPM flags frozen at q; the Courant numbers,
// fluxes and areas are parameters): derivatives of all six outputs, on Dual<T>.
template <class T, class M3>
oeb_status fvtp2d_tl_entry(const M3* dq_i, const M3* dq_j, const M3* dfx1, const M3* dfx2, const M3* dfy1,
                           const M3* dfy2, const M3* q, const M3* crx, const M3* cry, const M3* ra_x, const M3* ra_y,
                           const M3* xfx, const M3* yfx, const M3* area, const M3* dq, T p1, T p2,
                           const oeb_domain* dom, void* stream) {
  {
    ValidateOnly guard;
    OEB_TRY(fvtp2d_entry<T>(dq_i, dq_j, dfx1, dfx2, dfy1, dfy2, q, crx, cry, ra_x, ra_y, xfx, yfx, area, p1, p2, dom,
                            stream));
    OEB_TRY(fvtp2d_entry<T>(dq_i, dq_j, dfx1, dfx2, dfy1, dfy2, dq, crx, cry, ra_x, ra_y, xfx, yfx, area, p1, p2, dom,
                            stream));
  }
  OEB_RETURN_IF_VALIDATING();
  using D = Dual<T>;
  DualIn<T> x;
  OEB_TRY((dual_in<T>(q, dq, &x)));
  const DualIn<T> cx = dual_param<T>(crx), cy = dual_param<T>(cry), rx = dual_param<T>(ra_x),
                  ry = dual_param<T>(ra_y), xf = dual_param<T>(xfx), yf = dual_param<T>(yfx), ar = dual_param<T>(area);
  cudaStream_t st = (cudaStream_t)stream;
  // launch 2 reads the values of q_i, q_j, fx2 and fy2 as well as their derivatives: scratch for them,
  // each in its output's layout
  const M3* y[4] = {dq_i, dq_j, dfx2, dfy2};
  int64_t n[4], org[4], total = 0;
  for (int f = 0; f < 4; ++f) {
    const T* start = (y[f]->allocated && y[f]->allocated <= y[f]->aligned) ? y[f]->allocated : y[f]->aligned;
    int64_t last = 0;
    for (int r = 0; r < 3; ++r) last += (y[f]->sizes[r] - 1) * y[f]->strides[r];
    n[f] = (int64_t)(y[f]->aligned - start) + last + 1;
    org[f] = total + (int64_t)(y[f]->aligned - start) + y[f]->offset;
    total += n[f];
  }
  void* buf = nullptr;
  OEB_TRY(scratch_alloc(&buf, (size_t)total * sizeof(T), st));
  T* base = static_cast<T*>(buf);
  DualOut<T> o[4];
  DualIn<T> v[4];
  for (int f = 0; f < 4; ++f) {
    o[f] = DualOut<T>{base + org[f], y[f]->aligned + y[f]->offset};
    v[f] = DualIn<T>{o[f].v, o[f].d};
  }
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, q->strides[1], q->strides[0]};
  const int kb = tuned_kb(kKB);
  oeb_status stt = launch<fvtp2d_q_kernel<D>>(q_grid(d, kb), sizeof(FvQSmem<D>), st, o[0], o[1], o[2], o[3], x, cx, cy,
                                              rx, ry, xf, yf, ar, D(p1), D(p2), d, kb);
  if (stt == OEB_OK)
    stt = launch<fvtp2d_flux_kernel<D>>(flux_grid(d, kb), sizeof(FvFluxSmem<D>), st, dual_out<T>(dfx1),
                                        dual_out<T>(dfy1), v[0], v[1], v[2], v[3], cx, cy, xf, yf, D(p1), D(p2), d, kb);
  scratch_free(buf, st);
  return stt;
}

// ============================== adjoint ===========================================
// fvtp2d is linear in q once the PPM flags smt5 (and the upwind choice c > 0) are frozen
// at the state.  With ybar = (fx1b, fy1b) on the interior and gx = xfx fx1b / 2,
// gy = yfx fy1b / 2, the transpose is (fvtp2d.h:39-51, 115-127, 160-176 read backwards):
//   q_ib = PPMx^T(gx) on q_i's flags,  q_jb = PPMy^T(gy) on q_j's flags
//   fy2b = gy + yfx (q_ib / ra_y - q_ib(j-1) / ra_y(j-1)),  fx2b = gx + xfx (q_jb / ra_x - q_jb(i-1) / ra_x(i-1))
//   qb   = area/ra_y q_ib + area/ra_x q_jb + PPMy^T(fy2b) + PPMx^T(fx2b)
// q_i and q_j are recomputed by the forward kernel (recompute, not store).  The transpose
// of one PPM sweep (fvtp2d.h:20-34) is, per flux point j with tb = s (1 -+ c) Fb:
//   B0(j) = [c(j+1)>0] (-c(j+1)) tb(j+1) + [c(j)<=0] c(j) tb(j),  ALM(j) = [c(j)<=0] tb(j) + B0(j)
//   BR(j) = [c(j+1)>0] tb(j+1) + B0(j),  AL(j) = ALM(j) + BR(j-1)
//   gb(j) = [c(j+1)>0] Fb(j+1) + [c(j)<=0] Fb(j) - ALM(j) - BR(j)
//           + p1 (AL(j+1) + AL(j)) + p2 (AL(j+2) + AL(j-1))
// computed per CTA on a 32-line x 44-position shared window (positions A-5 .. A+38 along the
// sweep axis for the 32 outputs A .. A+31).

constexpr int kW = 44;  // window along the sweep axis: outputs A..A+31 need A-5 .. A+38

// Lines a CTA sweeps: 16 (23 KB a CTA: the registers, not shared memory, then bound the CTAs
// per SM, at five or six against four with 32 lines).
template <class T>
constexpr int adj_lines() {
  return 16;
}

// gs and als are dead once the flags smt are set; tb and al take their places
template <class T, int LN>
struct PpmAdjSmem {
  union {
    T gs[LN][kW];  // state values of the swept field
    T al[LN][kW];
  } u0;
  union {
    T als[LN][kW];  // state edge values al
    T tb[LN][kW];
  } u1;
  T alm[LN][kW];
  T br[LN][kW];
  unsigned char smt[LN][kW];
};

// One transposed PPM sweep along AXIS (0: i, 1: j) for outputs A..A+nout-1 on lines
// L0..L0+nl-1 (nout <= 32, nl <= LN: a tile at the edge of its output box works on its own part of
// the window and lines only; every phase's window shrinks by the 32 - nout missing outputs).
// gst(p, l): state value at axis position p of line l (any finite value where the field is not
// defined; its nearest defined one, since a zero takes F64i's slow path);
// cv(p, l): Courant number at flux point p (any value elsewhere);
// fb(p, l): flux adjoint at p (0 off the flux points);  put(a, l, v): receives gbar(a).
template <class T, int AXIS, int LN, class GS, class CV, class FB, class PUT>
__device__ __forceinline__ void ppm_sweep_adjoint(PpmAdjSmem<T, LN>& s, int A, int L0, int nout, int nl, T p1, T p2,
                                                  GS&& gst, CV&& cv, FB&& fb, PUT&& put) {
  const int cut = 32 - nout;
  const bool full = cut == 0 && nl == LN;
  auto region = [&](int w0, int w1, auto&& f) {
    const int tid = threadIdx.y * kTX + threadIdx.x;
    if (full) {  // compile-time extents
      const int W = w1 - w0;
      for (int e = tid; e < W * LN; e += kThreads) {
        int w, l;
        if (AXIS == 0) {
          l = e / W;
          w = w0 + (e - l * W);
        } else {
          w = w0 + e / LN;
          l = e - (e / LN) * LN;
        }
        f(w, l);
      }
      return;
    }
    const int W = w1 - cut - w0;
    if (W <= 0 || nl <= 0) return;
    for (int e = tid; e < W * nl; e += kThreads) {
      int w, l;
      if (AXIS == 0) {
        l = e / W;
        w = w0 + (e - l * W);
      } else {
        w = w0 + e / nl;
        l = e - (e / nl) * nl;
      }
      f(w, l);
    }
  };
  region(0, kW, [&](int w, int l) { s.u0.gs[l][w] = gst(A - 5 + w, L0 + l); });
  __syncthreads();
  region(2, kW - 1, [&](int w, int l) {
    s.u1.als[l][w] = (p1 * (s.u0.gs[l][w - 1] + s.u0.gs[l][w])) + (p2 * (s.u0.gs[l][w - 2] + s.u0.gs[l][w + 1]));
  });
  __syncthreads();
  region(2, kW - 2, [&](int w, int l) {
    s.smt[l][w] = Prec<T>::prod_lt0(s.u1.als[l][w] - s.u0.gs[l][w], s.u1.als[l][w + 1] - s.u0.gs[l][w]);
  });
  __syncthreads();
  region(3, kW - 2, [&](int w, int l) {
    const int p = A - 5 + w;
    const T f = fb(p, L0 + l);
    T t = T(0);
    if (f != T(0) && (s.smt[l][w - 1] | s.smt[l][w])) {
      const T c = cv(p, L0 + l);
      t = f * (T(1) + neg_abs(c));
    }
    s.u1.tb[l][w] = t;
  });
  __syncthreads();
  region(3, kW - 3, [&](int w, int l) {
    const int p = A - 5 + w;
    const T t0 = s.u1.tb[l][w], t1 = s.u1.tb[l][w + 1];
    T b0 = T(0), am = T(0), bb = T(0);
    if (t1 != T(0)) {
      const T c1 = cv(p + 1, L0 + l);
      if (c1 > T(0)) {
        b0 = -c1 * t1;
        bb = t1;
      }
    }
    if (t0 != T(0)) {
      const T c0 = cv(p, L0 + l);
      if (!(c0 > T(0))) {
        b0 = b0 + c0 * t0;
        am = t0;
      }
    }
    s.alm[l][w] = am + b0;
    s.br[l][w] = bb + b0;
  });
  __syncthreads();
  region(4, kW - 3, [&](int w, int l) { s.u0.al[l][w] = s.alm[l][w] + s.br[l][w - 1]; });
  __syncthreads();
  region(5, 5 + 32, [&](int w, int l) {
    const int a = A - 5 + w;
    T g = fma(p1, s.u0.al[l][w + 1] + s.u0.al[l][w], fma(p2, s.u0.al[l][w + 2] + s.u0.al[l][w - 1], -s.alm[l][w])) - s.br[l][w];
    const T f1 = fb(a + 1, L0 + l);
    if (f1 != T(0) && cv(a + 1, L0 + l) > T(0)) g = g + f1;
    const T f0 = fb(a, L0 + l);
    if (f0 != T(0) && !(cv(a, L0 + l) > T(0))) g = g + f0;
    put(a, L0 + l, g);
  });
  __syncthreads();
}

// Pass 1: q_ib over i in [-3,N+2), j in [0,N) and q_jb over i in [0,N), j in [-3,N+2).
template <class T>
struct fvtp2d_adj_qij_kernel {
  static constexpr int kStepOp = step_op<T>(kOpFvAdjQij);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, T* __restrict__ qib, T* __restrict__ qjb,
                                             const T* __restrict__ q_i, const T* __restrict__ q_j,
                                             const T* __restrict__ crx, const T* __restrict__ cry,
                                             const T* __restrict__ xfx, const T* __restrict__ yfx,
                                             const T* __restrict__ fx1b, const T* __restrict__ fy1b, T p1, T p2,
                                             Dims d, int AXIS_Y) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int LN = adj_lines<T>();
    PpmAdjSmem<T, LN>& s = *reinterpret_cast<PpmAdjSmem<T, LN>*>(smem_raw);
    const int nx = d.nx, ny = d.ny, sj = (int)d.sj;
    const int64_t kofs = (int64_t)blk.z * d.sk;
    if (!AXIS_Y) {
      // x sweep of fx1 on q_i: outputs i in [-3, nx+2), lines j in [0, ny)
      const int A = -3 + (int)blk.x * 32, L0 = (int)blk.y * LN;
      ppm_sweep_adjoint<T, 0, LN>(
          s, A, L0, max(0, min(32, nx + 2 - A)), max(0, min(LN, ny - L0)), p1, p2,
          [&](int p, int l) { return ld(q_i + kofs + max(-3, min(p, nx + 1)) + l * sj); },
          [&](int p, int l) { return ld(crx + kofs + p + l * sj); },
          [&](int p, int l) {
            return (p >= 0 && p < nx && l < ny) ? (T(0.5) * ld(xfx + kofs + p + l * sj)) * ld(fx1b + kofs + p + l * sj)
                                               : T(0);
          },
          [&](int a, int l, T v) {
            if (a >= -3 && a < nx + 2 && l < ny) qib[kofs + a + l * sj] = v;
          });
    } else {
      // y sweep of fy1 on q_j: outputs j in [-3, ny+2), lines i in [0, nx)
      const int A = -3 + (int)blk.x * 32, L0 = (int)blk.y * LN;
      ppm_sweep_adjoint<T, 1, LN>(
          s, A, L0, max(0, min(32, ny + 2 - A)), max(0, min(LN, nx - L0)), p1, p2,
          [&](int p, int l) { return ld(q_j + kofs + l + max(-3, min(p, ny + 1)) * sj); },
          [&](int p, int l) { return ld(cry + kofs + l + p * sj); },
          [&](int p, int l) {
            return (p >= 0 && p < ny && l < nx) ? (T(0.5) * ld(yfx + kofs + l + p * sj)) * ld(fy1b + kofs + l + p * sj)
                                               : T(0);
          },
          [&](int a, int l, T v) {
            if (a >= -3 && a < ny + 2 && l < nx) qjb[kofs + l + a * sj] = v;
          });
    }
  }
};

// Pass 2: fy2b on [-3,N+2) x [0,N+1) and fx2b on [0,N+1) x [-3,N+2).
// fy2b(i,j) = g + yfx (ry(i,j) - ry(i,j-1)) with ry = q_ib / ra_y on rows [0, N) (0 elsewhere),
// fx2b(i,j) = g + xfx (rx(i,j) - rx(i-1,j)) with rx = q_jb / ra_x on columns [0, N): each
// quotient is read by two neighbouring points, so a CTA divides once per cell into shared
// memory (ry over its 33 rows j0-1.., rx over its 33 columns i0-1..) and forms both fluxes
// from there.  Tile origin (i0, j0) = (-3 + 32 bx, -3 + 32 by).
template <class T>
struct AdjF2Smem {
  T ry[33][32];  // (i0+a, j0-1+b)
  T rx[32][33];  // (i0-1+a, j0+b)
};

template <class T>
struct fvtp2d_adj_f2_kernel {
  static constexpr int kStepOp = step_op<T>(kOpFvAdjF2);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, T* __restrict__ fx2b, T* __restrict__ fy2b,
                                             const T* __restrict__ qib, const T* __restrict__ qjb,
                                             const T* __restrict__ xfx, const T* __restrict__ yfx,
                                             const T* __restrict__ ra_x, const T* __restrict__ ra_y,
                                             const T* __restrict__ fx1b, const T* __restrict__ fy1b, Dims d, int kb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    AdjF2Smem<T>& s = *reinterpret_cast<AdjF2Smem<T>*>(smem_raw);
    const int nx = d.nx, ny = d.ny;
    const int64_t sj = d.sj;
    const int i0 = -3 + (int)blk.x * kT, j0 = -3 + (int)blk.y * kT;
    // outputs of this tile in the box [-3, nx+2) x [-3, ny+2)
    const int vx = max(0, min(kT, nx + 2 - i0)), vy = max(0, min(kT, ny + 2 - j0));
    const int k0 = blk.z * kb, k1 = min(k0 + kb, d.nz);
  #pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int64_t kofs = (int64_t)k * d.sk;
      for_region_lim<32, 33>(vx, vy + 1, [&](int a, int b) {
        const int i = i0 + a, r = j0 - 1 + b;
        const int64_t o = kofs + i + r * sj;
        s.ry[b][a] = (r >= 0 && r < ny && i < nx + 2) ? div_zero(qib[o], ld(ra_y + o)) : T(0);
      });
      for_region_lim<33, 32>(vx + 1, vy, [&](int a, int b) {
        const int c = i0 - 1 + a, j = j0 + b;
        const int64_t o = kofs + c + j * sj;
        s.rx[b][a] = (c >= 0 && c < nx && j < ny + 2) ? div_zero(qjb[o], ld(ra_x + o)) : T(0);
      });
      __syncthreads();
      for_region_lim<32, 32>(vx, vy, [&](int a, int b) {
        const int i = i0 + a, j = j0 + b;
        const int64_t o = kofs + i + j * sj;
        const bool interior = i >= 0 && i < nx && j >= 0 && j < ny;
        if (j >= 0 && j < ny + 1) {
          T g = interior ? (T(0.5) * ld(yfx + o)) * ld(fy1b + o) : T(0);
          fy2b[o] = g + mul_zero(s.ry[b + 1][a] - s.ry[b][a], ld(yfx + o));
        }
        if (i >= 0 && i < nx + 1) {
          T g = interior ? (T(0.5) * ld(xfx + o)) * ld(fx1b + o) : T(0);
          fx2b[o] = g + mul_zero(s.rx[b][a + 1] - s.rx[b][a], ld(xfx + o));
        }
      });
      __syncthreads();
    }
  }
};

// Pass 3: qb on [-3,N+3)^2: area terms + PPMx^T(fx2b) (x sweep, writes), then
// pass 4: + PPMy^T(fy2b) (y sweep, adds).
template <class T>
struct fvtp2d_adj_q_kernel {
  static constexpr int kStepOp = step_op<T>(kOpFvAdjQ);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, T* __restrict__ qb, const T* __restrict__ q,
                                             const T* __restrict__ crx, const T* __restrict__ cry,
                                             const T* __restrict__ area, const T* __restrict__ ra_x,
                                             const T* __restrict__ ra_y, const T* __restrict__ qib,
                                             const T* __restrict__ qjb, const T* __restrict__ fx2b,
                                             const T* __restrict__ fy2b, T p1, T p2, Dims d, int AXIS_Y) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int LN = adj_lines<T>();
    PpmAdjSmem<T, LN>& s = *reinterpret_cast<PpmAdjSmem<T, LN>*>(smem_raw);
    const int nx = d.nx, ny = d.ny, sj = (int)d.sj;
    const int64_t kofs = (int64_t)blk.z * d.sk;
    auto qval = [&](int i, int j) {
      return ld(q + kofs + max(-3, min(i, nx + 2)) + max(-3, min(j, ny + 2)) * sj);
    };
    const int A = -3 + (int)blk.x * 32, L0 = -3 + (int)blk.y * LN;
    if (!AXIS_Y) {
      // x sweep of fx2 on q: flux points i in [0, nx+1), lines j in [-3, ny+2)
      ppm_sweep_adjoint<T, 0, LN>(
          s, A, L0, max(0, min(32, nx + 3 - A)), max(0, min(LN, ny + 3 - L0)), p1, p2,
          [&](int p, int l) { return qval(p, l); },
          [&](int p, int l) { return ld(crx + kofs + p + l * sj); },
          [&](int p, int l) {
            return (p >= 0 && p < nx + 1 && l >= -3 && l < ny + 2) ? fx2b[kofs + p + l * sj] : T(0);
          },
          [&](int a, int l, T v) {
            if (a >= -3 && a < nx + 3 && l >= -3 && l < ny + 3) {
              const int64_t o = kofs + a + l * sj;
              T acc = v;
              if (a >= -3 && a < nx + 2 && l >= 0 && l < ny) acc = acc + mul_zero(qib[o], ld(area + o) / ld(ra_y + o));
              if (a >= 0 && a < nx && l >= -3 && l < ny + 2) acc = acc + mul_zero(qjb[o], ld(area + o) / ld(ra_x + o));
              qb[o] = acc;
            }
          });
    } else {
      // y sweep of fy2 on q: flux points j in [0, ny+1), lines i in [-3, nx+2); adds to qb
      ppm_sweep_adjoint<T, 1, LN>(
          s, A, L0, max(0, min(32, ny + 3 - A)), max(0, min(LN, nx + 3 - L0)), p1, p2,
          [&](int p, int l) { return qval(l, p); },
          [&](int p, int l) { return ld(cry + kofs + l + p * sj); },
          [&](int p, int l) {
            return (p >= 0 && p < ny + 1 && l >= -3 && l < nx + 2) ? fy2b[kofs + l + p * sj] : T(0);
          },
          [&](int a, int l, T v) {
            if (a >= -3 && a < ny + 3 && l >= -3 && l < nx + 3) qb[kofs + l + a * sj] = qb[kofs + l + a * sj] + v;
          });
    }
  }
};

// ------------------------------ FP32: the adjoint in three marching launches ----------
// The passes above as warps that march rows (march.cuh), with the same operations on the same
// operands (a term that is zero is added where the passes skip it, so that a zero may have the other
// sign):
//   A: q_ib.  The y sweep of q gives q_i a row at a time; its row's transposed x sweep follows at
//      once, the neighbours handed over by the lanes.
//   B: q_jb.  The x sweep of q gives q_j a row at a time, which feeds the transposed y sweep, its
//      window in registers.
//   C: qb.  fx2b and fy2b are formed where they are read, from q_jb and q_ib; a row's transposed x
//      sweep, the transposed y sweep and the area terms meet in one store.
// q_i, q_j, fx2b, fy2b and the partial qb are never stored: two scratch fields instead of eight.
//
// What bounds them: instruction issue (170, 180 and 380 instructions a row for A, B, C; 63, 67 and 75 % of
// the issue slots taken at 256 x 256 x 80).  Four, four and three CTAs an SM: 78.0 us a call at 128 x 128 x 80 (19 + 23 + 43
// with a cold cache), 222 at 256 x 256 x 80, 115 at 201 x 173 x 61 (three CTAs for all 83 / 235 / 113);
// the passes above, run for float, took 154.8, 521.5 and 229.4 us.  Zero numerators that reached the
// division's slow path (numerator(), div_zero()) were 12 us of it at 128 x 128 x 80.

// One face of a transposed sweep: t = tb, z = the product with c of B0 (-(|c| tb) on either side),
// each on the side that takes it (U: the cell below, where c > 0; L: the cell above), and the flux
// adjoint f likewise.
struct FaceT {
  float tU, tL, zU, zL, fU, fL;
};
__device__ __forceinline__ FaceT ppm_face_t(float f, float c, bool limited) {
  const bool pos = c > 0.f;
  const float n = neg_abs(c);
  const bool open = limited && f != 0.f;
  const float t = open ? f * (1.f + n) : 0.f;
  const float z = open ? n * t : 0.f;  // an infinite or NaN c counts only where something passes the face
  return FaceT{pos ? t : 0.f, pos ? 0.f : t, pos ? z : 0.f, pos ? 0.f : z, pos ? f : 0.f, pos ? 0.f : f};
}

// The transposed x sweep of one row: gs the state value at the lane, f and c the flux adjoint and the
// Courant number of its low face.  Valid from lane 5 to lane 26.
__device__ __forceinline__ float ppm_row_t(float p1, float p2, float gs, float f, float c) {
  constexpr float big = 1.2676506002282294e30f;  // 2^100 (ppm_cell)
  const float als = ppm_al(p1, p2, lane_below<2>(gs), lane_below<1>(gs), gs, lane_above<1>(gs));
  const bool smt = ((als - gs) * big) * ((lane_above<1>(als) - gs) * big) < 0.f;
  const FaceT w = ppm_face_t(f, c, here_or_below(smt));
  const float b0 = lane_above<1>(w.zU) + w.zL;
  const float alm = w.tL + b0, br = lane_above<1>(w.tU) + b0;
  const float al = alm + lane_below<1>(br);
  const float g =
      fmaf(p1, lane_above<1>(al) + al, fmaf(p2, lane_above<2>(al) + lane_below<1>(al), -alm)) - br;
  return (g + lane_above<1>(w.fU)) + w.fL;
}

// The transposed y sweep: step() takes the state value at row r and the face r - 2, and gives the
// sweep's value at row r - 5.
struct PpmColumnT {
  float g1 = 0.f, g2 = 0.f, g3 = 0.f;     // the state at r-1, r-2, r-3
  float als = 0.f;                        // its edge value at r-2
  bool smt = false;                       // its flag at r-3
  float tL = 0.f, zL = 0.f;               // of face r-3
  float alm1 = 0.f, alm2 = 0.f;           // alm at r-4, r-5
  float br1 = 0.f, br2 = 0.f;             // br at r-4, r-5
  float al1 = 0.f, al2 = 0.f, al3 = 0.f;  // al at r-4, r-5, r-6
  float fU1 = 0.f, fU2 = 0.f;             // fU of faces r-3, r-4
  float fL1 = 0.f, fL2 = 0.f, fL3 = 0.f;  // fL of faces r-3, r-4, r-5
  __device__ __forceinline__ float step(float p1, float p2, float g0, float f, float c) {
    constexpr float big = 1.2676506002282294e30f;
    const float alsn = ppm_al(p1, p2, g3, g2, g1, g0);  // at r-1
    const bool smtn = ((als - g2) * big) * ((alsn - g2) * big) < 0.f;
    const FaceT w = ppm_face_t(f, c, smt || smtn);
    const float b0 = w.zU + zL;  // of cell r-3
    const float alm = tL + b0, br = w.tU + b0;
    const float al = alm + br1;
    const float g = fmaf(p1, al1 + al2, fmaf(p2, al + al3, -alm2)) - br2;
    const float out = (g + fU2) + fL3;
    g3 = g2, g2 = g1, g1 = g0, als = alsn, smt = smtn;
    tL = w.tL, zL = w.zL;
    alm2 = alm1, alm1 = alm, br2 = br1, br1 = br, al3 = al2, al2 = al1, al1 = al;
    fU2 = fU1, fU1 = w.fU, fL3 = fL2, fL2 = fL1, fL1 = w.fL;
    return out;
  }
};

// A: q_ib over i in [-3, nx+2), j in [0, ny): 22 columns a strip.
struct fvtp2d_adj_qi_f32 {
  static constexpr int kStepOp = step_op<float>(kOpFvAdjQij);  // the step kernel's id
  static constexpr int kCols = 22, kApron = 4, kMinCtas = 4;
  struct Row {
    float q, cry, yfx, area, ray, crx, xfx, fb;  // q on row s + 3, cry and yfx on s + 1, the rest on s
  };
  static __device__ __forceinline__ void run(const uint3& blk, float* __restrict__ qib, const float* __restrict__ q,
                                             const float* __restrict__ crx, const float* __restrict__ cry,
                                             const float* __restrict__ xfx, const float* __restrict__ yfx,
                                             const float* __restrict__ ra_y, const float* __restrict__ area,
                                             const float* __restrict__ fx1b, float p1, float p2, Dims d, int rows,
                                             int wx_log) {
    const MarchPos pos = march_pos(blk, wx_log);
    const int nx = d.nx, ny = d.ny;
    const int a0 = -3 + pos.strip * kCols, ja = pos.chunk * rows, jb = min(ja + rows, ny);
    if (a0 >= nx + 2 || ja >= ny) return;
    const int lane = (int)threadIdx.x, i = a0 - 5 + lane;
    const bool in_y = i >= -3 && i < nx + 2, in_x = i >= 0 && i < nx;
    const bool st = in_y && lane >= 5 && lane < 5 + kCols;
    const int64_t sjb = d.sj * 4;
    int64_t o = ((int64_t)blk.z * d.sk + (int64_t)(ja - 3) * d.sj + i) * 4;  // (i, s)
    Row n{0.f, 0.f, 0.f, 0.f, 1.f, 0.f, 0.f, 0.f};
    auto fetch = [&](auto all, int s, int64_t c) {  // all: every row of them is this chunk's
      constexpr bool ALL = decltype(all)::value;
      if (in_y && (ALL || s + 3 <= jb + 2)) n.q = get(q, c + 3 * sjb);
      if (in_y && (ALL || (s + 1 >= ja && s < jb))) n.cry = get(cry, c + sjb), n.yfx = get(yfx, c + sjb);
      if (ALL || (s >= ja && s < jb)) {
        if (in_y) n.area = get(area, c), n.ray = get(ra_y, c);
        if (in_x) n.crx = get(crx, c), n.xfx = get(xfx, c), n.fb = get(fx1b, c);
      }
    };
    float q0 = 0.f, q1 = 0.f, q2 = 0.f;  // q on rows s, s+1, s+2
    if (in_y) q0 = get(q, o), q1 = get(q, o + sjb), q2 = get(q, o + 2 * sjb);
    float al_lo = 0.f, fyy0 = 0.f;
    PpmCell yc = ppm_cell(0.f, 0.f, 0.f);
    auto step_row = [&](auto all, int s) {
      constexpr bool ALL = decltype(all)::value;
      const Row w = n;
      fetch(all, s + 1, o + sjb);
      const float al_hi = ppm_al(p1, p2, q0, q1, q2, w.q);
      const PpmCell yn = ppm_cell(al_lo, al_hi, q1);
      const float fyy1 = w.yfx * ppm_face(w.cry, q0, yc.r, yc.b0, q1, yn.m, yn.b0, yc.smt || yn.smt);
      if (ALL || s >= ja) {
        const float num = ((q0 * w.area) + fyy0) - fyy1;
        const float qi = numerator(in_y, num) / w.ray;
        const float g = ppm_row_t(p1, p2, in_y ? qi : 0.f, in_x ? (0.5f * w.xfx) * w.fb : 0.f, w.crx);
        if (st) put(qib, o, g);
      }
      q0 = q1, q1 = q2, q2 = w.q;
      al_lo = al_hi, yc = yn, fyy0 = fyy1;
      o += sjb;
    };
    fetch(std::false_type{}, ja - 3, o);
    int s = ja - 3;
#pragma unroll 1
    for (; s < ja; ++s) step_row(std::false_type{}, s);
#pragma unroll 1
    for (; s < jb - 1; ++s) step_row(std::true_type{}, s);
#pragma unroll 1
    for (; s < jb; ++s) step_row(std::false_type{}, s);
  }
};

// B: q_jb over i in [0, nx), j in [-3, ny+2): 26 columns a strip.
struct fvtp2d_adj_qj_f32 {
  static constexpr int kStepOp = step_op<float>(kOpFvAdjF2);  // the step kernel's id
  static constexpr int kCols = 26, kApron = 10, kMinCtas = 4;
  struct Row {
    float q, crx, xfx, area, rax;  // on row r
    float cry, yfx, fb;            // on row r - 2
  };
  static __device__ __forceinline__ void run(const uint3& blk, float* __restrict__ qjb, const float* __restrict__ q,
                                             const float* __restrict__ crx, const float* __restrict__ cry,
                                             const float* __restrict__ xfx, const float* __restrict__ yfx,
                                             const float* __restrict__ ra_x, const float* __restrict__ area,
                                             const float* __restrict__ fy1b, float p1, float p2, Dims d, int rows,
                                             int wx_log) {
    const MarchPos pos = march_pos(blk, wx_log);
    const int nx = d.nx, ny = d.ny;
    const int i0 = pos.strip * kCols, oa = -3 + pos.chunk * rows, ob = min(oa + rows, ny + 2);
    if (i0 >= nx || oa >= ny + 2) return;
    const int lane = (int)threadIdx.x, i = i0 - 3 + lane;
    const bool in_q = i < nx + 3, in_x = i >= 0 && i < nx + 1, in_r = i >= 0 && i < nx;
    const bool st = in_r && lane >= 3 && lane < 3 + kCols;
    const int64_t sjb = d.sj * 4;
    int64_t o = ((int64_t)blk.z * d.sk + (int64_t)(oa - 5) * d.sj + i) * 4;  // (i, r)
    Row n{0.f, 0.f, 0.f, 0.f, 1.f, 0.f, 0.f, 0.f};
    auto fetch = [&](auto all, int r, int64_t c) {  // all: rows r and r - 2 lie in the interior
      constexpr bool ALL = decltype(all)::value;
      if (ALL || (r >= -3 && r < ny + 2)) {
        if (in_q) n.q = get(q, c);
        if (in_x) n.crx = get(crx, c), n.xfx = get(xfx, c);
        if (in_r) n.area = get(area, c), n.rax = get(ra_x, c);
      }
      if (in_r && (ALL || (r - 2 >= 0 && r - 2 < ny)))
        n.cry = get(cry, c - 2 * sjb), n.yfx = get(yfx, c - 2 * sjb), n.fb = get(fy1b, c - 2 * sjb);
    };
    PpmColumnT col;
    auto step_row = [&](auto all, int r) {
      constexpr bool ALL = decltype(all)::value;
      const Row w = n;
      if (ALL || r + 1 < ob + 5) fetch(all, r + 1, o + sjb);
      float qj = 0.f;
      if (ALL || (r >= -3 && r < ny + 2)) {
        const float fxx = w.xfx * ppm_row(p1, p2, w.q, w.crx);
        const float num = ((w.q * w.area) + fxx) - lane_above<1>(fxx);
        qj = numerator(in_r, num) / w.rax;
      }
      const float f = ALL || (r - 2 >= 0 && r - 2 < ny) ? (0.5f * w.yfx) * w.fb : 0.f;
      const float g = col.step(p1, p2, qj, f, w.cry);
      if (st && (ALL || r - 5 >= oa)) put(qjb, o - 5 * sjb, g);
      o += sjb;
    };
    fetch(std::false_type{}, oa - 5, o);
    int r = oa - 5;
    const int ra = min(max(oa + 5, 2), ob + 5), rb = max(ra, min(ob + 4, ny - 1));
#pragma unroll 1
    for (; r < ra; ++r) step_row(std::false_type{}, r);
#pragma unroll 1
    for (; r < rb; ++r) step_row(std::true_type{}, r);
#pragma unroll 1
    for (; r < ob + 5; ++r) step_row(std::false_type{}, r);
  }
};

// C: qb on [-3, n+3)^2: 22 columns a strip.
struct fvtp2d_adj_q_f32 {
  static constexpr int kStepOp = step_op<float>(kOpFvAdjQ);  // the step kernel's id
  static constexpr int kCols = 22, kApron = 10, kMinCtas = 3;
  struct Row {
    float q;                                             // on row r
    float cry, yfx, ray, qi, fy;                         // on row r - 2
    float x, crx, xfx, rax, qj, fx, area, ray5, qi5;     // on row w = r - 5 (x: q)
  };
  static __device__ __forceinline__ void run(const uint3& blk, float* __restrict__ qb, const float* __restrict__ q,
                                             const float* __restrict__ crx, const float* __restrict__ cry,
                                             const float* __restrict__ xfx, const float* __restrict__ yfx,
                                             const float* __restrict__ ra_x, const float* __restrict__ ra_y,
                                             const float* __restrict__ area, const float* __restrict__ fx1b,
                                             const float* __restrict__ fy1b, const float* __restrict__ qib,
                                             const float* __restrict__ qjb, float p1, float p2, Dims d, int rows,
                                             int wx_log) {
    const MarchPos pos = march_pos(blk, wx_log);
    const int nx = d.nx, ny = d.ny;
    const int a0 = -3 + pos.strip * kCols, oa = -3 + pos.chunk * rows, ob = min(oa + rows, ny + 3);
    if (a0 >= nx + 3 || oa >= ny + 3) return;
    const int lane = (int)threadIdx.x, i = a0 - 5 + lane;
    const bool in_q = i >= -3 && i < nx + 3, in_y = i >= -3 && i < nx + 2, in_x = i >= 0 && i < nx + 1,
               in_r = i >= 0 && i < nx;
    const bool st = in_q && lane >= 5 && lane < 5 + kCols;
    const int64_t sjb = d.sj * 4;
    int64_t o = ((int64_t)blk.z * d.sk + (int64_t)(oa - 5) * d.sj + i) * 4;  // (i, r)
    Row n{};
    n.ray = n.rax = n.ray5 = n.area = n.qi = n.qj = 1.f;  // quotients of lanes off the fields are 1 / 1
    auto fetch = [&](auto all, int r, int64_t c) {  // all: rows r, r - 2 and r - 5 lie in the interior
      constexpr bool ALL = decltype(all)::value;
      if (in_q && (ALL || (r >= -3 && r < ny + 3))) n.q = get(q, c);
      const int p = r - 2, w = r - 5;
      const int64_t cp = c - 2 * sjb, cw = c - 5 * sjb;
      if (in_y && (ALL || (p >= 0 && p < ny + 1))) {
        n.cry = get(cry, cp), n.yfx = get(yfx, cp);
        if (ALL || p < ny) {
          n.ray = get(ra_y, cp), n.qi = get(qib, cp);
          if (in_r) n.fy = get(fy1b, cp);
        }
      }
      if (ALL || w >= oa) {
        if (in_q) n.x = get(q, cw);
        if (ALL || w < ny + 2) {
          if (in_x) n.crx = get(crx, cw), n.xfx = get(xfx, cw);
          if (in_y) n.area = get(area, cw);
          if (in_r) n.rax = get(ra_x, cw), n.qj = get(qjb, cw);
        }
        if (ALL || (w >= 0 && w < ny)) {
          if (in_r) n.fx = get(fx1b, cw);
          if (in_y) n.ray5 = get(ra_y, cw), n.qi5 = get(qib, cw);
        }
      }
    };
    PpmColumnT col;
    float ry = 0.f;  // q_ib / ra_y on row r - 3
    auto step_row = [&](auto all, int r) {
      constexpr bool ALL = decltype(all)::value;
      const Row c = n;
      if (ALL || r + 1 < ob + 5) fetch(all, r + 1, o + sjb);
      const int p = r - 2, w = r - 5;
      // the y sweep: face p
      float f = 0.f, ryn = 0.f;
      if (ALL || (p >= 0 && p < ny + 1)) {
        if (ALL || p < ny) ryn = div_zero(c.qi, c.ray);
        const float g = ((ALL || p < ny) && in_r) ? (0.5f * c.yfx) * c.fy : 0.f;
        f = in_y ? g + c.yfx * (ryn - ry) : 0.f;
      }
      ry = ryn;
      const float gy = col.step(p1, p2, (ALL || (r >= -3 && r < ny + 3)) ? c.q : 0.f, f, c.cry);
      if (ALL || w >= oa) {
        // the x sweep of row w
        float fx = 0.f;
        if (ALL || w < ny + 2) {
          const float rxq = div_zero(c.qj, c.rax);
          const float rx = in_r ? rxq : 0.f, rm = lane_below<1>(rx);
          const float g = (in_r && (ALL || (w >= 0 && w < ny))) ? (0.5f * c.xfx) * c.fx : 0.f;
          fx = in_x ? g + c.xfx * (rx - rm) : 0.f;
        }
        float acc = ppm_row_t(p1, p2, c.x, fx, c.crx);
        const float ax = c.area / c.rax;
        if (ALL || (w >= 0 && w < ny)) {
          const float ay = c.area / c.ray5;
          acc = in_y ? acc + ay * c.qi5 : acc;
        }
        if (ALL || w < ny + 2) acc = in_r ? acc + ax * c.qj : acc;
        if (st) put(qb, o - 5 * sjb, acc + gy);
      }
      o += sjb;
    };
    fetch(std::false_type{}, oa - 5, o);
    int r = oa - 5;
    const int ra = min(max(oa + 5, 5), ob + 5), rb = max(ra, min(ob + 4, ny - 1));
#pragma unroll 1
    for (; r < ra; ++r) step_row(std::false_type{}, r);
#pragma unroll 1
    for (; r < rb; ++r) step_row(std::true_type{}, r);
#pragma unroll 1
    for (; r < ob + 5; ++r) step_row(std::false_type{}, r);
  }
};

template <class T, class M3>
oeb_status fvtp2d_adj_entry(const M3* qb, const M3* q, const M3* crx, const M3* cry, const M3* ra_x, const M3* ra_y,
                            const M3* xfx, const M3* yfx, const M3* area, const M3* fx1b, const M3* fy1b, T p1, T p2,
                            const oeb_domain* dom, void* stream) {
  OEB_TRY(check_domain(dom));
  Grid<T> gqb, gq, gcx, gcy, grx, gry, gxf, gyf, gar, gf1, gg1;
  OEB_TRY((check_field3<T>(qb, *dom, Reach{3, 3, 3, 3, 0, 0}, &gqb)));
  OEB_TRY((check_field3<T>(q, *dom, Reach{3, 3, 3, 3, 0, 0}, &gq)));
  OEB_TRY((check_field3<T>(crx, *dom, kFvFx2, &gcx)));
  OEB_TRY((check_field3<T>(cry, *dom, kFvFy2, &gcy)));
  OEB_TRY((check_field3<T>(ra_x, *dom, Reach{0, 0, 3, 2, 0, 0}, &grx)));
  OEB_TRY((check_field3<T>(ra_y, *dom, Reach{3, 2, 0, 0, 0, 0}, &gry)));
  OEB_TRY((check_field3<T>(xfx, *dom, kFvFx2, &gxf)));
  OEB_TRY((check_field3<T>(yfx, *dom, kFvFy2, &gyf)));
  OEB_TRY((check_field3<T>(area, *dom, Reach{3, 2, 3, 2, 0, 0}, &gar)));
  OEB_TRY((check_field3<T>(fx1b, *dom, kInterior, &gf1)));
  OEB_TRY((check_field3<T>(fy1b, *dom, kInterior, &gg1)));
  OEB_TRY(check_same_strides<T>({&gqb, &gq, &gcx, &gcy, &grx, &gry, &gxf, &gyf, &gar, &gf1, &gg1}));
  OEB_TRY(check_no_alias({gqb.lo, gqb.hi}, {gq.lo, gq.hi, gcx.lo, gcx.hi, gcy.lo, gcy.hi, grx.lo, grx.hi, gry.lo,
                                            gry.hi, gxf.lo, gxf.hi, gyf.lo, gyf.hi, gar.lo, gar.hi, gf1.lo, gf1.hi,
                                            gg1.lo, gg1.hi}));
  OEB_RETURN_IF_VALIDATING();
  cudaStream_t st = (cudaStream_t)stream;
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gq.sj, gq.sk};
  // scratch in q's layout: FP32 q_ib, q_jb; FP64 q_i, q_j, fx2, fy2 (forward recompute), q_ib, q_jb, fx2b, fy2b
  const T* start = (q->allocated && q->allocated <= q->aligned) ? q->allocated : q->aligned;
  const int64_t last = (q->sizes[0] - 1) * q->strides[0] + (q->sizes[1] - 1) * q->strides[1] +
                       (q->sizes[2] - 1) * q->strides[2];
  const int64_t n = (int64_t)(q->aligned - start) + last + 1;
  const int64_t org = (int64_t)(q->aligned - start) + q->offset;
  void* buf = nullptr;
  if constexpr (std::is_same<T, float>::value) {
    OEB_TRY(scratch_alloc(&buf, (size_t)n * 2 * sizeof(T), st));
    float *qib = static_cast<float*>(buf) + org, *qjb = qib + n;
    using A = fvtp2d_adj_qi_f32;
    using B = fvtp2d_adj_qj_f32;
    using C = fvtp2d_adj_q_f32;
    const MarchShape ma = march_shape(d.nx + 5, d.ny, d.nz, 1, A::kCols, A::kApron, A::kMinCtas);
    oeb_status stt = launch<A>(ma.grid, 0, st, qib, gq.origin, gcx.origin, gcy.origin, gxf.origin, gyf.origin, gry.origin,
                               gar.origin, gf1.origin, p1, p2, d, ma.rows, ma.wx_log);
    const MarchShape mb = march_shape(d.nx, d.ny + 5, d.nz, 1, B::kCols, B::kApron, B::kMinCtas);
    if (stt == OEB_OK)
      stt = launch<B>(mb.grid, 0, st, qjb, gq.origin, gcx.origin, gcy.origin, gxf.origin, gyf.origin, grx.origin, gar.origin,
                      gg1.origin, p1, p2, d, mb.rows, mb.wx_log);
    const MarchShape mc = march_shape(d.nx + 6, d.ny + 6, d.nz, 1, C::kCols, C::kApron, C::kMinCtas);
    if (stt == OEB_OK)
      stt = launch<C>(mc.grid, 0, st, gqb.origin, gq.origin, gcx.origin, gcy.origin, gxf.origin, gyf.origin, grx.origin,
                      gry.origin, gar.origin, gf1.origin, gg1.origin, qib, qjb, p1, p2, d, mc.rows, mc.wx_log);
    scratch_free(buf, st);
    return stt;
  } else {
    OEB_TRY(scratch_alloc(&buf, (size_t)n * 8 * sizeof(T), st));
    T* base = static_cast<T*>(buf);
    T *sqi = base + org, *sqj = base + n + org, *sfx2 = base + 2 * n + org, *sfy2 = base + 3 * n + org,
      *qib = base + 4 * n + org, *qjb = base + 5 * n + org, *fx2b = base + 6 * n + org, *fy2b = base + 7 * n + org;
    const int kb = tuned_kb(kKB);
    constexpr int LN = adj_lines<T>();
    const size_t ps = sizeof(PpmAdjSmem<T, LN>);
    oeb_status stt = launch<fvtp2d_q_kernel<T>>(q_grid(d, kb), sizeof(FvQSmem<T>), st,
                                                sqi, sqj, sfx2, sfy2, gq.origin, gcx.origin, gcy.origin, grx.origin,
                                                gry.origin, gxf.origin, gyf.origin, gar.origin, p1, p2, d, kb);
    // the x and y sweeps of the two PPM adjoints (axis flag 0 / 1)
    for (int axis = 0; axis < 2 && stt == OEB_OK; ++axis) {
      const int a = axis ? d.ny : d.nx, l = axis ? d.nx : d.ny;
      stt = launch<fvtp2d_adj_qij_kernel<T>>(dim3((a + 5 + 31) / 32, (l + LN - 1) / LN, d.nz), ps, st, qib, qjb, sqi, sqj,
                                             gcx.origin, gcy.origin, gxf.origin, gyf.origin, gf1.origin, gg1.origin, p1,
                                             p2, d, axis);
    }
    if (stt == OEB_OK)
      stt = launch<fvtp2d_adj_f2_kernel<T>>(tile_grid(d.nx + 5, d.ny + 5, d.nz, kT, kT, kb), sizeof(AdjF2Smem<T>), st,
                                            fx2b, fy2b, qib,
                                            qjb, gxf.origin, gyf.origin, grx.origin, gry.origin, gf1.origin, gg1.origin, d,
                                            kb);
    for (int axis = 0; axis < 2 && stt == OEB_OK; ++axis) {
      const int a = axis ? d.ny : d.nx, l = axis ? d.nx : d.ny;
      stt = launch<fvtp2d_adj_q_kernel<T>>(dim3((a + 6 + 31) / 32, (l + 6 + LN - 1) / LN, d.nz), ps, st, gqb.origin,
                                           gq.origin, gcx.origin, gcy.origin, gar.origin, grx.origin, gry.origin, qib, qjb,
                                           fx2b, fy2b, p1, p2, d, axis);
    }
    scratch_free(buf, st);
    return stt;
  }
}

}  // namespace
}  // namespace oeb

#ifndef OEB_BODIES_ONLY  // the entry points

using namespace oeb;

#define OEB_FV_ENTRY(S, T)                                                                                          \
  extern "C" oeb_status oeb_fvtp2d_##S(                                                                            \
      const oeb_memref3d_##S* q_i, const oeb_memref3d_##S* q_j, const oeb_memref3d_##S* fx1,                        \
      const oeb_memref3d_##S* fx2, const oeb_memref3d_##S* fy1, const oeb_memref3d_##S* fy2,                        \
      const oeb_memref3d_##S* q, const oeb_memref3d_##S* crx, const oeb_memref3d_##S* cry,                          \
      const oeb_memref3d_##S* ra_x, const oeb_memref3d_##S* ra_y, const oeb_memref3d_##S* xfx,                      \
      const oeb_memref3d_##S* yfx, const oeb_memref3d_##S* area, T p1, T p2, const oeb_domain* dom, void* stream) {  \
    return fvtp2d_entry<T>(q_i, q_j, fx1, fx2, fy1, fy2, q, crx, cry, ra_x, ra_y, xfx, yfx, area, p1, p2, dom,       \
                           stream);                                                                                \
  }                                                                                                                \
  extern "C" oeb_status oeb_fvtp2d_tl_##S(                                                                         \
      const oeb_memref3d_##S* dq_i, const oeb_memref3d_##S* dq_j, const oeb_memref3d_##S* dfx1,                     \
      const oeb_memref3d_##S* dfx2, const oeb_memref3d_##S* dfy1, const oeb_memref3d_##S* dfy2,                     \
      const oeb_memref3d_##S* q, const oeb_memref3d_##S* crx, const oeb_memref3d_##S* cry,                          \
      const oeb_memref3d_##S* ra_x, const oeb_memref3d_##S* ra_y, const oeb_memref3d_##S* xfx,                      \
      const oeb_memref3d_##S* yfx, const oeb_memref3d_##S* area, const oeb_memref3d_##S* dq, T p1, T p2,            \
      const oeb_domain* dom, void* stream) {                                                                       \
    return fvtp2d_tl_entry<T>(dq_i, dq_j, dfx1, dfx2, dfy1, dfy2, q, crx, cry, ra_x, ra_y, xfx, yfx, area, dq, p1,  \
                              p2, dom, stream);                                                                    \
  }                                                                                                                \
  extern "C" oeb_status oeb_fvtp2d_adj_##S(                                                                        \
      const oeb_memref3d_##S* qb, const oeb_memref3d_##S* q, const oeb_memref3d_##S* crx,                          \
      const oeb_memref3d_##S* cry, const oeb_memref3d_##S* ra_x, const oeb_memref3d_##S* ra_y,                      \
      const oeb_memref3d_##S* xfx, const oeb_memref3d_##S* yfx, const oeb_memref3d_##S* area,                       \
      const oeb_memref3d_##S* fx1b, const oeb_memref3d_##S* fy1b, T p1, T p2, const oeb_domain* dom,                \
      void* stream) {                                                                                              \
    return fvtp2d_adj_entry<T>(qb, q, crx, cry, ra_x, ra_y, xfx, yfx, area, fx1b, fy1b, p1, p2, dom, stream);      \
  }

OEB_FV_ENTRY(f64, double)
OEB_FV_ENTRY(f32, float)

#endif  // OEB_BODIES_ONLY
