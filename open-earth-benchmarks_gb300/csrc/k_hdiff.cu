// k_hdiff.cu -- horizontal diffusion stencils whose intermediates are shared by neighbouring
// points: hdiffsa (kernels/hdiffsa.h:95-123) and hdiffsmag (kernels/hdiffsmag.h:205-263), in
// FP64 (bit-identical to the reference) and FP32 (hdiffsa with exact limiter sign tests;
// hdiffsmag the reference's float sequence, bit-identical to the reference compiled for
// float; precision.cuh).
//
// The reference's OpenMP variants recompute each intermediate for every point that uses it
// (three laplacians per point in hdiffsa, three T^2 and three S^2 per point in hdiffsmag).
// On GB300 the FP64 pipe, not HBM, bounds these kernels, so here every intermediate is
// computed once per (i, j, k) into a shared-memory tile (plus a one- or two-cell apron) and
// read by its neighbours.  Reusing a value is exact: it is the same expression on the same
// operands.  Differences are stored once and their negations used where the reference
// subtracts in the other order (x - y == -(y - x) exactly in IEEE round-to-nearest).
//
// Compiled with --fmad=false (see k_pointwise.cu).  One CTA of 32 x 8 threads per tile
// and kb k-levels.
#include <mutex>
#include <type_traits>
#include <vector>

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

constexpr int kT = 32;  // tile edge

// Rows of a tile of hdiffsa_kernel and hdiffsmag_kernel.  16 let the registers, six CTAs of eight warps
// an SM, bound the warps in flight, where 32 rows' shared memory (46 and 53 KB in FP64) held them to
// four: FP64 hdiffsa 44.5 -> 38.9 us and hdiffsmag 98.3 -> 86.4 at 128 x 128 x 80, 145 -> 137 and
// 341 -> 324 at 256 x 256 x 80 (24 rows 41.6, 94.9, 133, 325), the tangent-linear hdiffsmag 305 -> 265.
// A grid of less than a wave of those takes 8 rows, whose CTAs are shorter: 13.0 -> 11.0 and
// 27.1 -> 21.3 us at 64 x 64 x 60 (16 rows 11.8 and 23.5), 8.1 -> 4.3 and 15.1 -> 6.9 at
// 33 x 20 x 10; at 128 x 128 x 80 8 rows are slower (44.1 and 89.4).  Recorded launches keep 16 rows,
// the step kernel's form.  Over the host link a tile's apron rows are read again by the next one: there
// hdiffsa keeps 32 rows (in place at 256 x 256 x 80 625 us, 16 rows 655; 64 x 64 x 60 56.5, 8 rows 58.9), and
// both take 8 only with fewer 32-row tiles than SMs (hdiffsa 32 x 32 x 10 25.1 us, 32 rows 33.4).
// The tangent-linear forms keep 16: 8 are shorter on the smallest grids (FP64 hdiffsmag 25.9 -> 15.6 us at
// 32 x 32 x 5) but FP32 is longer from 64 x 64 x 60 on (6.8 -> 7.5 us), and at 100 x 100 x 40 nothing is gained.
constexpr int kJ = 16, kJShort = 8;
inline bool short_tiles(const Dims& d, int kb) {
  if (fields_in_host_memory()) return under_a_wave(tile_grid(d.nx, d.ny, d.nz, kT, kT, kb), 1);
  return !recorder() && under_a_wave(tile_grid(d.nx, d.ny, d.nz, kT, kJ, kb), 6);
}

// ============================== hdiffsa ===========================================
// Shared layout (per k-level), tile origin (i0, j0), J rows:
//   in  : 36 x J+4, (i0-2+a, j0-2+b)
//   dy  : 34 x J+3, (i0-1+a, j0-2+b)   dy(i,j)  = in(i,j+1) - in(i,j);  fly(i,j) then takes its place
//   lap : 34 x J+2, (i0-1+a, j0-1+b)
//   flx : 33 x J,   (i0-1+a, j0+b)
template <class T, int J>
struct HdiffsaSmem {
  T in[J + 4][36];
  T dy[J + 3][34];
  T lap[J + 2][34];
  T flx[J][33];
  T crlato[J + 2];  // j0-1+b
  T crlatu[J + 2];
};

template <class T, int J>
struct hdiffsa_kernel {
  static constexpr bool kAnyGrid = true;
  static __device__ __forceinline__ void run(const uint3& blk, OutPtr<T> out, InPtr<T> in,
                                             InPtr<T> mask, InPtr<T> crlato,
                                             InPtr<T> crlatu, int64_t s1d, Dims d, int kb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HdiffsaSmem<T, J>& s = *reinterpret_cast<HdiffsaSmem<T, J>*>(smem_raw);
    const int i0 = blk.x * kT, j0 = blk.y * J;
    const int sj = (int)d.sj;
    const int tid = threadIdx.y * kTX + threadIdx.x;
    if (tid < J + 2) {
      const int j = j0 - 1 + tid;
      const bool ok = j >= -1 && j < d.ny + 1;
      s.crlato[tid] = ok ? ld(crlato + (int64_t)j * s1d) : T(0);
      s.crlatu[tid] = ok ? ld(crlatu + (int64_t)j * s1d) : T(0);
    }
    const int k0 = blk.z * kb, k1 = min(k0 + kb, d.nz);
    // outputs of this tile (fewer at the domain's far edge) and what each phase needs for them
    const int vx = max(0, min(kT, d.nx - i0)), vy = max(0, min(J, d.ny - j0));
  #pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int64_t kofs = (int64_t)k * d.sk;
      const InPtr<T> pin = in + kofs;
      for_region_lim<36, J + 4>(vx + 4, vy + 4, [&](int a, int b) {
        const int i = i0 - 2 + a, j = j0 - 2 + b;
        const bool ok = i >= -2 && i < d.nx + 2 && j >= -2 && j < d.ny + 2;
        s.in[b][a] = ok ? ld(pin + i + j * sj) : T(0);
      });
      __syncthreads();
      for_region_lim<34, J + 3>(vx + 2, vy + 3, [&](int a, int b) { s.dy[b][a] = isub(s.in[b + 1][a + 1], s.in[b][a + 1]); });
      __syncthreads();
      // hdiffsa.h:101: in(i-1)+in(i+1) - 2 in + crlato (in(j+1)-in) + crlatu (in(j-1)-in)
      for_region_lim<34, J + 2>(vx + 2, vy + 2, [&](int a, int b) {
        const T c = s.in[b + 1][a + 1];
        s.lap[b][a] = ((iadd(s.in[b + 1][a], s.in[b + 1][a + 2]) - scale2<1>(c)) + s.crlato[b] * s.dy[b + 1][a]) +
                      s.crlatu[b] * (-s.dy[b][a]);
      });
      __syncthreads();
      // hdiffsa.h:106-113: limited fluxes
      for_region_lim<33, J>(vx + 1, vy, [&](int a, int b) {
        T f = s.lap[b + 1][a + 1] - s.lap[b + 1][a];
        if (Prec<T>::prod_gt0(f, s.in[b + 2][a + 2] - s.in[b + 2][a + 1])) f = T(0);
        s.flx[b][a] = f;
      });
      for_region_lim<32, J + 1>(vx, vy + 1, [&](int a, int b) {  // fly(i0+a, j0-1+b)
        T f = s.crlato[b] * (s.lap[b + 1][a + 1] - s.lap[b][a + 1]);
        T& g = s.dy[b + 1][a + 1];  // read by this cell alone
        if (Prec<T>::prod_gt0(f, g)) f = T(0);
        g = f;
      });
      __syncthreads();
      // hdiffsa.h:118-119
      for_region_lim<32, J>(vx, vy, [&](int a, int b) {
        const int64_t o = kofs + (i0 + a) + (j0 + b) * sj;
        out[o] = s.in[b + 2][a + 2] +
                 (((s.flx[b][a] - s.flx[b][a + 1]) + s.dy[b + 1][a + 1]) - s.dy[b + 2][a + 1]) * ld(mask + o);
      });
      __syncthreads();
    }
  }
};

// FP32 hdiffsa, marching rows (march.cuh): lane = column i0 - 1 + lane, 30 columns a strip.  At row j
// a lane holds `in` on rows j .. j+2 (its x neighbours, loaded with each row, on j and j+1) and forms
// the laplacian at j+1 and from it fly at j; flx at j takes the laplacian of the lane above, the
// output the flx of the lane below.  Each laplacian and flux is formed once.  hdiffsa_kernel<float>'s
// operations on the same operands (the limiter tests on the exact product, its factors scaled by
// 2^100, so that a nonzero product neither underflows nor loses its sign): the same bits.
//
// What bounds it: instruction issue (about 98 instructions a row of 30 columns, 69 % of the issue
// slots taken) and the ends of a short launch.  48 registers, five CTAs an SM, two rows unrolled:
// 23.4 us at 256 x 256 x 80 and 50.3 at 320 x 304 x 137 (four CTAs 24.1 / 50.6, six 28.1 / 61.7,
// one row unrolled 26.5 / 58.9; two rows of loads in flight instead of one 26.4 / 59.0); the form
// before it, a 32 x 32 shared-memory tile marched over the levels, took 37.4 and 94.7 us.
struct hdiffsa_march_f32 {
  static constexpr bool kAnyGrid = true;
  static constexpr int kCols = 30, kApron = 3, kMinCtas = 5;
  static __device__ __forceinline__ float limited(float f, float d) {
    constexpr float s = 1.2676506002282294e30f;
    return (f * s) * (d * s) > 0.f ? 0.f : f;
  }
  static __device__ __forceinline__ void run(const uint3& blk, float* __restrict__ out, const float* __restrict__ in,
                                             const float* __restrict__ mask, const float* __restrict__ crlato,
                                             const float* __restrict__ crlatu, int64_t s1d, Dims d, int rows,
                                             int wx_log) {
    const MarchPos pos = march_pos(blk, wx_log);
    const int nx = d.nx, ny = d.ny;
    const int i0 = pos.strip * kCols, ja = pos.chunk * rows, jb = min(ja + rows, ny);
    if (i0 >= nx || ja >= ny) return;
    const int lane = (int)threadIdx.x, i = min(i0 - 1 + lane, nx);  // lanes past the reach repeat its last column
    const bool st = lane >= 1 && lane <= kCols && i0 - 1 + lane < nx;
    const int64_t sjb = d.sj * 4;
    int64_t o = ((int64_t)blk.z * d.sk + (int64_t)ja * d.sj + i) * 4;  // (i, j)
    const int64_t om = (int64_t)(max(0, min(i, nx - 1)) - i) * 4;      // to the mask's column
    // the metric terms of rows ja - 1 + lane
    float lo, lu;
    auto metric = [&](int j) {
      const int64_t jo = (int64_t)min(j + lane, ny) * s1d;
      lo = ld(crlato + jo), lu = ld(crlatu + jo);
    };
    metric(ja - 1);
    auto lapl = [](float m, float c, float p, float co, float dyp, float cu, float dym) {
      return (((m + p) - 2.f * c) + co * dyp) + cu * (-dym);
    };
    // rows ja - 2 .. ja + 1: the laplacian at ja - 1 and ja, and fly at ja - 1
    const float a0 = get(in, o - 2 * sjb), a1 = get(in, o - sjb);
    float c0 = get(in, o), c1 = get(in, o + sjb);
    const float a1m = get(in, o - sjb - 4), a1p = get(in, o - sjb + 4), c0m = get(in, o - 4), c0p = get(in, o + 4);
    float c1m = get(in, o + sjb - 4), c1p = get(in, o + sjb + 4);
    // `in` on row j + 2 and the mask on j, loaded a row ahead
    float n = get(in, o + 2 * sjb), nm = get(in, o + 2 * sjb - 4), np = get(in, o + 2 * sjb + 4), w = get(mask, o + om);
    float cm = __shfl_sync(kWarpMask, lo, 0), co = __shfl_sync(kWarpMask, lo, 1);
    const float dm = c0 - a1;
    float dy = c1 - c0, dx = c0p - c0;
    const float lm = lapl(a1m, a1, a1p, cm, dm, __shfl_sync(kWarpMask, lu, 0), a1 - a0);
    float lap = lapl(c0m, c0, c0p, co, dy, __shfl_sync(kWarpMask, lu, 1), dm);
    float fly = limited(cm * (lap - lm), dm);  // at ja - 1
#pragma unroll 2
    for (int j = ja; j < jb; ++j) {
      const float x = n, xm = nm, xp = np, wj = w;
      if (j + 1 < jb) {
        n = get(in, o + 3 * sjb), nm = get(in, o + 3 * sjb - 4), np = get(in, o + 3 * sjb + 4);
        w = get(mask, o + om + sjb);
      }
      const int src = (j + 2 - ja) & 31;
      if (src == 0) metric(j + 1);
      const float cn = __shfl_sync(kWarpMask, lo, src), un = __shfl_sync(kWarpMask, lu, src);  // at j + 1
      const float dn = x - c1;
      const float ln = lapl(c1m, c1, c1p, cn, dn, un, dy);
      const float fn = limited(co * (ln - lap), dy);
      const float fx = limited(lane_above<1>(lap) - lap, dx);
      const float r = c0 + (((lane_below<1>(fx) - fx) + fly) - fn) * wj;
      if (st) put(out, o, r);
      dx = c1p - c1, c0 = c1, c1 = x, c1m = xm, c1p = xp;
      dy = dn, lap = ln, fly = fn, co = cn;
      o += sjb;
    }
  }
};

// ============================== hdiffsmag =========================================
// Shared layout (per k-level), tile origin (i0, j0), J rows:
//   u, v : 34 x J+2, (i0-1+a, j0-1+b)
//   dyv  : 33 x J+1, (i0+a,   j0-1+b)   v(i,j+1) - v(i,j)
//   dyu  : 33 x J+1, (i0-1+a, j0-1+b)   u(i,j+1) - u(i,j)
// (the x differences dxu = u(i+1,j) - u(i,j) at (i0-1+a, j0+b) and dxv = v(i+1,j) - v(i,j)
// at (i0-1+a, j0-1+b) are each read once, by the deformations of the same cell: they live in
// registers, which keeps a tile of 16 rows at 28 KB)
//   tsq  : 33 x J+1, (i0+a,   j0+b)     T_s^2
//   ssq  : 33 x J+1, (i0-1+a, j0-1+b)   S_uv^2
template <class T, int J>
struct HdiffsmagSmem {
  T u[J + 2][34];
  T v[J + 2][34];
  T dyv[J + 1][33];
  T dyu[J + 1][33];
  T tsq[J + 1][33];
  T ssq[J + 1][33];
  T acrlat0[J + 2];  // j0-1+b
  T crlato[J], crlatu[J], crlavo[J], crlavu[J];
};

template <class T, int J>
struct hdiffsmag_kernel {
  static constexpr bool kAnyGrid = true;
  static constexpr int kStepOp = step_op<T>(J == kJ ? kOpSmagFwd : -1);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, OutPtr<T> uout, OutPtr<T> vout,
                                             InPtr<T> uin, InPtr<T> vin,
                                             InPtr<T> mask, InPtr<T> crlavo,
                                             InPtr<T> crlavu, InPtr<T> crlato,
                                             InPtr<T> crlatu, InPtr<T> acrlat0, int64_t s1d,
                                             T eddlat, T eddlon, T tau_smag, T weight_smag, Dims d, int kb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HdiffsmagSmem<T, J>& s = *reinterpret_cast<HdiffsmagSmem<T, J>*>(smem_raw);
    const int i0 = blk.x * kT, j0 = blk.y * J;
    const int sj = (int)d.sj;
    const int tid = threadIdx.y * kTX + threadIdx.x;
    constexpr T rr = earth_radius_recip<T>();
    if (tid < J + 2) {
      const int j = j0 - 1 + tid;
      s.acrlat0[tid] = (j >= -1 && j < d.ny + 1) ? ld(acrlat0 + (int64_t)j * s1d) : T(0);
    } else if (tid >= 64 && tid < 64 + J) {
      const int b = tid - 64, j = j0 + b;
      const bool ok = j < d.ny;
      const int64_t jo = (int64_t)j * s1d;
      s.crlato[b] = ok ? ld(crlato + jo) : T(0);
      s.crlatu[b] = ok ? ld(crlatu + jo) : T(0);
      s.crlavo[b] = ok ? ld(crlavo + jo) : T(0);
      s.crlavu[b] = ok ? ld(crlavu + jo) : T(0);
    }
    const int k0 = blk.z * kb, k1 = min(k0 + kb, d.nz);
    // outputs of this tile (fewer at the domain's far edge) and what each phase needs for them
    const int vx = max(0, min(kT, d.nx - i0)), vy = max(0, min(J, d.ny - j0));
  #pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int64_t kofs = (int64_t)k * d.sk;
      for_region_lim<34, J + 2>(vx + 2, vy + 2, [&](int a, int b) {
        const int i = i0 - 1 + a, j = j0 - 1 + b;
        const bool ok = i >= -1 && i < d.nx + 1 && j >= -1 && j < d.ny + 1;
        const int64_t o = kofs + i + j * sj;
        s.u[b][a] = ok ? ld(uin + o) : T(0);
        s.v[b][a] = ok ? ld(vin + o) : T(0);
      });
      __syncthreads();
      // hdiffsmag.h:213 T_s = (v(j-1)-v) eddlat R^-1 - (u(i-1)-u) acrlat0(j) eddlon
      //              :221 S_uv = (u(j+1)-u) eddlat R^-1 + (v(i+1)-v) acrlat0(j) eddlon
      for_region_lim<33, J + 1>(vx + 1, vy + 1, [&](int a, int b) {
        const T dxu = s.u[b + 1][a + 1] - s.u[b + 1][a];
        const T dyv = s.v[b + 1][a + 1] - s.v[b][a + 1];
        const T dyu = s.u[b + 1][a] - s.u[b][a];
        const T dxv = s.v[b][a + 1] - s.v[b][a];
        s.dyv[b][a] = dyv;
        s.dyu[b][a] = dyu;
        const T ts = ((-dyv) * eddlat) * rr - ((-dxu) * s.acrlat0[b + 1]) * eddlon;
        s.tsq[b][a] = ts * ts;
        const T su = (dyu * eddlat) * rr + (dxv * s.acrlat0[b]) * eddlon;
        s.ssq[b][a] = su * su;
      });
      __syncthreads();
      for_region_lim<32, J>(vx, vy, [&](int a, int b) {
        const int i = i0 + a, j = j0 + b;
        const int64_t o = kofs + i + j * sj;
        const T hdweight = weight_smag * ld(mask + o);
        // hdiffsmag.h:233-244 (the T^2 pair sums as integer-pipe additions: the FP64 pipe is the
        // busier one here; two per point measured best, four 6 % slower)
        T smag_u = tau_smag * Prec<T>::sqrt_(scale2<-1>(iadd(s.tsq[b][a + 1], s.tsq[b][a])) +
                                             scale2<-1>(s.ssq[b][a + 1] + s.ssq[b + 1][a + 1])) -
                   hdweight;
        smag_u = clamp_smag(smag_u);
        const T uc = s.u[b + 1][a + 1];
        // u(i+1) + u(i-1) - 2u + crlato (u(j+1) - u) + crlatu (u(j-1) - u), the reference's
        // sum in every precision: FP32 is then bit-identical to the reference compiled for
        // float.  A compensated FP32 sum (TwoSum / TwoProduct) measured the same largest error
        // against the FP64 oracle (5.5e-8) at about five times the sum's operations.
        Acc<T> lu(s.u[b + 1][a + 2]);
        lu.add(s.u[b + 1][a]);
        lu.add(-scale2<1>(uc));
        lu.add_prod(s.crlato[b], s.dyu[b + 1][a + 1]);
        lu.add_prod(s.crlatu[b], -s.dyu[b][a + 1]);
        uout[o] = uc + mul_zero(smag_u, lu.get());  // the clamp gives many zeros
        // hdiffsmag.h:248-259
        T smag_v = tau_smag * Prec<T>::sqrt_(scale2<-1>(iadd(s.tsq[b + 1][a], s.tsq[b][a])) +
                                             scale2<-1>(s.ssq[b + 1][a] + s.ssq[b + 1][a + 1])) -
                   hdweight;
        smag_v = clamp_smag(smag_v);
        const T vc = s.v[b + 1][a + 1];
        Acc<T> lv(s.v[b + 1][a + 2]);
        lv.add(s.v[b + 1][a]);
        lv.add(-scale2<1>(vc));
        lv.add_prod(s.crlavo[b], s.dyv[b + 1][a]);
        lv.add_prod(s.crlavu[b], -s.dyv[b][a]);
        vout[o] = vc + mul_zero(smag_v, lv.get());
      });
      __syncthreads();
    }
  }
};

// FP32 hdiffsmag, marching rows (march.cuh): lane = column i0 - 1 + lane, 30 columns a strip.  At row j
// a lane holds u and v on rows j and j+1 (their x neighbours handed over by the neighbouring lanes as
// each row arrives) and forms T^2 at j+1 and S^2 at j, each once; T^2(i+1) and S^2(i-1) come from the
// lanes beside it.  hdiffsmag_kernel's operations on the same operands in the same order.
//
// What bounds it: instruction issue (about 165 instructions a row, two square roots among them; 72 %) and
// load latency.  48 registers, five CTAs an SM: 39.1 us at 256 x 256 x 80, 89.0 at 320 x 304 x 137
// and 19.7 at 201 x 173 x 61 (four CTAs 47.6 / 107 / 23.3, six, which spills, 43.7 / 102 / 19.5);
// hdiffsmag_kernel<float>'s shared-memory tile took 44.2, 103.8 and 24.2 us.
struct hdiffsmag_march_f32 {
  static constexpr bool kAnyGrid = true;
  static constexpr int kStepOp = step_op<float>(kOpSmagFwd);  // the step kernel's id
  static constexpr int kCols = 30, kApron = 2, kMinCtas = 5;
  static __device__ __forceinline__ void run(const uint3& blk, float* __restrict__ uout, float* __restrict__ vout,
                                             const float* __restrict__ uin, const float* __restrict__ vin,
                                             const float* __restrict__ mask, const float* __restrict__ crlavo,
                                             const float* __restrict__ crlavu, const float* __restrict__ crlato,
                                             const float* __restrict__ crlatu, const float* __restrict__ acrlat0,
                                             int64_t s1d, float eddlat, float eddlon, float tau_smag,
                                             float weight_smag, Dims d, int rows, int wx_log) {
    const MarchPos pos = march_pos(blk, wx_log);
    const int nx = d.nx, ny = d.ny;
    const int i0 = pos.strip * kCols, ja = pos.chunk * rows, jb = min(ja + rows, ny);
    if (i0 >= nx || ja >= ny) return;
    constexpr float rr = earth_radius_recip<float>();
    const int lane = (int)threadIdx.x, i = min(i0 - 1 + lane, nx);  // lanes past the reach repeat its last column
    const bool st = lane >= 1 && lane <= kCols && i0 - 1 + lane < nx;
    const int64_t sjb = d.sj * 4;
    int64_t o = ((int64_t)blk.z * d.sk + (int64_t)ja * d.sj + i) * 4;  // (i, j)
    const int64_t om = (int64_t)(max(0, min(i, nx - 1)) - i) * 4;      // to the mask's column
    // the metric terms of 32 rows, one a lane: acrlat0 from row ja - 1, the others from ja
    float la, lto, ltu, lvo, lvu;
    auto metric_a = [&](int j) { la = ld(acrlat0 + (int64_t)min(j + lane, ny) * s1d); };
    auto metric = [&](int j) {
      const int64_t jo = (int64_t)min(j + lane, ny - 1) * s1d;
      lto = ld(crlato + jo), ltu = ld(crlatu + jo), lvo = ld(crlavo + jo), lvu = ld(crlavu + jo);
    };
    metric_a(ja - 1);
    metric(ja);
    // T from dyv(j-1) and dxu(j), S from dyu(j) and dxv(j)
    auto tsq_of = [&](float dyv, float dxu, float ac) {
      const float t = ((-dyv) * eddlat) * rr - ((-dxu) * ac) * eddlon;
      return t * t;
    };
    auto ssq_of = [&](float dyu, float dxv, float ac) {
      const float q = (dyu * eddlat) * rr + (dxv * ac) * eddlon;
      return q * q;
    };
    const float ua = get(uin, o - sjb), va = get(vin, o - sjb);
    float u0 = get(uin, o), v0 = get(vin, o);
    // u and v on row j + 1 and the mask on j, loaded a row ahead
    float un = get(uin, o + sjb), vn = get(vin, o + sjb), w = get(mask, o + om);
    const float am = __shfl_sync(kWarpMask, la, 0);
    float ac = __shfl_sync(kWarpMask, la, 1);
    float dyu = u0 - ua, dyv = v0 - va;                                    // at j - 1
    float um = lane_below<1>(u0), up = lane_above<1>(u0), vm = lane_below<1>(v0), vp = lane_above<1>(v0);  // on row j
    float tsq = tsq_of(dyv, u0 - um, ac);                                  // at j
    float ssq = ssq_of(dyu, lane_above<1>(va) - va, am);                   // at j - 1
#pragma unroll 1
    for (int j = ja; j < jb; ++j) {
      const float u1 = un, v1 = vn, wj = w;
      if (j + 1 < jb) un = get(uin, o + 2 * sjb), vn = get(vin, o + 2 * sjb), w = get(mask, o + om + sjb);
      const int src = (j - ja) & 31, sra = (j + 2 - ja) & 31;
      if (src == 0 && j > ja) metric(j);
      if (sra == 0) metric_a(j + 1);
      const float an = __shfl_sync(kWarpMask, la, sra);
      const float cto = __shfl_sync(kWarpMask, lto, src), ctu = __shfl_sync(kWarpMask, ltu, src),
                  cvo = __shfl_sync(kWarpMask, lvo, src), cvu = __shfl_sync(kWarpMask, lvu, src);
      const float um1 = lane_below<1>(u1), up1 = lane_above<1>(u1), vm1 = lane_below<1>(v1), vp1 = lane_above<1>(v1);
      const float dyu1 = u1 - u0, dyv1 = v1 - v0;
      const float tsq1 = tsq_of(dyv1, u1 - um1, an);
      const float ssq1 = ssq_of(dyu1, vp - v0, ac);
      const float hdweight = weight_smag * wj;
      // hdiffsmag.h:233-244
      const float su = clamp_smag(
          tau_smag * sqrtf(0.5f * (lane_above<1>(tsq) + tsq) + 0.5f * (ssq + ssq1)) - hdweight);
      const float lu = (((up + um) + -(2.f * u0)) + cto * dyu1) + ctu * (-dyu);
      // hdiffsmag.h:248-259
      const float sv = clamp_smag(
          tau_smag * sqrtf(0.5f * (tsq1 + tsq) + 0.5f * (lane_below<1>(ssq1) + ssq1)) - hdweight);
      const float lv = (((vp + vm) + -(2.f * v0)) + cvo * dyv1) + cvu * (-dyv);
      if (st) {
        put(uout, o, u0 + su * lu);
        put(vout, o, v0 + sv * lv);
      }
      u0 = u1, v0 = v1, um = um1, up = up1, vm = vm1, vp = vp1;
      dyu = dyu1, dyv = dyv1, tsq = tsq1, ssq = ssq1, ac = an;
      o += sjb;
    }
  }
};

constexpr int kKB = 1;  // k-levels per CTA by default (the most CTAs hide latency best)

template <class T, class M3, class M1>
oeb_status hdiffsa_entry(const M3* out, const M3* in, const M3* mask, const M1* crlato, const M1* crlatu,
                         const oeb_domain* dom, void* stream) {
  OEB_TRY(check_domain(dom));
  Grid<T> gout, gin, gmask;
  Line<T> lo, lu;
  OEB_TRY((check_field3<T>(out, *dom, kInterior, &gout)));
  OEB_TRY((check_field3<T>(in, *dom, Reach{2, 2, 2, 2, 0, 0}, &gin)));
  OEB_TRY((check_field3<T>(mask, *dom, kInterior, &gmask)));
  OEB_TRY((check_field1<T>(crlato, *dom, 1, 1, &lo)));
  OEB_TRY((check_field1<T>(crlatu, *dom, 1, 1, &lu)));
  if (lo.s != lu.s) return OEB_ERR_LAYOUT;
  OEB_TRY(check_same_strides<T>({&gout, &gin, &gmask}));
  OEB_TRY(check_no_alias({gout.lo, gout.hi}, {gin.lo, gin.hi, gmask.lo, gmask.hi, lo.lo, lo.hi, lu.lo, lu.hi}));
  OEB_RETURN_IF_VALIDATING();
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gin.sj, gin.sk};
  if constexpr (std::is_same<T, float>::value) {
    using B = hdiffsa_march_f32;
    const MarchShape m = march_shape(d.nx, d.ny, d.nz, 1, B::kCols, B::kApron, B::kMinCtas);
    return launch<B>(m.grid, 0, (cudaStream_t)stream, gout.origin, gin.origin, gmask.origin, lo.origin, lu.origin, lo.s,
                     d, m.rows, m.wx_log);
  } else {
    const int kb = tuned_kb(kKB);
    auto run = [&](auto rows) {
      constexpr int J = decltype(rows)::value;
      return launch<hdiffsa_kernel<T, J>>(tile_grid(d.nx, d.ny, d.nz, kT, J, kb), sizeof(HdiffsaSmem<T, J>),
                                          (cudaStream_t)stream, gout.origin, gin.origin, gmask.origin, lo.origin,
                                          lu.origin, lo.s, d, kb);
    };
    if (short_tiles(d, kb)) return run(std::integral_constant<int, kJShort>());
    if (fields_in_host_memory()) return run(std::integral_constant<int, kT>());
    return run(std::integral_constant<int, kJ>());
  }
}

template <class T, class M3, class M1>
oeb_status hdiffsmag_entry(const M3* uout, const M3* vout, const M3* uin, const M3* vin, const M3* mask,
                           const M1* crlavo, const M1* crlavu, const M1* crlato, const M1* crlatu, const M1* acrlat0,
                           T eddlat, T eddlon, T tau_smag, T weight_smag, const oeb_domain* dom, void* stream) {
  OEB_TRY(check_domain(dom));
  Grid<T> gu, gv, gui, gvi, gm;
  Line<T> lvo, lvu, lto, ltu, la0;
  OEB_TRY((check_field3<T>(uout, *dom, kInterior, &gu)));
  OEB_TRY((check_field3<T>(vout, *dom, kInterior, &gv)));
  OEB_TRY((check_field3<T>(uin, *dom, Reach{1, 1, 1, 1, 0, 0}, &gui)));
  OEB_TRY((check_field3<T>(vin, *dom, Reach{1, 1, 1, 1, 0, 0}, &gvi)));
  OEB_TRY((check_field3<T>(mask, *dom, kInterior, &gm)));
  OEB_TRY((check_field1<T>(crlavo, *dom, 0, 0, &lvo)));
  OEB_TRY((check_field1<T>(crlavu, *dom, 0, 0, &lvu)));
  OEB_TRY((check_field1<T>(crlato, *dom, 0, 0, &lto)));
  OEB_TRY((check_field1<T>(crlatu, *dom, 0, 0, &ltu)));
  OEB_TRY((check_field1<T>(acrlat0, *dom, 1, 1, &la0)));
  if (lvu.s != lvo.s || lto.s != lvo.s || ltu.s != lvo.s || la0.s != lvo.s) return OEB_ERR_LAYOUT;
  OEB_TRY(check_same_strides<T>({&gu, &gv, &gui, &gvi, &gm}));
  OEB_TRY(check_no_alias({gu.lo, gu.hi, gv.lo, gv.hi},
                         {gui.lo, gui.hi, gvi.lo, gvi.hi, gm.lo, gm.hi, lvo.lo, lvo.hi, lvu.lo, lvu.hi, lto.lo,
                          lto.hi, ltu.lo, ltu.hi, la0.lo, la0.hi}));
  OEB_RETURN_IF_VALIDATING();
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gui.sj, gui.sk};
  if constexpr (std::is_same<T, float>::value) {
    using B = hdiffsmag_march_f32;
    const MarchShape m = march_shape(d.nx, d.ny, d.nz, 1, B::kCols, B::kApron, B::kMinCtas);
    return launch<B>(m.grid, 0, (cudaStream_t)stream, gu.origin, gv.origin, gui.origin, gvi.origin, gm.origin, lvo.origin,
                     lvu.origin, lto.origin, ltu.origin, la0.origin, lvo.s, eddlat, eddlon, tau_smag, weight_smag, d,
                     m.rows, m.wx_log);
  } else {
    const int kb = tuned_kb(kKB);
    auto run = [&](auto tile_rows) {
      constexpr int J = decltype(tile_rows)::value;
      return launch<hdiffsmag_kernel<T, J>>(
          tile_grid(d.nx, d.ny, d.nz, kT, J, kb), sizeof(HdiffsmagSmem<T, J>), (cudaStream_t)stream, gu.origin, gv.origin,
          gui.origin, gvi.origin, gm.origin, lvo.origin, lvu.origin, lto.origin, ltu.origin, la0.origin, lvo.s, eddlat,
          eddlon, tau_smag, weight_smag, d, kb);
    };
    return short_tiles(d, kb) ? run(std::integral_constant<int, kJShort>()) : run(std::integral_constant<int, kJ>());
  }
}

// Tangent-linear hdiffsmag: d(uout, vout) = J(uin, vin) d(uin, vin), the kernel on Dual<T>.
template <class T, class M3, class M1>
oeb_status hdiffsmag_tl_entry(const M3* duout, const M3* dvout, const M3* uin, const M3* vin, const M3* mask,
                              const M1* crlavo, const M1* crlavu, const M1* crlato, const M1* crlatu,
                              const M1* acrlat0, const M3* duin, const M3* dvin, T eddlat, T eddlon, T tau_smag,
                              T weight_smag, const oeb_domain* dom, void* stream) {
  {
    ValidateOnly guard;
    OEB_TRY(hdiffsmag_entry<T>(duout, dvout, uin, vin, mask, crlavo, crlavu, crlato, crlatu, acrlat0, eddlat, eddlon,
                               tau_smag, weight_smag, dom, stream));
    OEB_TRY(hdiffsmag_entry<T>(duout, dvout, duin, dvin, mask, crlavo, crlavu, crlato, crlatu, acrlat0, eddlat,
                               eddlon, tau_smag, weight_smag, dom, stream));
  }
  OEB_RETURN_IF_VALIDATING();
  using D = Dual<T>;
  DualIn<T> u, v;
  OEB_TRY((dual_in<T>(uin, duin, &u)));
  OEB_TRY((dual_in<T>(vin, dvin, &v)));
  const DualIn<T> m = dual_param<T>(mask), l0 = dual_param<T>(crlavo), l1 = dual_param<T>(crlavu),
                  l2 = dual_param<T>(crlato), l3 = dual_param<T>(crlatu), l4 = dual_param<T>(acrlat0);
  const DualOut<T> ou = dual_out<T>(duout), ov = dual_out<T>(dvout);
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, uin->strides[1], uin->strides[0]};
  const int kb = tuned_kb(kKB);
  return launch<hdiffsmag_kernel<D, kJ>>(tile_grid(d.nx, d.ny, d.nz, kT, kJ, kb), sizeof(HdiffsmagSmem<D, kJ>),
                                      (cudaStream_t)stream, ou, ov, u, v, m, l0, l1, l2, l3, l4, crlavo->strides[0],
                                      D(eddlat), D(eddlon), D(tau_smag), D(weight_smag), d, kb);
}

// ============================== hdiffsa: tangent-linear and adjoint ===============
// Linearised at `in` with the flux limiters of hdiffsa.h:106-113 frozen:
//   out = in + mask (flx(i-1) - flx + fly(j-1) - fly),
//   flx = fx (lap(i+1) - lap),  fly = fy crlato(j) (lap(j+1) - lap),
//   fx = 0 where flx (in(i+1) - in) > 0 at the state, else 1 (fy likewise with j),
//   lap = in(i-1) + in(i+1) - 2 in + crlato(j) (in(j+1) - in) + crlatu(j) (in(j-1) - in).
// Active input: in (mask, crlato, crlatu are parameters).  The transpose for outb, with
// G = mask outb on the interior and 0 elsewhere:
//   Fx = fx (G(i+1) - G) on [-1,N) x [0,N),  Fy = fy crlato(j) (G(j+1) - G) on [0,N) x [-1,N),
//   lapb = Fx(i-1) - Fx + Fy(j-1) - Fy,
//   inb = outb (interior) + lapb(i-1) + lapb(i+1) - (2 + crlato(j) + crlatu(j)) lapb
//         + crlato(j-1) lapb(j-1) + crlatu(j+1) lapb(j+1)    on in's reach box [-2, N+2)^2.
// One kernel: a CTA stages its tile's in and G in shared memory, recomputes lap and the limiter
// flags exactly as the forward kernel does (the same operations on the same operands), then
// forms Fx, Fy, lapb and inb in shared memory.  Shared layout (per k-level), inb tile origin
// (i0, j0), J rows:
//   in   : 38 x J+6, (i0-3+a, j0-3+b)
//   lap  : 36 x J+4, (i0-2+a, j0-2+b)
//   gl   : 36 x J+4, G at (i0-2+a, j0-2+b); then lapb, 34 x J+2 at (i0-1+a, j0-1+b)
//   fx   : 35 x J+2, (i0-2+a, j0-1+b);   fy : 34 x J+3, (i0-1+a, j0-2+b)
// A tile at the box's far edge forms only what its own columns and rows need.
template <class T, int J>
struct HdiffsaAdjSmem {
  T in[J + 6][38];
  T lap[J + 4][36];
  T gl[J + 4][36];
  T fx[J + 2][35];
  T fy[J + 3][34];
  T crlato[J + 6], crlatu[J + 6];  // j0-3+b
};

template <class T, int J>
struct hdiffsa_adj_kernel {
  static constexpr bool kAnyGrid = true;
  static __device__ __forceinline__ void run(const uint3& blk, T* __restrict__ inb, const T* __restrict__ in,
                                             const T* __restrict__ mask, const T* __restrict__ crlato,
                                             const T* __restrict__ crlatu, int64_t s1d, const T* __restrict__ outb,
                                             Dims d, int kb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    HdiffsaAdjSmem<T, J>& s = *reinterpret_cast<HdiffsaAdjSmem<T, J>*>(smem_raw);
    T(*lapb)[34] = reinterpret_cast<T(*)[34]>(&s.gl[0][0]);
    const int i0 = -2 + (int)blk.x * kT, j0 = -2 + (int)blk.y * J;
    const int64_t sj = d.sj;
    const int tid = threadIdx.y * kTX + threadIdx.x;
    if (tid < J + 6) {
      const int j = j0 - 3 + tid;
      const bool ok = j >= -1 && j < d.ny + 1;
      s.crlato[tid] = ok ? ld(crlato + (int64_t)j * s1d) : T(0);
      s.crlatu[tid] = ok ? ld(crlatu + (int64_t)j * s1d) : T(0);
    }
    auto interior = [&](int i, int j) { return i >= 0 && i < d.nx && j >= 0 && j < d.ny; };
    const int vx = min(kT, d.nx + 2 - i0), vy = min(J, d.ny + 2 - j0);
    const int k0 = blk.z * kb, k1 = min(k0 + kb, d.nz);
  #pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int64_t kofs = (int64_t)k * d.sk;
      for_region_lim<38, J + 6>(vx + 6, vy + 6, [&](int a, int b) {
        const int i = i0 - 3 + a, j = j0 - 3 + b;
        const bool ok = i >= -2 && i < d.nx + 2 && j >= -2 && j < d.ny + 2;
        s.in[b][a] = ok ? ld(in + kofs + i + j * sj) : T(0);
      });
      for_region_lim<36, J + 4>(vx + 4, vy + 4, [&](int a, int b) {
        const int i = i0 - 2 + a, j = j0 - 2 + b;
        const int64_t o = kofs + i + j * sj;
        s.gl[b][a] = interior(i, j) ? ld(outb + o) * ld(mask + o) : T(0);
      });
      __syncthreads();
      // hdiffsa.h:101 where the forward forms lap (i, j in [-1, N+1)), its operations in its order
      for_region_lim<36, J + 4>(vx + 4, vy + 4, [&](int a, int b) {
        const int i = i0 - 2 + a, j = j0 - 2 + b;
        T v = T(0);
        if (i >= -1 && i < d.nx + 1 && j >= -1 && j < d.ny + 1) {
          const T c = s.in[b + 1][a + 1];
          v = (((s.in[b + 1][a] + s.in[b + 1][a + 2]) - scale2<1>(c)) + s.crlato[b + 1] * (s.in[b + 2][a + 1] - c)) +
              s.crlatu[b + 1] * (s.in[b][a + 1] - c);
        }
        s.lap[b][a] = v;
      });
      __syncthreads();
      // hdiffsa.h:106-109: Fx at (i, j), kept where the forward keeps flx
      for_region_lim<35, J + 2>(vx + 3, vy + 2, [&](int a, int b) {
        const int i = i0 - 2 + a, j = j0 - 1 + b;
        T v = T(0);
        if (i >= -1 && i < d.nx && j >= 0 && j < d.ny) {
          const T f = s.lap[b + 1][a + 1] - s.lap[b + 1][a];
          if (!Prec<T>::prod_gt0(f, s.in[b + 2][a + 2] - s.in[b + 2][a + 1])) v = s.gl[b + 1][a + 1] - s.gl[b + 1][a];
        }
        s.fx[b][a] = v;
      });
      // hdiffsa.h:110-113: Fy at (i, j), crlato(j) folded in
      for_region_lim<34, J + 3>(vx + 2, vy + 3, [&](int a, int b) {
        const int i = i0 - 1 + a, j = j0 - 2 + b;
        T v = T(0);
        if (i >= 0 && i < d.nx && j >= -1 && j < d.ny) {
          const T co = s.crlato[b + 1];
          const T f = co * (s.lap[b + 1][a + 1] - s.lap[b][a + 1]);
          if (!Prec<T>::prod_gt0(f, s.in[b + 2][a + 2] - s.in[b + 1][a + 2])) v = co * (s.gl[b + 1][a + 1] - s.gl[b][a + 1]);
        }
        s.fy[b][a] = v;
      });
      __syncthreads();
      // lapb over the dead G
      for_region_lim<34, J + 2>(vx + 2, vy + 2, [&](int a, int b) { lapb[b][a] = (s.fx[b][a] - s.fx[b][a + 1]) + (s.fy[b][a] - s.fy[b + 1][a]); });
      __syncthreads();
      for_region_lim<32, J>(vx, vy, [&](int a, int b) {
        const int i = i0 + a, j = j0 + b;
        const int64_t o = kofs + i + j * sj;
        const T c = lapb[b + 1][a + 1];
        T v = (lapb[b + 1][a] + lapb[b + 1][a + 2]) - mul_zero(c, (T(2) + s.crlato[b + 3]) + s.crlatu[b + 3]);
        v = fma(s.crlato[b + 2], lapb[b][a + 1], v);
        v = fma(s.crlatu[b + 4], lapb[b + 2][a + 1], v);
        if (interior(i, j)) v = v + ld(outb + o);
        inb[o] = v;
      });
      __syncthreads();
    }
  }
};

template <class T, class M3, class M1>
oeb_status hdiffsa_tl_entry(const M3* dout, const M3* in, const M3* mask, const M1* crlato, const M1* crlatu,
                            const M3* din, const oeb_domain* dom, void* stream) {
  {
    ValidateOnly guard;
    OEB_TRY(hdiffsa_entry<T>(dout, in, mask, crlato, crlatu, dom, stream));
    OEB_TRY(hdiffsa_entry<T>(dout, din, mask, crlato, crlatu, dom, stream));
  }
  OEB_RETURN_IF_VALIDATING();
  using D = Dual<T>;
  DualIn<T> x;
  OEB_TRY((dual_in<T>(in, din, &x)));
  const DualIn<T> m = dual_param<T>(mask), lo = dual_param<T>(crlato), lu = dual_param<T>(crlatu);
  const DualOut<T> y = dual_out<T>(dout);
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, in->strides[1], in->strides[0]};
  const int kb = tuned_kb(kKB);
  return launch<hdiffsa_kernel<D, kJ>>(tile_grid(d.nx, d.ny, d.nz, kT, kJ, kb), sizeof(HdiffsaSmem<D, kJ>),
                                      (cudaStream_t)stream, y, x, m, lo, lu, crlato->strides[0], d, kb);
}

template <class T, class M3, class M1>
oeb_status hdiffsa_adj_entry(const M3* inb, const M3* in, const M3* mask, const M1* crlato, const M1* crlatu,
                             const M3* outb, const oeb_domain* dom, void* stream) {
  {
    ValidateOnly guard;
    OEB_TRY(hdiffsa_entry<T>(outb, in, mask, crlato, crlatu, dom, stream));
  }
  Grid<T> gib, gin, gm, gob;
  Line<T> lo, lu;
  OEB_TRY((check_field3<T>(inb, *dom, Reach{2, 2, 2, 2, 0, 0}, &gib)));
  OEB_TRY((check_field3<T>(in, *dom, Reach{2, 2, 2, 2, 0, 0}, &gin)));
  OEB_TRY((check_field3<T>(mask, *dom, kInterior, &gm)));
  OEB_TRY((check_field3<T>(outb, *dom, kInterior, &gob)));
  OEB_TRY((check_field1<T>(crlato, *dom, 1, 1, &lo)));
  OEB_TRY((check_field1<T>(crlatu, *dom, 1, 1, &lu)));
  OEB_TRY(check_same_strides<T>({&gib, &gin, &gm, &gob}));
  OEB_TRY(check_no_alias({gib.lo, gib.hi},
                         {gin.lo, gin.hi, gm.lo, gm.hi, gob.lo, gob.hi, lo.lo, lo.hi, lu.lo, lu.hi}));
  OEB_RETURN_IF_VALIDATING();
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gin.sj, gin.sk};
  const int kb = tuned_kb(kKB);
  auto run = [&](auto rows) {
    constexpr int J = decltype(rows)::value;
    return launch<hdiffsa_adj_kernel<T, J>>(tile_grid(d.nx + 4, d.ny + 4, d.nz, kT, J, kb),
                                            sizeof(HdiffsaAdjSmem<T, J>), (cudaStream_t)stream, gib.origin, gin.origin,
                                            gm.origin, lo.origin, lu.origin, lo.s, gob.origin, d, kb);
  };
  // 16 rows keep more FP64 CTAs an SM (128 x 128 x 80 84.8 us, 32 rows 90.5; whole edge tiles of 32
  // rows 103.9).  FP32 pays for the larger apron (256 x 256 x 80 77.4 us, 32 rows 68.2, were 73.0) unless
  // the 32-row grid is under a wave (33 x 20 x 10 4.5 us, 32 rows 6.1).
  if constexpr (std::is_same<T, float>::value) {
    if (!under_a_wave(tile_grid(d.nx + 4, d.ny + 4, d.nz, kT, kT, kb), 8)) return run(std::integral_constant<int, kT>());
  }
  return run(std::integral_constant<int, kJ>());
}

// ============================== hdiffsmag adjoint ================================
// Linearised at (uin, vin) with the clamp of hdiffsmag.h:236/251 frozen:
//   uout = u + su Lu,  su = clamp(tau sqrt(Xu) - w mask),  Xu = (T(i+1)^2 + T^2)/2 + (S(j-1)^2 + S^2)/2
//   T = c1 (v(j-1) - v) - c2 (u(i-1) - u),  S = c1 (u(j+1) - u) + c2 (v(i+1) - v),
//   c1 = eddlat R^-1, c2(j) = acrlat0(j) eddlon, and likewise vout.
// The transpose for (uoutb, voutb), in three gather passes over scratch:
//   1. at interior points: LU = su uoutb, LV = sv voutb, and XU = Lu uoutb tau / (2 sqrt Xu)
//      where the clamp is open (0 < smag < 0.5), else 0; XV likewise;
//   2. TB = T (XU(i-1) + XU + XV(j-1) + XV) on [0,N]^2, SB = S (XU(j+1) + XU + XV(i+1) + XV)
//      on [-1,N)^2 (the T and S adjoints);
//   3. ubar, vbar on [-1,N+1)^2: identity, the transposed laplacians of LU/LV, and the T/S
//      differences of TB/SB.
template <class T>
struct SmagTerms {
  T *lu, *lv, *xu, *xv, *tb, *sb;
};

template <class T>
__device__ __forceinline__ T smag_T(const T* __restrict__ u, const T* __restrict__ v, int64_t o, int64_t sj, T c1,
                                    T c2) {
  return c1 * (ld(v + o - sj) - ld(v + o)) - c2 * (ld(u + o - 1) - ld(u + o));
}
template <class T>
__device__ __forceinline__ T smag_S(const T* __restrict__ u, const T* __restrict__ v, int64_t o, int64_t sj, T c1,
                                    T c2) {
  return c1 * (ld(u + o + sj) - ld(u + o)) + c2 * (ld(v + o + 1) - ld(v + o));
}

// T^2 and S^2 of a tile's cells, each computed once (every point reads three of each):
//   tsq : 33 x 33, (i0+a,   j0+b)     T_s^2
//   ssq : 33 x 33, (i0-1+a, j0-1+b)   S_uv^2
template <class T>
struct SmagAdjSmem {
  T tsq[33][33];
  T ssq[33][33];
};

template <class T>
struct hdiffsmag_adj_terms_kernel {
  static constexpr int kStepOp = step_op<T>(kOpSmagAdjTerms);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, SmagTerms<T> tm, const T* __restrict__ uin,
                                             const T* __restrict__ vin, const T* __restrict__ mask,
                                             const T* __restrict__ crlavo, const T* __restrict__ crlavu,
                                             const T* __restrict__ crlato, const T* __restrict__ crlatu,
                                             const T* __restrict__ acrlat0, int64_t s1d, const T* __restrict__ uoutb,
                                             const T* __restrict__ voutb, T eddlat, T eddlon, T tau_smag,
                                             T weight_smag, Dims d, int kb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmagAdjSmem<T>& s = *reinterpret_cast<SmagAdjSmem<T>*>(smem_raw);
    constexpr T rr = earth_radius_recip<T>();
    const T c1 = eddlat * rr;
    const int64_t sj = d.sj;
    const int i0 = blk.x * kT, j0 = blk.y * kT;
    const int vx = max(0, min(kT, d.nx - i0)), vy = max(0, min(kT, d.ny - j0));
    const int k0 = blk.z * kb, k1 = min(k0 + kb, d.nz);
  #pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int64_t kofs = (int64_t)k * d.sk;
      // T at (i, j) for i in [i0, i0+vx], j in [j0, j0+vy]; S at (i, j) for i in [i0-1, i0+vx),
      // j in [j0-1, j0+vy): every cell the tile's points read
      for_region_lim<33, 33>(vx + 1, vy + 1, [&](int a, int b) {
        const int i = i0 + a, j = j0 + b;
        const T t = smag_T(uin, vin, kofs + i + j * sj, sj, c1, ld(acrlat0 + (int64_t)j * s1d) * eddlon);
        s.tsq[b][a] = t * t;
      });
      for_region_lim<33, 33>(vx + 1, vy + 1, [&](int a, int b) {
        const int i = i0 - 1 + a, j = j0 - 1 + b;
        const T v = smag_S(uin, vin, kofs + i + j * sj, sj, c1, ld(acrlat0 + (int64_t)j * s1d) * eddlon);
        s.ssq[b][a] = v * v;
      });
      __syncthreads();
      for_region_lim<32, 32>(vx, vy, [&](int a, int b) {
        const int i = i0 + a, j = j0 + b;
        const int64_t o = kofs + i + j * sj;
        const T hdw = weight_smag * ld(mask + o);
        // T(i+1,j)^2 + T(i,j)^2, S(i,j-1)^2 + S(i,j)^2; T(i,j+1)^2 + T(i,j)^2, S(i-1,j)^2 + S(i,j)^2
        const T xu = T(0.5) * (s.tsq[b][a + 1] + s.tsq[b][a]) + T(0.5) * (s.ssq[b][a + 1] + s.ssq[b + 1][a + 1]);
        const T xv = T(0.5) * (s.tsq[b + 1][a] + s.tsq[b][a]) + T(0.5) * (s.ssq[b + 1][a] + s.ssq[b + 1][a + 1]);
        const T ru = Prec<T>::sqrt_(xu), rv = Prec<T>::sqrt_(xv);
        const T smu = tau_smag * ru - hdw, smv = tau_smag * rv - hdw;
        const T su = clamp_smag(smu), sv = clamp_smag(smv);
        const int64_t jo = (int64_t)j * s1d;
        const T u0 = ld(uin + o), v0 = ld(vin + o);
        const T lapu = (ld(uin + o + 1) + ld(uin + o - 1) - T(2) * u0) + ld(crlato + jo) * (ld(uin + o + sj) - u0) +
                       ld(crlatu + jo) * (ld(uin + o - sj) - u0);
        const T lapv = (ld(vin + o + 1) + ld(vin + o - 1) - T(2) * v0) + ld(crlavo + jo) * (ld(vin + o + sj) - v0) +
                       ld(crlavu + jo) * (ld(vin + o - sj) - v0);
        const T yu = ld(uoutb + o), yv = ld(voutb + o);
        tm.lu[o] = mul_zero(su, yu);
        tm.lv[o] = mul_zero(sv, yv);
        tm.xu[o] = (smu > T(0) && smu < T(0.5)) ? (lapu * yu) * (tau_smag / (T(2) * ru)) : T(0);
        tm.xv[o] = (smv > T(0) && smv < T(0.5)) ? (lapv * yv) * (tau_smag / (T(2) * rv)) : T(0);
      });
      __syncthreads();
    }
  }
};

template <class T>
struct hdiffsmag_adj_ts_kernel {
  static constexpr int kStepOp = step_op<T>(kOpSmagAdjTs);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, SmagTerms<T> tm, const T* __restrict__ uin,
                                             const T* __restrict__ vin, const T* __restrict__ acrlat0, int64_t s1d,
                                             T eddlat, T eddlon, Dims d, int kb) {
    constexpr T rr = earth_radius_recip<T>();
    const T c1 = eddlat * rr;
    const int64_t sj = d.sj;
    auto in = [&](int i, int j) { return i >= 0 && i < d.nx && j >= 0 && j < d.ny; };
    for_box<RowUnroll<T>::value>(blk, d, -1, -1, d.nx + 2, d.ny + 2, kb, [&](int64_t o, int i, int j) {
      const T c2 = ld(acrlat0 + (int64_t)j * s1d) * eddlon;
      if (i >= 0 && i <= d.nx && j >= 0 && j <= d.ny) {
        T w = T(0);
        if (in(i - 1, j)) w = tm.xu[o - 1];
        if (in(i, j)) w = w + tm.xu[o] + tm.xv[o];
        if (in(i, j - 1)) w = w + tm.xv[o - sj];
        tm.tb[o] = (w == T(0)) ? T(0) : smag_T(uin, vin, o, sj, c1, c2) * w;
      }
      if (i >= -1 && i < d.nx && j >= -1 && j < d.ny) {
        T w = T(0);
        if (in(i, j + 1)) w = tm.xu[o + sj];
        if (in(i, j)) w = w + tm.xu[o] + tm.xv[o];
        if (in(i + 1, j)) w = w + tm.xv[o + 1];
        tm.sb[o] = (w == T(0)) ? T(0) : smag_S(uin, vin, o, sj, c1, c2) * w;
      }
    });
  }
};

template <class T>
struct hdiffsmag_adj_gather_kernel {
  static constexpr int kStepOp = step_op<T>(kOpSmagAdjGather);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, T* __restrict__ uinb, T* __restrict__ vinb,
                                             SmagTerms<T> tm, const T* __restrict__ uoutb,
                                             const T* __restrict__ voutb, const T* __restrict__ crlavo,
                                             const T* __restrict__ crlavu, const T* __restrict__ crlato,
                                             const T* __restrict__ crlatu, const T* __restrict__ acrlat0, int64_t s1d,
                                             T eddlat, T eddlon, Dims d, int kb) {
    constexpr T rr = earth_radius_recip<T>();
    const T c1 = eddlat * rr;
    const int64_t sj = d.sj;
    auto in = [&](int i, int j) { return i >= 0 && i < d.nx && j >= 0 && j < d.ny; };
    auto inT = [&](int i, int j) { return i >= 0 && i <= d.nx && j >= 0 && j <= d.ny; };
    auto inS = [&](int i, int j) { return i >= -1 && i < d.nx && j >= -1 && j < d.ny; };
    for_box<RowUnroll<T>::value>(blk, d, -1, -1, d.nx + 2, d.ny + 2, kb, [&](int64_t o, int a, int b) {
      const T c2 = ld(acrlat0 + (int64_t)b * s1d) * eddlon;
      T ub = T(0), vb = T(0);
      if (in(a, b)) {
        const int64_t bo = (int64_t)b * s1d;
        ub = ld(uoutb + o) - mul_zero(tm.lu[o], T(2) + ld(crlato + bo) + ld(crlatu + bo));
        vb = ld(voutb + o) - mul_zero(tm.lv[o], T(2) + ld(crlavo + bo) + ld(crlavu + bo));
      }
      if (in(a - 1, b)) ub = ub + tm.lu[o - 1], vb = vb + tm.lv[o - 1];
      if (in(a + 1, b)) ub = ub + tm.lu[o + 1], vb = vb + tm.lv[o + 1];
      if (in(a, b - 1)) {
        const int64_t bo = (int64_t)(b - 1) * s1d;
        ub = fma(ld(crlato + bo), tm.lu[o - sj], ub);
        vb = fma(ld(crlavo + bo), tm.lv[o - sj], vb);
      }
      if (in(a, b + 1)) {
        const int64_t bo = (int64_t)(b + 1) * s1d;
        ub = fma(ld(crlatu + bo), tm.lu[o + sj], ub);
        vb = fma(ld(crlavu + bo), tm.lv[o + sj], vb);
      }
      const T tb0 = inT(a, b) ? tm.tb[o] : T(0);
      const T sb0 = inS(a, b) ? tm.sb[o] : T(0);
      if (inT(a + 1, b)) ub = fma(-c2, tm.tb[o + 1], ub);
      ub = fma(-c1, sb0, fma(c2, tb0, ub));
      if (inS(a, b - 1)) ub = fma(c1, tm.sb[o - sj], ub);
      if (inT(a, b + 1)) vb = fma(c1, tm.tb[o + sj], vb);
      vb = fma(-c2, sb0, fma(-c1, tb0, vb));
      if (inS(a - 1, b)) vb = fma(c2, tm.sb[o - 1], vb);
      uinb[o] = ub;
      vinb[o] = vb;
    });
  }
};

// FP32 adjoint in one launch, marching rows (march.cuh): lane = column i0 - 2 + lane, 28 columns of
// the box [-1, n+1)^2 a strip.  When row r of u and v arrives, a lane forms T at r and S at r - 1; the
// terms lu, lv, xu, xv of point p = r - 1; TB at p and SB at r - 2; and gathers (ubar, vbar) of row
// j = r - 2.  Neighbouring columns come from the lanes beside it, earlier rows from registers, each
// value formed once a warp.  Every value is the same expression on the same operands as in the three
// passes above (a term that is zero is added where they skip it), so the results are theirs, bit for
// bit but for the sign of a zero at the box's edge, without their 48 bytes a point of term scratch.
//
// What bounds it: instruction issue (about 320 instructions a row, two square roots and two divisions
// among them; 86 % of the issue slots taken).  79 registers, three CTAs an SM: 25.7 us at 128 x 128 x 80, 82.0 at 256 x 256 x 80, 35.4 at
// 201 x 173 x 61 (four, which spills, 34.9 / 88.8 / 42.8); the 32 x 32 shared-memory tile it replaces took
// 43.6, 125.7 and 56.3 us.
struct hdiffsmag_adj_f32 {
  static constexpr bool kAnyGrid = true;
  static constexpr int kStepOp = step_op<float>(kOpSmagAdjFused);  // the step kernel's id
  static constexpr int kCols = 28, kApron = 4, kMinCtas = 3;
  struct Row {
    float u, v, m, yu, yv;  // u and v on row r; mask, uoutb, voutb on row r - 1
  };
  static __device__ __forceinline__ void run(const uint3& blk, float* __restrict__ uinb, float* __restrict__ vinb,
                                             const float* __restrict__ uin, const float* __restrict__ vin,
                                             const float* __restrict__ mask, const float* __restrict__ crlavo,
                                             const float* __restrict__ crlavu, const float* __restrict__ crlato,
                                             const float* __restrict__ crlatu, const float* __restrict__ acrlat0,
                                             int64_t s1d, const float* __restrict__ uoutb,
                                             const float* __restrict__ voutb, float eddlat, float eddlon,
                                             float tau_smag, float weight_smag, Dims d, int rows, int wx_log) {
    const MarchPos pos = march_pos(blk, wx_log);
    const int nx = d.nx, ny = d.ny;
    const int i0 = -1 + pos.strip * kCols, oa = -1 + pos.chunk * rows, ob = min(oa + rows, ny + 1);
    if (i0 >= nx + 1 || oa >= ny + 1) return;
    constexpr float rr = earth_radius_recip<float>();
    const float c1 = eddlat * rr;
    const int lane = (int)threadIdx.x, i = i0 - 2 + lane;
    const bool ok_i = i >= -1 && i < nx + 1, in_i = i >= 0 && i < nx, t_i = i >= 0 && i <= nx, s_i = i >= -1 && i < nx;
    const bool st = ok_i && lane >= 2 && lane < 2 + kCols;
    const int64_t sjb = d.sj * 4;
    int64_t o = ((int64_t)blk.z * d.sk + (int64_t)(oa - 2) * d.sj + i) * 4;  // (i, r)
    // the metric terms of 32 rows, one a lane, handed round by shuffles
    float la, lto, ltu, lvo, lvu;
    auto metric = [&](int j) {
      const int64_t ja = (int64_t)max(-1, min(j + lane, ny)) * s1d, jo = (int64_t)max(0, min(j + lane, ny - 1)) * s1d;
      la = ld(acrlat0 + ja) * eddlon;
      lto = ld(crlato + jo), ltu = ld(crlatu + jo), lvo = ld(crlavo + jo), lvu = ld(crlavu + jo);
    };
    metric(oa - 2);
    Row n{0.f, 0.f, 0.f, 0.f, 0.f};
    auto fetch = [&](int r, int64_t q) {
      const bool ok = ok_i && r >= -1 && r <= ny, in = in_i && r >= 1 && r <= ny;
      n.u = ok ? get(uin, q) : 0.f, n.v = ok ? get(vin, q) : 0.f;
      n.m = in ? get(mask, q - sjb) : 0.f;
      n.yu = in ? get(uoutb, q - sjb) : 0.f, n.yv = in ? get(voutb, q - sjb) : 0.f;
    };
    fetch(oa - 2, o);
    float u1 = 0.f, u2 = 0.f, v1 = 0.f, v2 = 0.f;      // u, v on rows r-1, r-2
    float um1 = 0.f;                                   // u(i-1) on row r-1
    float t1 = 0.f, s2 = 0.f;                          // T at r-1, S at r-2
    float xu2 = 0.f, xv2 = 0.f;                        // at r-2
    float lu2 = 0.f, lu3 = 0.f, lv2 = 0.f, lv3 = 0.f;  // at r-2, r-3
    float tb2 = 0.f, sb3 = 0.f, yu2 = 0.f, yv2 = 0.f;  // TB at r-2, SB at r-3, the seeds at r-2
    float c21 = 0.f, c22 = 0.f;                        // acrlat0 eddlon on rows r-1, r-2
    // of rows r-2 and r-3
    float to2 = 0.f, to3 = 0.f, tu2 = 0.f, vo2 = 0.f, vo3 = 0.f, vu2 = 0.f;
    bool in2 = false, in3 = false;  // whether those rows' points are interior
#pragma unroll 1
    for (int r = oa - 2; r < ob + 2; ++r) {
      const Row c = n;
      if (r + 1 < ob + 2) fetch(r + 1, o + sjb);
      const int src = (r + 2 - oa) & 31, srp = (r + 1 - oa) & 31;
      // the terms of row p = r - 1 are handed round before the lanes move on to the next 32 rows
      const float to = __shfl_sync(kWarpMask, lto, srp), tu = __shfl_sync(kWarpMask, ltu, srp),
                  vo = __shfl_sync(kWarpMask, lvo, srp), vu = __shfl_sync(kWarpMask, lvu, srp);
      if (src == 0 && r > oa - 2) metric(r);
      const float c2 = __shfl_sync(kWarpMask, la, src);
      const int p = r - 1, j = r - 2;
      const bool in_p = in_i && p >= 0 && p < ny;
      // T at r and S at p (smag_T, smag_S)
      const float um = lane_below<1>(c.u);
      const float tv = c1 * (v1 - c.v) - c2 * (um - c.u);
      const float t0 = t_i && r >= 0 && r <= ny ? tv : 0.f;
      const float sv = c1 * (c.u - u1) + c21 * (lane_above<1>(v1) - v1);
      const float s1 = s_i && p >= -1 && p < ny ? sv : 0.f;
      // the terms at p (hdiffsmag_adj_terms_kernel)
      const float tip = lane_above<1>(t1), sim = lane_below<1>(s1);
      const float xuu = 0.5f * (tip * tip + t1 * t1) + 0.5f * (s2 * s2 + s1 * s1);
      const float xvv = 0.5f * (t0 * t0 + t1 * t1) + 0.5f * (sim * sim + s1 * s1);
      const float hdw = weight_smag * c.m;
      const float ru = sqrtf(numerator(in_p, xuu)), rv = sqrtf(numerator(in_p, xvv));
      const float smu = tau_smag * ru - hdw, smv = tau_smag * rv - hdw;
      const float lapu = (lane_above<1>(u1) + um1 - 2.f * u1) + to * (c.u - u1) + tu * (u2 - u1);
      const float lapv = (lane_above<1>(v1) + lane_below<1>(v1) - 2.f * v1) + vo * (c.v - v1) + vu * (v2 - v1);
      const bool open_u = in_p && smu > 0.f && smu < 0.5f, open_v = in_p && smv > 0.f && smv < 0.5f;
      const float xuv = (lapu * c.yu) * (tau_smag / (2.f * numerator(open_u, ru)));
      const float xvw = (lapv * c.yv) * (tau_smag / (2.f * numerator(open_v, rv)));
      const float lu1 = in_p ? clamp_smag(smu) * c.yu : 0.f, lv1 = in_p ? clamp_smag(smv) * c.yv : 0.f;
      const float xu1 = open_u ? xuv : 0.f, xv1 = open_v ? xvw : 0.f;
      // TB at p and SB at j (hdiffsmag_adj_ts_kernel)
      const float wt = (((0.f + lane_below<1>(xu1)) + xu1) + xv1) + xv2;
      const float tb1 = (wt == 0.f || !(t_i && p >= 0 && p <= ny)) ? 0.f : t1 * wt;
      const float ws = (((0.f + xu1) + xu2) + xv2) + lane_above<1>(xv2);
      const float sb2 = (ws == 0.f || !(s_i && j >= -1 && j < ny)) ? 0.f : s2 * ws;
      // the gather at row j (hdiffsmag_adj_gather_kernel)
      float ub = 0.f, vb = 0.f;
      if (in_i && j >= 0 && j < ny) {
        ub = yu2 - (2.f + to2 + tu2) * lu2;
        vb = yv2 - (2.f + vo2 + vu2) * lv2;
      }
      ub = ub + lane_below<1>(lu2), vb = vb + lane_below<1>(lv2);
      ub = ub + lane_above<1>(lu2), vb = vb + lane_above<1>(lv2);
      // (guarded: a metric term need not be finite, and off the interior lu and lv are only stand-ins)
      if (in3) ub = fmaf(to3, lu3, ub), vb = fmaf(vo3, lv3, vb);
      if (in_p) ub = fmaf(tu, lu1, ub), vb = fmaf(vu, lv1, vb);
      ub = fmaf(-c22, lane_above<1>(tb2), ub);
      ub = fmaf(-c1, sb2, fmaf(c22, tb2, ub));
      ub = fmaf(c1, sb3, ub);
      vb = fmaf(c1, tb1, vb);
      vb = fmaf(-c22, sb2, fmaf(-c1, tb2, vb));
      vb = fmaf(c22, lane_below<1>(sb2), vb);
      if (st && j >= oa) put(uinb, o - 2 * sjb, ub), put(vinb, o - 2 * sjb, vb);
      u2 = u1, u1 = c.u, v2 = v1, v1 = c.v, um1 = um;
      t1 = t0, s2 = s1, xu2 = xu1, xv2 = xv1;
      lu3 = lu2, lu2 = lu1, lv3 = lv2, lv2 = lv1;
      tb2 = tb1, sb3 = sb2, yu2 = c.yu, yv2 = c.yv;
      c22 = c21, c21 = c2;
      to3 = to2, to2 = to, tu2 = tu, vo3 = vo2, vo2 = vo, vu2 = vu;
      in3 = in2, in2 = in_p;
      o += sjb;
    }
  }
};

template <class T, class M3, class M1>
oeb_status hdiffsmag_adj_entry(const M3* uinb, const M3* vinb, const M3* uin, const M3* vin, const M3* mask,
                               const M1* crlavo, const M1* crlavu, const M1* crlato, const M1* crlatu,
                               const M1* acrlat0, const M3* uoutb, const M3* voutb, T eddlat, T eddlon, T tau_smag,
                               T weight_smag, const oeb_domain* dom, void* stream) {
  {
    ValidateOnly guard;
    OEB_TRY(hdiffsmag_entry<T>(uoutb, voutb, uin, vin, mask, crlavo, crlavu, crlato, crlatu, acrlat0, eddlat, eddlon,
                               tau_smag, weight_smag, dom, stream));
  }
  Grid<T> gub, gvb, gui, guo;
  OEB_TRY((check_field3<T>(uinb, *dom, Reach{1, 1, 1, 1, 0, 0}, &gub)));
  OEB_TRY((check_field3<T>(vinb, *dom, Reach{1, 1, 1, 1, 0, 0}, &gvb)));
  OEB_TRY((check_field3<T>(uin, *dom, Reach{1, 1, 1, 1, 0, 0}, &gui)));
  OEB_TRY((check_field3<T>(uoutb, *dom, kInterior, &guo)));
  OEB_TRY(check_same_strides<T>({&gub, &gvb, &gui, &guo}));
  OEB_TRY(check_no_alias({gub.lo, gub.hi, gvb.lo, gvb.hi}, {gui.lo, gui.hi, guo.lo, guo.hi}));
  OEB_RETURN_IF_VALIDATING();
  cudaStream_t st = (cudaStream_t)stream;
  if constexpr (std::is_same<T, float>::value) if (adjoint_tiles()) {
    const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gui.sj, gui.sk};
    using B = hdiffsmag_adj_f32;
    const MarchShape m = march_shape(d.nx + 2, d.ny + 2, d.nz, 1, B::kCols, B::kApron, B::kMinCtas);
    auto org1 = [](const M1* m1) { return (const float*)m1->aligned + m1->offset; };
    return launch<B>(m.grid, 0, st, gub.origin, gvb.origin, gui.origin, (const float*)vin->aligned + vin->offset,
                     (const float*)mask->aligned + mask->offset, org1(crlavo), org1(crlavu), org1(crlato), org1(crlatu),
                     org1(acrlat0), acrlat0->strides[0], guo.origin, (const float*)voutb->aligned + voutb->offset,
                     eddlat, eddlon, tau_smag, weight_smag, d, m.rows, m.wx_log);
  }
  const T* start = (uin->allocated && uin->allocated <= uin->aligned) ? uin->allocated : uin->aligned;
  const int64_t last = (uin->sizes[0] - 1) * uin->strides[0] + (uin->sizes[1] - 1) * uin->strides[1] +
                       (uin->sizes[2] - 1) * uin->strides[2];
  const int64_t n = (int64_t)(uin->aligned - start) + last + 1;
  const int64_t org = (int64_t)(uin->aligned - start) + uin->offset;
  void* buf = nullptr;
  OEB_TRY(scratch_alloc(&buf, (size_t)n * 6 * sizeof(T), st));
  T* base = static_cast<T*>(buf);
  SmagTerms<T> tm{base + org, base + n + org, base + 2 * n + org, base + 3 * n + org, base + 4 * n + org,
                  base + 5 * n + org};
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gui.sj, gui.sk};
  auto org1 = [](const M1* m) { return (const T*)m->aligned + m->offset; };
  const int64_t s1d = acrlat0->strides[0];
  const int kb = tuned_kb(kKB);
  oeb_status stt = launch<hdiffsmag_adj_terms_kernel<T>>(
      tile_grid(d.nx, d.ny, d.nz, kT, kT, kb), sizeof(SmagAdjSmem<T>), st, tm, gui.origin, (const T*)vin->aligned + vin->offset,
      (const T*)mask->aligned + mask->offset, org1(crlavo), org1(crlavu), org1(crlato), org1(crlatu), org1(acrlat0), s1d,
      guo.origin, (const T*)voutb->aligned + voutb->offset, eddlat, eddlon, tau_smag, weight_smag, d, kb);
  Dims dp = d;
  dp.tj = point_rows<T>(tile_grid(d.nx + 2, d.ny + 2, d.nz, kT, kT, kb), kDerivativeTiles);
  if (stt == OEB_OK)
    stt = launch<hdiffsmag_adj_ts_kernel<T>>(tile_grid(d.nx + 2, d.ny + 2, d.nz, kT, dp.tj, kb), 0, st, tm, gui.origin,
                                             (const T*)vin->aligned + vin->offset, org1(acrlat0), s1d, eddlat, eddlon,
                                             dp, kb);
  if (stt == OEB_OK)
    stt = launch<hdiffsmag_adj_gather_kernel<T>>(
        tile_grid(d.nx + 2, d.ny + 2, d.nz, kT, dp.tj, kb), 0, st, gub.origin, gvb.origin, tm, guo.origin,
        (const T*)voutb->aligned + voutb->offset, org1(crlavo), org1(crlavu), org1(crlato), org1(crlatu), org1(acrlat0),
        s1d, eddlat, eddlon, dp, kb);
  scratch_free(buf, st);
  return stt;
}

#ifndef OEB_BODIES_ONLY
// ==================== hdiffsmag adjoint without any allocation (FP64) ====================
// oeb_hdiffsmag_adj_noalloc_f64 is for callers that cannot allocate device memory while they
// run: a host whose own allocator has already claimed the GPU's memory up front (an
// allocation from this library's pool could then fail in the middle of a run), or a
// time-stepping loop that must not take an allocation inside its step.  It runs the same three
// kernels as oeb_hdiffsmag_adj_f64, on the same validated arguments, but its six term fields
// live in one fixed array compiled into the library instead of coming from the pool.
//
//  * Limit: each term field holds kNoAllocCells = 2^21 cells, so the span of uin's
//    allocation (halo and padding included) may be at most 2^21 cells; a larger field is
//    rejected with OEB_ERR_TOO_LARGE before anything runs.  The array is 6 x 2^21 doubles =
//    96 MiB, and every GPU that loads the library holds it until the process exits.
//  * Every call uses the same array, which keeps the last call's contents.  Each cell the
//    kernels read is written earlier in the same call (the terms on the interior, the T/S
//    adjoints on their boxes), so nothing has to start at zero and nothing is cleared.  Calls
//    that overlap on the GPU -- on two streams, or from two host threads -- race on the array.
//  * Set-up: the array's name is only a host-side stand-in for the device variable.  The first
//    call on a device looks up its device address with cudaGetSymbolAddress, with that device
//    current, and keeps it for later calls; make that first call before any stream capture.
//    The kept address outlives a cudaDeviceReset of that device, after which it is stale: the
//    entry point is not for use on a device after such a reset.
constexpr int64_t kNoAllocCells = int64_t(1) << 21;
static __device__ __align__(256) double g_hdiffsmag_adj_scratch[6 * kNoAllocCells];

oeb_status hdiffsmag_adj_scratch_address(double** out) {
  static std::mutex mu;
  static std::vector<double*> addr;  // per device
  int dev = 0;
  OEB_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  if ((int)addr.size() <= dev) addr.resize(dev + 1, nullptr);
  if (!addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_hdiffsmag_adj_scratch);
    if (e != cudaSuccess) return cuda_fail(e);
    addr[dev] = static_cast<double*>(p);
  }
  *out = addr[dev];
  return OEB_OK;
}

oeb_status hdiffsmag_adj_noalloc_entry(const oeb_memref3d_f64* uinb, const oeb_memref3d_f64* vinb,
                                       const oeb_memref3d_f64* uin, const oeb_memref3d_f64* vin,
                                       const oeb_memref3d_f64* mask, const oeb_memref1d_f64* crlavo,
                                       const oeb_memref1d_f64* crlavu, const oeb_memref1d_f64* crlato,
                                       const oeb_memref1d_f64* crlatu, const oeb_memref1d_f64* acrlat0,
                                       const oeb_memref3d_f64* uoutb, const oeb_memref3d_f64* voutb, double eddlat,
                                       double eddlon, double tau_smag, double weight_smag, const oeb_domain* dom,
                                       void* stream) {
  using T = double;
  {
    // every check of the pool-backed entry point, nothing launched
    ValidateOnly guard;
    OEB_TRY(hdiffsmag_adj_entry<T>(uinb, vinb, uin, vin, mask, crlavo, crlavu, crlato, crlatu, acrlat0, uoutb, voutb,
                                   eddlat, eddlon, tau_smag, weight_smag, dom, stream));
  }
  Grid<T> gub, gvb, gui, guo;
  OEB_TRY((check_field3<T>(uinb, *dom, Reach{1, 1, 1, 1, 0, 0}, &gub)));
  OEB_TRY((check_field3<T>(vinb, *dom, Reach{1, 1, 1, 1, 0, 0}, &gvb)));
  OEB_TRY((check_field3<T>(uin, *dom, Reach{1, 1, 1, 1, 0, 0}, &gui)));
  OEB_TRY((check_field3<T>(uoutb, *dom, kInterior, &guo)));
  const T* start = (uin->allocated && uin->allocated <= uin->aligned) ? uin->allocated : uin->aligned;
  const int64_t last = (uin->sizes[0] - 1) * uin->strides[0] + (uin->sizes[1] - 1) * uin->strides[1] +
                       (uin->sizes[2] - 1) * uin->strides[2];
  const int64_t n = (int64_t)(uin->aligned - start) + last + 1;
  const int64_t org = (int64_t)(uin->aligned - start) + uin->offset;
  if (n > kNoAllocCells) return OEB_ERR_TOO_LARGE;
  OEB_RETURN_IF_VALIDATING();
  T* base = nullptr;
  OEB_TRY(hdiffsmag_adj_scratch_address(&base));
  SmagTerms<T> tm{base + org, base + kNoAllocCells + org, base + 2 * kNoAllocCells + org,
                  base + 3 * kNoAllocCells + org, base + 4 * kNoAllocCells + org, base + 5 * kNoAllocCells + org};
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gui.sj, gui.sk};
  auto org1 = [](const oeb_memref1d_f64* m) { return (const T*)m->aligned + m->offset; };
  const int64_t s1d = acrlat0->strides[0];
  cudaStream_t st = (cudaStream_t)stream;
  OEB_TRY(launch<hdiffsmag_adj_terms_kernel<T>>(
      tile_grid(d.nx, d.ny, d.nz, kT, kT, kKB), sizeof(SmagAdjSmem<T>), st, tm, gui.origin, (const T*)vin->aligned + vin->offset,
      (const T*)mask->aligned + mask->offset, org1(crlavo), org1(crlavu), org1(crlato), org1(crlatu), org1(acrlat0), s1d,
      guo.origin, (const T*)voutb->aligned + voutb->offset, eddlat, eddlon, tau_smag, weight_smag, d, kKB));
  OEB_TRY(launch<hdiffsmag_adj_ts_kernel<T>>(tile_grid(d.nx + 2, d.ny + 2, d.nz, kT, kT, kKB), 0, st, tm, gui.origin,
                                             (const T*)vin->aligned + vin->offset, org1(acrlat0), s1d, eddlat, eddlon,
                                             d, kKB));
  return launch<hdiffsmag_adj_gather_kernel<T>>(
      tile_grid(d.nx + 2, d.ny + 2, d.nz, kT, kT, kKB), 0, st, gub.origin, gvb.origin, tm, guo.origin,
      (const T*)voutb->aligned + voutb->offset, org1(crlavo), org1(crlavu), org1(crlato), org1(crlatu), org1(acrlat0),
      s1d, eddlat, eddlon, d, kKB);
}
#endif  // OEB_BODIES_ONLY

}  // namespace
}  // namespace oeb

#ifndef OEB_BODIES_ONLY  // the entry points

using namespace oeb;

#define OEB_HDIFF_ENTRIES(S, T)                                                                                     \
  extern "C" oeb_status oeb_hdiffsa_##S(const oeb_memref3d_##S* out, const oeb_memref3d_##S* in,                   \
                                        const oeb_memref3d_##S* mask, const oeb_memref1d_##S* crlato,             \
                                        const oeb_memref1d_##S* crlatu, const oeb_domain* dom, void* stream) {    \
    return hdiffsa_entry<T>(out, in, mask, crlato, crlatu, dom, stream);                                          \
  }                                                                                                                \
  extern "C" oeb_status oeb_hdiffsmag_##S(                                                                         \
      const oeb_memref3d_##S* uout, const oeb_memref3d_##S* vout, const oeb_memref3d_##S* uin,                      \
      const oeb_memref3d_##S* vin, const oeb_memref3d_##S* mask, const oeb_memref1d_##S* crlavo,                    \
      const oeb_memref1d_##S* crlavu, const oeb_memref1d_##S* crlato, const oeb_memref1d_##S* crlatu,               \
      const oeb_memref1d_##S* acrlat0, T eddlat, T eddlon, T tau_smag, T weight_smag, const oeb_domain* dom,       \
      void* stream) {                                                                                              \
    return hdiffsmag_entry<T>(uout, vout, uin, vin, mask, crlavo, crlavu, crlato, crlatu, acrlat0, eddlat, eddlon,\
                              tau_smag, weight_smag, dom, stream);                                                 \
  }                                                                                                                \
  extern "C" oeb_status oeb_hdiffsmag_tl_##S(                                                                      \
      const oeb_memref3d_##S* duout, const oeb_memref3d_##S* dvout, const oeb_memref3d_##S* uin,                    \
      const oeb_memref3d_##S* vin, const oeb_memref3d_##S* mask, const oeb_memref1d_##S* crlavo,                    \
      const oeb_memref1d_##S* crlavu, const oeb_memref1d_##S* crlato, const oeb_memref1d_##S* crlatu,               \
      const oeb_memref1d_##S* acrlat0, const oeb_memref3d_##S* duin, const oeb_memref3d_##S* dvin, T eddlat,        \
      T eddlon, T tau_smag, T weight_smag, const oeb_domain* dom, void* stream) {                                  \
    return hdiffsmag_tl_entry<T>(duout, dvout, uin, vin, mask, crlavo, crlavu, crlato, crlatu, acrlat0, duin, dvin, \
                                 eddlat, eddlon, tau_smag, weight_smag, dom, stream);                             \
  }                                                                                                                \
  extern "C" oeb_status oeb_hdiffsmag_adj_##S(                                                                     \
      const oeb_memref3d_##S* uinb, const oeb_memref3d_##S* vinb, const oeb_memref3d_##S* uin,                      \
      const oeb_memref3d_##S* vin, const oeb_memref3d_##S* mask, const oeb_memref1d_##S* crlavo,                    \
      const oeb_memref1d_##S* crlavu, const oeb_memref1d_##S* crlato, const oeb_memref1d_##S* crlatu,               \
      const oeb_memref1d_##S* acrlat0, const oeb_memref3d_##S* uoutb, const oeb_memref3d_##S* voutb, T eddlat,      \
      T eddlon, T tau_smag, T weight_smag, const oeb_domain* dom, void* stream) {                                  \
    return hdiffsmag_adj_entry<T>(uinb, vinb, uin, vin, mask, crlavo, crlavu, crlato, crlatu, acrlat0, uoutb,     \
                                  voutb, eddlat, eddlon, tau_smag, weight_smag, dom, stream);                     \
  }

#define OEB_HDIFFSA_DIFF_ENTRIES(S, T)                                                                              \
  extern "C" oeb_status oeb_hdiffsa_tl_##S(const oeb_memref3d_##S* dout, const oeb_memref3d_##S* in,               \
                                           const oeb_memref3d_##S* mask, const oeb_memref1d_##S* crlato,          \
                                           const oeb_memref1d_##S* crlatu, const oeb_memref3d_##S* din,           \
                                           const oeb_domain* dom, void* stream) {                                  \
    return hdiffsa_tl_entry<T>(dout, in, mask, crlato, crlatu, din, dom, stream);                                  \
  }                                                                                                                \
  extern "C" oeb_status oeb_hdiffsa_adj_##S(const oeb_memref3d_##S* inb, const oeb_memref3d_##S* in,              \
                                            const oeb_memref3d_##S* mask, const oeb_memref1d_##S* crlato,         \
                                            const oeb_memref1d_##S* crlatu, const oeb_memref3d_##S* outb,         \
                                            const oeb_domain* dom, void* stream) {                                 \
    return hdiffsa_adj_entry<T>(inb, in, mask, crlato, crlatu, outb, dom, stream);                                 \
  }

OEB_HDIFF_ENTRIES(f64, double)
OEB_HDIFF_ENTRIES(f32, float)
OEB_HDIFFSA_DIFF_ENTRIES(f64, double)
OEB_HDIFFSA_DIFF_ENTRIES(f32, float)

extern "C" oeb_status oeb_hdiffsmag_adj_noalloc_f64(
    const oeb_memref3d_f64* uinb, const oeb_memref3d_f64* vinb, const oeb_memref3d_f64* uin,
    const oeb_memref3d_f64* vin, const oeb_memref3d_f64* mask, const oeb_memref1d_f64* crlavo,
    const oeb_memref1d_f64* crlavu, const oeb_memref1d_f64* crlato, const oeb_memref1d_f64* crlatu,
    const oeb_memref1d_f64* acrlat0, const oeb_memref3d_f64* uoutb, const oeb_memref3d_f64* voutb, double eddlat,
    double eddlon, double tau_smag, double weight_smag, const oeb_domain* dom, void* stream) {
  return hdiffsmag_adj_noalloc_entry(uinb, vinb, uin, vin, mask, crlavo, crlavu, crlato, crlatu, acrlat0, uoutb, voutb,
                                     eddlat, eddlon, tau_smag, weight_smag, dom, stream);
}

#endif  // OEB_BODIES_ONLY
