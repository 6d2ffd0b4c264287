// k_fastwavesuv.cu -- fastwavesuv (kernels/fastwavesuv.h:154-191) in FP64 and FP32 (the latter by
// fastwavesuv_march_f32 below).
//
// The OpenMP variant evaluates ppgk = wgtfac*ppuv + (1-wgtfac)*ppuv(k-1) six times per point
// ((i,j),(i+1,j),(i,j+1) at k and k+1).  Here each CTA marches upward through kb k-levels
// of a 32 x 32 tile: at level k every point of the tile plus a one-cell apron in i and j
// computes ppgk(k+1) once, keeps it in a register for level k+1, and publishes
// ppgc = ppgk(k+1) - ppgk(k) and the hhl sum and difference of its column through shared
// memory; the output pass then reads its i+1 and j+1 neighbours from there.
//
// Compiled with --fmad=false (see k_pointwise.cu).
#include <type_traits>

#include "march.cuh"
#include "precision.cuh"
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
constexpr int kR = kT + 1;                                // apron of one cell in i and j
constexpr int kOwned = (kR * kR + kThreads - 1) / kThreads;  // region points per thread

template <class T>
struct FastwavesSmem {
  T ppgc[kR][kR];
  T hs[kR][kR];  // hhl(k+1) + hhl(k)
  T hd[kR][kR];  // hhl(k+1) - hhl(k)
  T fx2[kT];     // 2 * fx(j)
};

template <class T>
struct fastwavesuv_kernel {
  static constexpr int kStepOp = step_op<T>(kOpFwsFwd);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, OutPtr<T> uout, OutPtr<T> vout,
                                             InPtr<T> uin, InPtr<T> vin,
                                             InPtr<T> utens, InPtr<T> vtens,
                                             InPtr<T> wgtfac, InPtr<T> ppuv,
                                             InPtr<T> hhl, InPtr<T> rho,
                                             InPtr<T> fx, int64_t s1d, T ed2, T dt, Dims d, int kb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FastwavesSmem<T>& s = *reinterpret_cast<FastwavesSmem<T>*>(smem_raw);
    const int i0 = blk.x * kT, j0 = blk.y * kT;
    const int sj = (int)d.sj;
    const int64_t sk = d.sk;
    const int tid = threadIdx.y * kTX + threadIdx.x;
    if (tid < kT) {
      const int j = j0 + tid;
      s.fx2[tid] = (j < d.ny) ? T(2.0) * ld(fx + (int64_t)j * s1d) : T(0);
    }
    const int k0 = blk.z * kb, k1 = min(k0 + kb, d.nz);

    // Region points owned by this thread, and ppgk at the current level for each.
    int own_off[kOwned];
    bool own_ok[kOwned];
    T ppgk_cur[kOwned];
  #pragma unroll
    for (int t = 0; t < kOwned; ++t) {
      const int e = tid + t * kThreads;
      const int b = e / kR, a = e - (e / kR) * kR;
      const int i = i0 + a, j = j0 + b;
      own_ok[t] = e < kR * kR && i < d.nx + 1 && j < d.ny + 1;
      own_off[t] = i + j * sj;
      ppgk_cur[t] = T(0);
      if (own_ok[t]) {
        const int64_t o = (int64_t)k0 * sk + own_off[t];
        const T w = ld(wgtfac + o);
        ppgk_cur[t] = w * ld(ppuv + o) + (T(1.0) - w) * ld(ppuv + o - sk);  // fastwavesuv.h:162
      }
    }

  #pragma unroll 1
    for (int k = k0; k < k1; ++k) {
      const int64_t kofs = (int64_t)k * sk;
      const InPtr<T> late[6] = {ppuv, rho, uin, utens, vin, vtens};  // read in the last phase
      prefetch_tile<T>(late, kofs, i0, j0, d.nx, d.ny, sj);
  #pragma unroll
      for (int t = 0; t < kOwned; ++t) {
        const int e = tid + t * kThreads;
        if (e < kR * kR) {
          const int b = e / kR, a = e - b * kR;
          T pc = T(0), hsum = T(0), hdif = T(0);
          if (own_ok[t]) {
            const int64_t o = kofs + own_off[t];
            const T w1 = ld(wgtfac + o + sk);
            const T next = w1 * ld(ppuv + o + sk) + (T(1.0) - w1) * ld(ppuv + o);  // ppgk at k+1
            pc = next - ppgk_cur[t];
            ppgk_cur[t] = next;
            const T h1 = ld(hhl + o + sk), h0 = ld(hhl + o);
            hsum = h1 + h0;
            hdif = h1 - h0;
          }
          s.ppgc[b][a] = pc;
          s.hs[b][a] = hsum;
          s.hd[b][a] = hdif;
        }
      }
      __syncthreads();
      for_region<kT, kT>([&](int a, int b) {
        const int i = i0 + a, j = j0 + b;
        if (i < d.nx && j < d.ny) {
          const int64_t o = kofs + i + j * sj;
          const T p0 = ld(ppuv + o);
          const T r0 = ld(rho + o);
          // fastwavesuv.h:172-175
          const T ppgu = (ld(ppuv + o + 1) - p0) + (scale2<-1>(s.ppgc[b][a + 1] + s.ppgc[b][a]) *
                                                        (s.hs[b][a] - s.hs[b][a + 1])) /
                                                           (s.hd[b][a] + s.hd[b][a + 1]);
          // fastwavesuv.h:177-180
          const T ppgv = (ld(ppuv + o + sj) - p0) + (scale2<-1>(s.ppgc[b + 1][a] + s.ppgc[b][a]) *
                                                         (s.hs[b][a] - s.hs[b + 1][a])) /
                                                            (s.hd[b][a] + s.hd[b + 1][a]);
          // fastwavesuv.h:182-186
          uout[o] = ld(uin + o) + dt * (ld(utens + o) - ppgu * (s.fx2[b] / (ld(rho + o + 1) + r0)));
          vout[o] = ld(vin + o) + dt * (ld(vtens + o) - ppgv * (ed2 / (ld(rho + o + sj) + r0)));
        }
      });
      __syncthreads();
    }
  }
};

// FP32 fastwavesuv, marching rows (march.cuh) of one level: lane = column i0 + lane, 31 columns a strip.
// Each row's ppgc, hhl sum and difference, ppuv and rho are formed once; uout at that row takes the
// lane above's, vout at the row before takes the row's own.  ppgk at k and k+1 are both formed (the
// level's neighbours are read again from L2, where the CTAs of the levels beside it have just read
// them).  fastwavesuv_kernel's operations on the same operands in the same order: the same bits.
//
// What bounds it: instruction issue (about 190 instructions a row, its four IEEE divisions a quarter of
// them) and DRAM latency; DRAM moves the inputs and outputs once.  64 registers, four CTAs an SM:
// 49.8 us at 256 x 256 x 80 (0.62 of the HBM copy rate), 17.3 at 128 x 128 x 80, 113.9 at
// 320 x 304 x 137 (five CTAs 48.3 / 17.3 / 114.0, slower on small domains; six, which spills, 75.2);
// fastwavesuv_kernel<float>'s shared-memory tile took 95.7, 33.5 and 228.8 us.
struct fastwavesuv_march_f32 {
  static constexpr bool kAnyGrid = true;
  static constexpr int kStepOp = step_op<float>(kOpFwsFwd);  // the step kernel's id
  static constexpr int kCols = 31, kApron = 1, kMinCtas = 4;
  struct Row {
    float w0, w1, pm, p0, p1, h0, h1, r;  // row j: wgtfac, ppuv, hhl at k (and beside it), rho
    float u, ut, v, vt;                   // uin, utens on row j; vin, vtens on row j - 1
  };
  static __device__ __forceinline__ void run(const uint3& blk, float* __restrict__ uout, float* __restrict__ vout,
                                             const float* __restrict__ uin, const float* __restrict__ vin,
                                             const float* __restrict__ utens, const float* __restrict__ vtens,
                                             const float* __restrict__ wgtfac, const float* __restrict__ ppuv,
                                             const float* __restrict__ hhl, const float* __restrict__ rho,
                                             const float* __restrict__ fx, int64_t s1d, float ed2, float dt, Dims d,
                                             int rows, int wx_log) {
    const MarchPos pos = march_pos(blk, wx_log);
    const int nx = d.nx, ny = d.ny;
    const int i0 = pos.strip * kCols, ja = pos.chunk * rows, jb = min(ja + rows, ny);
    if (i0 >= nx || ja >= ny) return;
    const int lane = (int)threadIdx.x, i = min(i0 + lane, nx);  // lanes past the reach repeat its last column
    const bool st = lane < kCols && i0 + lane < nx;
    const int64_t sjb = d.sj * 4, skb = d.sk * 4;
    int64_t o = ((int64_t)blk.z * d.sk + (int64_t)ja * d.sj + i) * 4;  // (i, j)
    const int64_t oi = (int64_t)(min(i, nx - 1) - i) * 4;              // to an interior column
    float lf;
    auto metric = [&](int j) { lf = 2.f * ld(fx + (int64_t)min(j + lane, ny - 1) * s1d); };
    metric(ja);
    Row n;
    auto fetch = [&](int j, int64_t q) {
      n.w0 = get(wgtfac, q), n.w1 = get(wgtfac, q + skb);
      n.pm = get(ppuv, q - skb), n.p0 = get(ppuv, q), n.p1 = get(ppuv, q + skb);
      n.h0 = get(hhl, q), n.h1 = get(hhl, q + skb), n.r = get(rho, q);
      if (j < jb) n.u = get(uin, q + oi), n.ut = get(utens, q + oi);
      if (j > ja) n.v = get(vin, q + oi - sjb), n.vt = get(vtens, q + oi - sjb);
    };
    fetch(ja, o);
    float pc = 0.f, hs = 0.f, hd = 0.f, p = 0.f, r = 0.f;  // of row j - 1
#pragma unroll 1
    for (int j = ja; j <= jb; ++j) {
      const Row c = n;
      if (j < jb) fetch(j + 1, o + sjb);
      const float cur = c.w0 * c.p0 + (1.f - c.w0) * c.pm;   // ppgk at k (fastwavesuv.h:162)
      const float next = c.w1 * c.p1 + (1.f - c.w1) * c.p0;  // and at k + 1
      const float pcj = next - cur, hsj = c.h1 + c.h0, hdj = c.h1 - c.h0;
      if (j < jb) {
        const int src = (j - ja) & 31;
        if (src == 0 && j > ja) metric(j);
        const float fx2 = __shfl_sync(kWarpMask, lf, src);
        // fastwavesuv.h:172-175, :182-183
        // a lane that writes nothing has itself or a copy above it: its numerator is zero
        const float num = (0.5f * (lane_above<1>(pcj) + pcj)) * (hsj - lane_above<1>(hsj));
        const float ppgu = (lane_above<1>(c.p0) - c.p0) + numerator(st, num) / (hdj + lane_above<1>(hdj));
        const float uo = c.u + dt * (c.ut - ppgu * (fx2 / (lane_above<1>(c.r) + c.r)));
        if (st) put(uout, o, uo);
      }
      if (j > ja) {
        // fastwavesuv.h:177-180, :185-186, at row j - 1
        const float ppgv = (c.p0 - p) + ((0.5f * (pcj + pc)) * (hs - hsj)) / (hd + hdj);
        const float vo = c.v + dt * (c.vt - ppgv * (ed2 / (c.r + r)));
        if (st) put(vout, o - sjb, vo);
      }
      pc = pcj, hs = hsj, hd = hdj, p = c.p0, r = c.r;
      o += sjb;
    }
  }
};

constexpr int kKB = 1;  // k-levels per CTA by default (the most CTAs hide latency best)
template <class T, class M3, class M1>
oeb_status fastwavesuv_entry(const M3* uout, const M3* vout, const M3* uin, const M3* vin, const M3* utens,
                             const M3* vtens, const M3* wgtfac, const M3* ppuv, const M3* hhl, const M3* rho,
                             const M1* fx, T edadlat, T dt, const oeb_domain* dom, void* stream) {
  OEB_TRY(check_domain(dom));
  Grid<T> gu, gv, gui, gvi, gut, gvt, gw, gp, gh, gr;
  Line<T> lfx;
  OEB_TRY((check_field3<T>(uout, *dom, kInterior, &gu)));
  OEB_TRY((check_field3<T>(vout, *dom, kInterior, &gv)));
  OEB_TRY((check_field3<T>(uin, *dom, kInterior, &gui)));
  OEB_TRY((check_field3<T>(vin, *dom, kInterior, &gvi)));
  OEB_TRY((check_field3<T>(utens, *dom, kInterior, &gut)));
  OEB_TRY((check_field3<T>(vtens, *dom, kInterior, &gvt)));
  OEB_TRY((check_field3<T>(wgtfac, *dom, Reach{0, 1, 0, 1, 0, 1}, &gw)));
  OEB_TRY((check_field3<T>(ppuv, *dom, Reach{0, 1, 0, 1, 1, 1}, &gp)));
  OEB_TRY((check_field3<T>(hhl, *dom, Reach{0, 1, 0, 1, 0, 1}, &gh)));
  OEB_TRY((check_field3<T>(rho, *dom, Reach{0, 1, 0, 1, 0, 0}, &gr)));
  OEB_TRY((check_field1<T>(fx, *dom, 0, 0, &lfx)));
  OEB_TRY(check_same_strides<T>({&gu, &gv, &gui, &gvi, &gut, &gvt, &gw, &gp, &gh, &gr}));
  OEB_TRY(check_no_alias({gu.lo, gu.hi, gv.lo, gv.hi},
                         {gui.lo, gui.hi, gvi.lo, gvi.hi, gut.lo, gut.hi, gvt.lo, gvt.hi, gw.lo, gw.hi, gp.lo, gp.hi,
                          gh.lo, gh.hi, gr.lo, gr.hi, lfx.lo, lfx.hi}));
  OEB_RETURN_IF_VALIDATING();
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gu.sj, gu.sk};
  const T ed2 = T(2.0) * edadlat;  // ElementType(2.0) * edadlat, fastwavesuv.h:186
  if constexpr (std::is_same<T, float>::value) {
    using B = fastwavesuv_march_f32;
    const MarchShape m = march_shape(d.nx, d.ny, d.nz, 1, B::kCols, B::kApron, B::kMinCtas);
    return launch<B>(m.grid, 0, (cudaStream_t)stream, gu.origin, gv.origin, gui.origin, gvi.origin, gut.origin,
                     gvt.origin, gw.origin, gp.origin, gh.origin, gr.origin, lfx.origin, lfx.s, ed2, dt, d, m.rows,
                     m.wx_log);
  } else {
    const int kb = tuned_kb(kKB);
    return launch<fastwavesuv_kernel<T>>(tile_grid(d.nx, d.ny, d.nz, kT, kT, kb), sizeof(FastwavesSmem<T>),
                                       (cudaStream_t)stream, gu.origin, gv.origin, gui.origin, gvi.origin, gut.origin,
                                       gvt.origin, gw.origin, gp.origin, gh.origin, gr.origin, lfx.origin, lfx.s, ed2,
                                       dt, d, kb);
  }
}

// Tangent-linear fastwavesuv with respect to (uin, vin, utens, vtens, ppuv); wgtfac, hhl,
// rho and fx are parameters.  The map is linear in these inputs, so this is also the
// forward stencil applied to the perturbation; it runs on Dual<T> like the others.
template <class T, class M3, class M1>
oeb_status fastwavesuv_tl_entry(const M3* duout, const M3* dvout, const M3* uin, const M3* vin, const M3* utens,
                                const M3* vtens, const M3* wgtfac, const M3* ppuv, const M3* hhl, const M3* rho,
                                const M1* fx, const M3* duin, const M3* dvin, const M3* dutens, const M3* dvtens,
                                const M3* dppuv, T edadlat, T dt, const oeb_domain* dom, void* stream) {
  {
    ValidateOnly guard;
    OEB_TRY(fastwavesuv_entry<T>(duout, dvout, uin, vin, utens, vtens, wgtfac, ppuv, hhl, rho, fx, edadlat, dt, dom,
                                 stream));
    OEB_TRY(fastwavesuv_entry<T>(duout, dvout, duin, dvin, dutens, dvtens, wgtfac, dppuv, hhl, rho, fx, edadlat, dt,
                                 dom, stream));
  }
  OEB_RETURN_IF_VALIDATING();
  using D = Dual<T>;
  DualIn<T> u, v, ut, vt, p;
  OEB_TRY((dual_in<T>(uin, duin, &u)));
  OEB_TRY((dual_in<T>(vin, dvin, &v)));
  OEB_TRY((dual_in<T>(utens, dutens, &ut)));
  OEB_TRY((dual_in<T>(vtens, dvtens, &vt)));
  OEB_TRY((dual_in<T>(ppuv, dppuv, &p)));
  const DualIn<T> w = dual_param<T>(wgtfac), h = dual_param<T>(hhl), r = dual_param<T>(rho), f = dual_param<T>(fx);
  const DualOut<T> ou = dual_out<T>(duout), ov = dual_out<T>(dvout);
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, uin->strides[1], uin->strides[0]};
  const D ed2 = D(T(2.0) * edadlat);
  const int kb = tuned_kb(kKB);
  return launch<fastwavesuv_kernel<D>>(tile_grid(d.nx, d.ny, d.nz, kT, kT, kb), sizeof(FastwavesSmem<D>),
                                        (cudaStream_t)stream, ou, ov, u, v, ut, vt, w, p, h, r, f, fx->strides[0], ed2,
                                        D(dt), d, kb);
}

// ============================== adjoint ===========================================
// fastwavesuv is linear in x = (uin, vin, utens, vtens, ppuv) for fixed wgtfac, hhl, rho, fx:
//   uout = uin + dt (utens - ppgu qx),  qx = 2 fx(j) / (rho(i+1) + rho(i))
//   ppgu = (ppuv(i+1) - ppuv(i)) + (ppgc(i+1) + ppgc(i)) gx,  gx = 0.5 Hs / Hd   (fastwavesuv.h:172-175)
//   ppgc(k) = ppgk(k+1) - ppgk(k),  ppgk(k) = w(k) ppuv(k) + (1 - w(k)) ppuv(k-1)
// and likewise in j.  Its transpose, written as gathers (no atomics), for ybar = (uoutb, voutb):
//   uinb = uoutb, utensb = dt uoutb (and v), and with au = -dt qx uoutb, av = -dt qy voutb,
//   cb(i,j,k)  = au(i) gx(i) + au(i-1) gx(i-1) + av(j) gy(j) + av(j-1) gy(j-1)     (ppgc adjoint)
//   kb(k)      = cb(k-1) - cb(k)                                                   (ppgk adjoint)
//   ppuvb(k)   = w(k) kb(k) + (1 - w(k+1)) kb(k+1) + au(i-1) - au(i) + av(j-1) - av(j)
// with every coefficient zero off the interior.  ppuvb covers i in [0,N], j in [0,N],
// k in [-1,N_z] (the reach of ppuv).  One CTA marches a 32 x 32 tile of that box through a
// chunk of k-levels, keeping cb at three levels in registers.
// The adjoint's coefficients at every interior point, once (pass 1): au = -dt qx uoutb and
// au gx, av = -dt qy voutb and av gy (each division once; the g-weighted term is 0 where a
// is).  The march (pass 2) reads them at the kb + 2 levels of its k-block instead of
// recomputing them there.
template <class T>
struct FastwavesAdjTerms {
  T *au, *ax, *av, *ay;  // in the layout of the state fields, 0 outside the interior unread
};

// What the terms are formed from.
template <class T>
struct FastwavesAdjState {
  const T *hhl, *rho, *fx;
  int64_t s1d;
  T ed2;
};

// The coefficients au = -dt qx uoutb and au gx at interior point o (fastwavesuv_adj_terms_kernel's
// expressions), and av, av gy with dir = sj.
template <class T, bool U>
__device__ __forceinline__ T fastwaves_adj_coef(const FastwavesAdjState<T>& st, const T* __restrict__ yb, int64_t o,
                                                int j, int64_t sj, int64_t sk, T dt, T* ag) {
  const int64_t s = U ? 1 : sj;
  const T q = U ? (T(2.0) * ld(st.fx + (int64_t)j * st.s1d)) / (ld(st.rho + o + 1) + ld(st.rho + o))
                : st.ed2 / (ld(st.rho + o + sj) + ld(st.rho + o));
  const T a = -(dt * q) * ld(yb + o);
  T g = T(0);
  if (a != T(0)) {
    const T hs0 = ld(st.hhl + o + sk) + ld(st.hhl + o), hs1 = ld(st.hhl + o + s + sk) + ld(st.hhl + o + s);
    const T hd0 = ld(st.hhl + o + sk) - ld(st.hhl + o), hd1 = ld(st.hhl + o + s + sk) - ld(st.hhl + o + s);
    g = a * ((T(0.5) * (hs0 - hs1)) / (hd0 + hd1));
  }
  *ag = g;
  return a;
}

template <class T>
struct fastwavesuv_adj_terms_kernel {
  // six CTAs an SM: 97.8 us a call at 128 x 128 x 80, five (43 registers) 99.6
  static constexpr int kMinCtas = std::is_same<T, F64i>::value ? 6 : 0;
  static constexpr int kStepOp = step_op<T>(kOpFwsAdjTerms);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, FastwavesAdjTerms<T> tm, FastwavesAdjState<T> st,
                                             const T* __restrict__ uoutb, const T* __restrict__ voutb, T dt, Dims d,
                                             int kb) {
    const int64_t sk = d.sk, sj = d.sj;
    for_box<RowUnroll<T>::value>(blk, d, 0, 0, d.nx, d.ny, kb, [&](int64_t o, int, int j) {
      tm.au[o] = fastwaves_adj_coef<T, true>(st, uoutb, o, j, sj, sk, dt, &tm.ax[o]);
      tm.av[o] = fastwaves_adj_coef<T, false>(st, voutb, o, j, sj, sk, dt, &tm.ay[o]);
    });
  }
};

constexpr int kAdjJ = 8;  // rows of the transpose's tile: one cell a thread

// The transpose from the terms, a thread a cell of the box [0, nx] x [0, ny] and kb output levels: at level L a cell reads the eight terms that reach it, its own and those of the cells before it
// in i and j (L1 serves the neighbours), and keeps the two levels of cb behind it in registers.
//
// What bounds it: the FP64 pipe (13 additions an output level, the cb of the chunk's two outer levels
// among them) and the latency of the terms' loads.  FP64 adjoint at 128 x 128 x 80: 102 us (tiles of 16
// rows 109, of 32 rows, fewer blocks and so shorter ones, 121; the shared-memory tile of the terms it
// replaces, which added half as many cells again at the box's far edges, 144); at 64 x 64 x 60 36 us,
// was 72.
template <class T>
struct fastwavesuv_adj_kernel {
  static constexpr bool kAnyGrid = true;
  static constexpr int kStepOp = step_op<T>(kOpFwsAdj);  // the step kernel's id
  static __device__ __forceinline__ void run(const uint3& blk, T* __restrict__ uinb, T* __restrict__ vinb,
                                             T* __restrict__ utensb, T* __restrict__ vtensb, T* __restrict__ ppuvb,
                                             const T* __restrict__ wgtfac, FastwavesAdjTerms<T> tm,
                                             const T* __restrict__ uoutb, const T* __restrict__ voutb, T dt, Dims d, int kb) {
    const int i0 = (int)blk.x * kT, j0 = (int)blk.y * kAdjJ, sj = (int)d.sj;
    const int64_t sk = d.sk;
    // output levels K in [Ks, Ke) of the extended range [-1, nz+1)
    const int Ks = -1 + (int)blk.z * kb, Ke = min(Ks + kb, d.nz + 1);
    const TileCells t(d.nx + 1 - i0, min(d.ny + 1 - j0, kAdjJ));
    if (t.r0 < t.rows) {  // a cell a thread
      const int i = i0 + t.c, j = j0 + t.r0;
      const bool own = i < d.nx && j < d.ny, west = i > 0 && j < d.ny, south = j > 0 && i < d.nx;
      int64_t o = (int64_t)(Ks - 1) * sk + i + j * sj;
      T cm1 = T(0), kbK = T(0), dir = T(0);  // cb(L-1), kb(L-1) = cb(L-2) - cb(L-1), direct terms of level L-1
#pragma unroll 1
      for (int L = Ks - 1; L <= Ke; ++L, o += sk) {
        const bool in_k = L >= 0 && L < d.nz;
        const bool p = in_k && own, w = in_k && west, q = in_k && south;
        // cb(L) at (i, j): ppgc(i) feeds ppgu(i), ppgu(i-1), ppgv(j), ppgv(j-1)
        const T x0 = p ? ld(tm.ax + o) : T(0), x1 = w ? ld(tm.ax + o - 1) : T(0);
        const T y0 = p ? ld(tm.ay + o) : T(0), y1 = q ? ld(tm.ay + o - sj) : T(0);
        const T cl = (x0 + x1) + (y0 + y1);
        const T kbL = cm1 - cl;
        if (L > Ks) {
          const int K = L - 1;  // output level
          const int64_t oK = o - sk;
          T acc = dir;
          if (K >= 0) acc = acc + ld(wgtfac + oK) * kbK;
          if (K + 1 <= d.nz) acc = acc + (T(1.0) - ld(wgtfac + o)) * kbL;
          ppuvb[oK] = acc;
          if (K >= 0 && K < d.nz && own) {
            const T ub = ld(uoutb + oK), vb = ld(voutb + oK);
            uinb[oK] = ub;
            vinb[oK] = vb;
            utensb[oK] = dt * ub;
            vtensb[oK] = dt * vb;
          }
        }
        if (L >= Ks && L < Ke) {
          // direct terms of level L: au(i-1) - au(i) + av(j-1) - av(j)
          const T u0 = p ? ld(tm.au + o) : T(0), u1 = w ? ld(tm.au + o - 1) : T(0);
          const T v0 = p ? ld(tm.av + o) : T(0), v1 = q ? ld(tm.av + o - sj) : T(0);
          dir = (u1 - u0) + (v1 - v0);
        }
        cm1 = cl;
        kbK = kbL;
      }
    }
  }
};

// FP32, marching levels: a warp owns 30 columns (lane = i0 - 1 + lane) and R rows of the box
// [0, nx] x [0, ny], and marches up a chunk of levels.  At level L every lane forms au, au gx of its R
// rows and av, av gy of those and the row below; the lane below hands over au(i-1), and the
// three-level window of cb stays in registers, as do hhl and wgtfac of the level before.  Nothing
// waits on a barrier.  fastwavesuv_adj_kernel's operations on the same operands in the same order: the
// same bits.
//
// What bounds it: DRAM at large domains (0.47 of the HBM copy rate over the ten fields it must move at
// 256 x 256 x 80) and issue, its divisions first.  One row a warp, four CTAs an SM: 22.5 us at
// 128 x 128 x 80, 66.2 at 256 x 256 x 80, 31.6 at 201 x 173 x 61 (two rows and three CTAs 27.0 / 83.3 /
// 39.9, three rows and two CTAs 24.4 / 64.8 / 33.2: fewer coefficients twice, but fewer warps); the
// shared-memory march of fastwavesuv_adj_kernel that formed its coefficients itself took 73.0, 161.6
// and 76.3 us.
struct fastwavesuv_adj_march_f32 {
  static constexpr bool kAnyGrid = true;
  static constexpr int kStepOp = step_op<float>(kOpFwsAdjFused);  // the step kernel's id
  static constexpr int R = 1, kCols = 30, kMinCtas = 4;
  // level L: hhl at L + 1 and rho on rows ja - 1 .. ja + R, voutb on ja - 1 .. ja + R - 1, uoutb and
  // wgtfac on ja .. ja + R - 1
  struct Level {
    float h[R + 2], r[R + 2], yv[R + 1], yu[R], w[R];
  };
  static __device__ __forceinline__ void run(const uint3& blk, float* __restrict__ uinb, float* __restrict__ vinb,
                                             float* __restrict__ utensb, float* __restrict__ vtensb,
                                             float* __restrict__ ppuvb, const float* __restrict__ wgtfac,
                                             FastwavesAdjState<float> st, const float* __restrict__ uoutb,
                                             const float* __restrict__ voutb, float dt, Dims d, int kb) {
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    const int i0 = (int)blk.x * kCols, ja = ((int)blk.y * kTY + (int)threadIdx.y) * R;
    if (ja > ny) return;
    const int lane = (int)threadIdx.x, i = i0 - 1 + lane, ic = max(0, min(i, nx));
    const bool own = lane >= 1 && lane <= kCols && i <= nx, in_i = i >= 0 && i < nx;
    const int Ks = -1 + (int)blk.z * kb, Ke = min(Ks + kb, nz + 1);
    const int64_t sjb = d.sj * 4, skb = d.sk * 4;
    // offsets of rows ja - 1 .. ja + R (clamped to the fields) at level 0
    int64_t row[R + 2];
    float fx2[R];
#pragma unroll
    for (int b = 0; b < R + 2; ++b) row[b] = ((int64_t)max(0, min(ja - 1 + b, ny)) * d.sj + ic) * 4;
#pragma unroll
    for (int b = 0; b < R; ++b) fx2[b] = 2.f * ld(st.fx + (int64_t)min(ja + b, ny - 1) * st.s1d);
    auto in_j = [&](int j) { return j >= 0 && j < ny; };
    // hhl at the chunk's first level, wgtfac one level below
    float h0[R + 2], w0[R];
#pragma unroll
    for (int b = 0; b < R + 2; ++b) h0[b] = get(st.hhl, row[b] + (int64_t)max(0, Ks - 1) * skb);
#pragma unroll
    for (int b = 0; b < R; ++b) w0[b] = 0.f;
    Level n;
    auto fetch = [&](int L) {
      const int64_t k = (int64_t)L * skb;
      if (L >= 0 && L < nz) {
#pragma unroll
        for (int b = 0; b < R + 2; ++b) n.h[b] = get(st.hhl, row[b] + k + skb), n.r[b] = get(st.rho, row[b] + k);
#pragma unroll
        for (int b = 0; b < R + 1; ++b) n.yv[b] = (in_i && in_j(ja - 1 + b)) ? get(voutb, row[b] + k) : 0.f;
#pragma unroll
        for (int b = 0; b < R; ++b) n.yu[b] = (in_i && in_j(ja + b)) ? get(uoutb, row[b + 1] + k) : 0.f;
      }
      if (L >= 0 && L <= nz) {
#pragma unroll
        for (int b = 0; b < R; ++b) n.w[b] = get(wgtfac, row[b + 1] + k);
      }
    };
    n = Level{};
    fetch(Ks - 1);
    float cm2[R], cm1[R], dir[R], yu0[R], yv0[R];
#pragma unroll
    for (int b = 0; b < R; ++b) cm2[b] = cm1[b] = dir[b] = yu0[b] = yv0[b] = 0.f;
#pragma unroll 1
    for (int L = Ks - 1; L <= Ke; ++L) {
      const Level c = n;
      if (L < Ke) fetch(L + 1);
      const bool in_l = L >= 0 && L < nz;
      float au[R], ax[R], av[R + 1], ay[R + 1], aum[R], axm[R];
#pragma unroll
      for (int b = 0; b < R + 1; ++b) {
        av[b] = ay[b] = 0.f;
        if (b < R) au[b] = ax[b] = aum[b] = axm[b] = 0.f;
      }
      if (in_l) {
        // the hhl sums and differences and rho of the rows, and of the lane above for the R rows
        float hs[R + 2], hd[R + 2];
#pragma unroll
        for (int b = 0; b < R + 2; ++b) hs[b] = c.h[b] + h0[b], hd[b] = c.h[b] - h0[b], h0[b] = c.h[b];
#pragma unroll
        for (int b = 0; b < R + 1; ++b) {
          const bool ok = in_i && in_j(ja - 1 + b);
          const float q = st.ed2 / (c.r[b + 1] + c.r[b]);
          const float a = -(dt * q) * c.yv[b];
          const float g = numerator(ok, 0.5f * (hs[b] - hs[b + 1])) / (hd[b] + hd[b + 1]);
          av[b] = ok ? a : 0.f;
          ay[b] = ok && a != 0.f ? a * g : 0.f;
        }
#pragma unroll
        for (int b = 0; b < R; ++b) {
          const bool ok = in_i && in_j(ja + b);
          const float hsn = lane_above<1>(hs[b + 1]), hdn = lane_above<1>(hd[b + 1]), rn = lane_above<1>(c.r[b + 1]);
          const float q = fx2[b] / (rn + c.r[b + 1]);
          const float a = -(dt * q) * c.yu[b];
          const float g = numerator(ok, 0.5f * (hs[b + 1] - hsn)) / (hd[b + 1] + hdn);
          au[b] = ok ? a : 0.f;
          ax[b] = ok && a != 0.f ? a * g : 0.f;
          aum[b] = lane_below<1>(au[b]), axm[b] = lane_below<1>(ax[b]);
        }
      }
      const int K = L - 1;
#pragma unroll
      for (int b = 0; b < R; ++b) {
        const float cl = in_l ? ((ax[b] + axm[b]) + (ay[b + 1] + ay[b])) : 0.f;
        if (K >= Ks && own && ja + b <= ny) {
          const int64_t o = row[b + 1] + (int64_t)K * skb;
          const float kbK = cm2[b] - cm1[b], kbK1 = cm1[b] - cl;
          float acc = dir[b];
          if (K >= 0) acc = acc + w0[b] * kbK;
          if (K + 1 <= nz) acc = acc + (1.f - c.w[b]) * kbK1;
          put(ppuvb, o, acc);
          if (K >= 0 && K < nz && in_i && ja + b < ny) {
            put(uinb, o, yu0[b]);
            put(vinb, o, yv0[b]);
            put(utensb, o, dt * yu0[b]);
            put(vtensb, o, dt * yv0[b]);
          }
        }
        dir[b] = (aum[b] - au[b]) + (av[b] - av[b + 1]);
        cm2[b] = cm1[b], cm1[b] = cl;
        yu0[b] = c.yu[b], yv0[b] = c.yv[b + 1], w0[b] = c.w[b];
      }
    }
  }
};

template <class T, class M3, class M1>
oeb_status fastwavesuv_adj_entry(const M3* uinb, const M3* vinb, const M3* utensb, const M3* vtensb,
                                 const M3* ppuvb, const M3* uin, const M3* vin, const M3* utens, const M3* vtens,
                                 const M3* wgtfac, const M3* ppuv, const M3* hhl, const M3* rho, const M1* fx,
                                 const M3* uoutb, const M3* voutb, T edadlat, T dt, const oeb_domain* dom,
                                 void* stream) {
  {
    // the state as the forward sees it, with the adjoint seeds in the outputs' places
    ValidateOnly guard;
    OEB_TRY(fastwavesuv_entry<T>(uoutb, voutb, uin, vin, utens, vtens, wgtfac, ppuv, hhl, rho, fx, edadlat, dt, dom,
                                 stream));
  }
  OEB_TRY(check_domain(dom));
  Grid<T> gub, gvb, gutb, gvtb, gpb, gw, gh, gr, guo, gvo;
  Line<T> lfx;
  OEB_TRY((check_field3<T>(uinb, *dom, kInterior, &gub)));
  OEB_TRY((check_field3<T>(vinb, *dom, kInterior, &gvb)));
  OEB_TRY((check_field3<T>(utensb, *dom, kInterior, &gutb)));
  OEB_TRY((check_field3<T>(vtensb, *dom, kInterior, &gvtb)));
  OEB_TRY((check_field3<T>(ppuvb, *dom, Reach{0, 1, 0, 1, 1, 1}, &gpb)));
  OEB_TRY((check_field3<T>(wgtfac, *dom, Reach{0, 1, 0, 1, 0, 1}, &gw)));
  OEB_TRY((check_field3<T>(hhl, *dom, Reach{0, 1, 0, 1, 0, 1}, &gh)));
  OEB_TRY((check_field3<T>(rho, *dom, Reach{0, 1, 0, 1, 0, 0}, &gr)));
  OEB_TRY((check_field3<T>(uoutb, *dom, kInterior, &guo)));
  OEB_TRY((check_field3<T>(voutb, *dom, kInterior, &gvo)));
  OEB_TRY((check_field1<T>(fx, *dom, 0, 0, &lfx)));
  OEB_TRY(check_same_strides<T>({&gub, &gvb, &gutb, &gvtb, &gpb, &gw, &gh, &gr, &guo, &gvo}));
  OEB_TRY(check_no_alias({gub.lo, gub.hi, gvb.lo, gvb.hi, gutb.lo, gutb.hi, gvtb.lo, gvtb.hi, gpb.lo, gpb.hi},
                         {gw.lo, gw.hi, gh.lo, gh.hi, gr.lo, gr.hi, guo.lo, guo.hi, gvo.lo, gvo.hi, lfx.lo, lfx.hi}));
  OEB_RETURN_IF_VALIDATING();
  const Dims d{(int)dom->nx, (int)dom->ny, (int)dom->nz, gw.sj, gw.sk};
  const T ed2 = T(2.0) * edadlat;
  cudaStream_t st = (cudaStream_t)stream;
  const FastwavesAdjState<T> state{gh.origin, gr.origin, lfx.origin, lfx.s, ed2};
  if constexpr (std::is_same<T, float>::value) if (adjoint_tiles()) {
    // one launch: the march forms the coefficients at the kb + 2 levels of its k-block
    using B = fastwavesuv_adj_march_f32;
    const int gx = (d.nx + B::kCols) / B::kCols, gy = (d.ny + kTY * B::R) / (kTY * B::R);
    const int kb = tuned_levels(march_levels(gx * gy, d.nz + 2, B::kMinCtas));
    return launch<B>(dim3((unsigned)gx, (unsigned)gy, (unsigned)((d.nz + 1 + kb) / kb)), 0, st, gub.origin, gvb.origin,
                     gutb.origin, gvtb.origin, gpb.origin, gw.origin, state, guo.origin, gvo.origin, dt, d, kb);
  }
  // scratch for the four coefficient fields, in uoutb's layout
  const T* start = (uoutb->allocated && uoutb->allocated <= uoutb->aligned) ? uoutb->allocated : uoutb->aligned;
  const int64_t last = (uoutb->sizes[0] - 1) * uoutb->strides[0] + (uoutb->sizes[1] - 1) * uoutb->strides[1] +
                       (uoutb->sizes[2] - 1) * uoutb->strides[2];
  const int64_t n = (int64_t)(uoutb->aligned - start) + last + 1;
  const int64_t org = (int64_t)(uoutb->aligned - start) + uoutb->offset;
  void* buf = nullptr;
  OEB_TRY(scratch_alloc(&buf, (size_t)n * 4 * sizeof(T), st));
  T* base = static_cast<T*>(buf);
  const FastwavesAdjTerms<T> tm{base + org, base + n + org, base + 2 * n + org, base + 3 * n + org};
  Dims dp = d;
  dp.tj = point_rows<T>(tile_grid(d.nx, d.ny, d.nz, kT, kT, 1), kDerivativeTiles);
  oeb_status stt = launch<fastwavesuv_adj_terms_kernel<T>>(tile_grid(d.nx, d.ny, d.nz, kT, dp.tj, 1), 0, st, tm, state,
                                                           guo.origin, gvo.origin, dt, dp, 1);
  // a block of kb levels reads the terms of kb + 2: about one wave of blocks, five CTAs an SM (three
  // 114 us at 128 x 128 x 80 and 322 at 256 x 256 x 80, eight 104 and 329, five 102 and 329)
  const dim3 cells = tile_grid(d.nx + 1, d.ny + 1, 1, kT, kAdjJ, 1);
  const int kb = tuned_levels(march_levels((int)(cells.x * cells.y), d.nz + 2, 5));
  if (stt == OEB_OK)
    stt = launch<fastwavesuv_adj_kernel<T>>(tile_grid(d.nx + 1, d.ny + 1, d.nz + 2, kT, kAdjJ, kb),
                                            0, st, gub.origin, gvb.origin, gutb.origin,
                                            gvtb.origin, gpb.origin, gw.origin, tm, guo.origin, gvo.origin, dt,
                                            d, kb);
  scratch_free(buf, st);
  return stt;
}

}  // namespace
}  // namespace oeb

#ifndef OEB_BODIES_ONLY  // the entry points

using namespace oeb;

#define OEB_FW_ENTRY(S, T)                                                                                          \
  extern "C" oeb_status oeb_fastwavesuv_##S(                                                                       \
      const oeb_memref3d_##S* uout, const oeb_memref3d_##S* vout, const oeb_memref3d_##S* uin,                      \
      const oeb_memref3d_##S* vin, const oeb_memref3d_##S* utens, const oeb_memref3d_##S* vtens,                    \
      const oeb_memref3d_##S* wgtfac, const oeb_memref3d_##S* ppuv, const oeb_memref3d_##S* hhl,                    \
      const oeb_memref3d_##S* rho, const oeb_memref1d_##S* fx, T edadlat, T dt, const oeb_domain* dom,             \
      void* stream) {                                                                                              \
    return fastwavesuv_entry<T>(uout, vout, uin, vin, utens, vtens, wgtfac, ppuv, hhl, rho, fx, edadlat, dt, dom,  \
                                stream);                                                                           \
  }                                                                                                                \
  extern "C" oeb_status oeb_fastwavesuv_tl_##S(                                                                    \
      const oeb_memref3d_##S* duout, const oeb_memref3d_##S* dvout, const oeb_memref3d_##S* uin,                    \
      const oeb_memref3d_##S* vin, const oeb_memref3d_##S* utens, const oeb_memref3d_##S* vtens,                    \
      const oeb_memref3d_##S* wgtfac, const oeb_memref3d_##S* ppuv, const oeb_memref3d_##S* hhl,                    \
      const oeb_memref3d_##S* rho, const oeb_memref1d_##S* fx, const oeb_memref3d_##S* duin,                        \
      const oeb_memref3d_##S* dvin, const oeb_memref3d_##S* dutens, const oeb_memref3d_##S* dvtens,                 \
      const oeb_memref3d_##S* dppuv, T edadlat, T dt, const oeb_domain* dom, void* stream) {                        \
    return fastwavesuv_tl_entry<T>(duout, dvout, uin, vin, utens, vtens, wgtfac, ppuv, hhl, rho, fx, duin, dvin,    \
                                   dutens, dvtens, dppuv, edadlat, dt, dom, stream);                               \
  }                                                                                                                \
  extern "C" oeb_status oeb_fastwavesuv_adj_##S(                                                                   \
      const oeb_memref3d_##S* uinb, const oeb_memref3d_##S* vinb, const oeb_memref3d_##S* utensb,                   \
      const oeb_memref3d_##S* vtensb, const oeb_memref3d_##S* ppuvb, const oeb_memref3d_##S* uin,                   \
      const oeb_memref3d_##S* vin, const oeb_memref3d_##S* utens, const oeb_memref3d_##S* vtens,                    \
      const oeb_memref3d_##S* wgtfac, const oeb_memref3d_##S* ppuv, const oeb_memref3d_##S* hhl,                    \
      const oeb_memref3d_##S* rho, const oeb_memref1d_##S* fx, const oeb_memref3d_##S* uoutb,                       \
      const oeb_memref3d_##S* voutb, T edadlat, T dt, const oeb_domain* dom, void* stream) {                        \
    return fastwavesuv_adj_entry<T>(uinb, vinb, utensb, vtensb, ppuvb, uin, vin, utens, vtens, wgtfac, ppuv, hhl,   \
                                    rho, fx, uoutb, voutb, edadlat, dt, dom, stream);                              \
  }

OEB_FW_ENTRY(f64, double)
OEB_FW_ENTRY(f32, float)

#endif  // OEB_BODIES_ONLY
