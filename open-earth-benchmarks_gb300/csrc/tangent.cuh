// tangent.cuh -- running a stencil kernel on dual numbers: the tangent-linear entry points.
//
// oeb_<k>_tl_<f64|f32>(dy..., x..., dx..., scalars) computes dy = J(x) dx, the stencil's
// Jacobian at the state x applied to the perturbation dx of its active inputs, with every
// branch frozen at x.  The kernel is the forward kernel instantiated with Dual<T>: it reads a
// value from x and its derivative from dx at the same offset (zero for a parameter, DualIn in
// dual.cuh) and writes the derivatives to dy (DualOut), so a call is the forward kernel's
// launches and nothing else.  Packing every field into an array of (value, derivative) pairs
// first, and copying the derivatives out after, took longer than the kernels: in FP32 at
// 128 x 128 x 80 hdiffsmag 60.7 -> 33.0 us, hadvuv5th 56.2 -> 31.4, fastwavesuv 111.1 -> 46.4,
// fvtp2d 175.1 -> 77.5, uvbke 48.4 -> 14.3, p_grad_c 80.9 -> 25.2 without it.
#pragma once

#include "dual.cuh"
#include "oeb_common.cuh"
#include "stencil_util.cuh"

namespace oeb {

// The dual field of state field `x` with perturbation `dx` (null: a parameter).  The two must share
// their layout.
template <class T, class M>
oeb_status dual_in(const M* x, const M* dx, DualIn<T>* out) {
  if (dx) {
    for (size_t r = 0; r < sizeof(x->sizes) / sizeof(x->sizes[0]); ++r)
      if (dx->sizes[r] != x->sizes[r] || dx->strides[r] != x->strides[r]) return OEB_ERR_LAYOUT;
    if (dx->offset != x->offset || (dx->aligned - dx->allocated) != (x->aligned - x->allocated)) return OEB_ERR_LAYOUT;
  }
  *out = DualIn<T>{x->aligned + x->offset, dx ? dx->aligned + dx->offset : nullptr};
  return OEB_OK;
}
template <class T, class M>
DualIn<T> dual_param(const M* x) {
  return DualIn<T>{x->aligned + x->offset, nullptr};
}
// The output whose derivatives go to `dy`.
template <class T, class M>
DualOut<T> dual_out(const M* dy) {
  return DualOut<T>{nullptr, dy->aligned + dy->offset};
}

}  // namespace oeb
