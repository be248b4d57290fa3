// The amplitude types: float2 / double2, interleaved (re, im).  No host
// headers: the run-time compiled pass kernels include it too.
#pragma once

namespace vqc {

template <class R>
struct CT;
template <>
struct CT<float> {
  using T = float2;
};
template <>
struct CT<double> {
  using T = double2;
};
template <class R>
using cplx = typename CT<R>::T;

template <class R>
__host__ __device__ __forceinline__ cplx<R> mkc(R a, R b) {
  cplx<R> r;
  r.x = a;
  r.y = b;
  return r;
}

}  // namespace vqc
