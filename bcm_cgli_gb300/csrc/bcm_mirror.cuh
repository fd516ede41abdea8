// FP32 mirror of the state for the split-precision path.
//
// The split kernels read the state as FP32 deltas from each case's reference
// state (rho0, 0, 0, 0, P0/(K-1)), rounded to nearest even from the FP64
// values.  Two buffers hold it: during an RK stage the flux kernel reads the
// current buffer (the halo of its tile belongs to other CTAs, which update
// their cells during the launch) and writes the deltas of its own cells
// into the other one, which is the current one from the next launch on (a
// launch argument within a step, a device flag across them).  Every other kernel that writes the FP64 state (boundary
// fill, IBM ghost cells, interface copies, edge fill, LU-SGS update) writes
// the same cells of the current buffer too, so the mirror stays the exact
// rounding of the state without a pass over all cells each stage.
#pragma once

#include <cuda_runtime.h>

#include "bcm_common.cuh"

namespace bcmg {

#ifdef __CUDACC__
// double -> float, round to nearest even (IEEE 754), and float -> double on the
// integer pipes: this part's FP64 pipe, where the hardware conversions run, is
// its narrowest (12 and 8 integer instructions against a slot of 73 cycles a
// warp).  Operands outside the normal float range other than zero go through
// calls: inlined, the hardware conversion is predicated instead of branched
// around and takes its FP64 slot every time.
static __device__ __noinline__ float to_float_rare(double x) { return __double2float_rn(x); }
static __device__ __noinline__ double to_double_rare(float f) { return (double)f; }
__device__ __forceinline__ float to_float_int(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const bool zero = ((hi << 1) | lo) == 0;
  const int e = (int)((hi >> 20) & 0x7FF) - 896;  // float exponent field
  if (!zero && (unsigned)(e - 1) >= 254u) return to_float_rare(x);
  const unsigned m = __funnelshift_l(lo, hi & 0xFFFFFu, 3);  // top 23 fraction bits
  const unsigned up = ((lo & 0x1FFFFFFFu) + 0x0FFFFFFFu + (m & 1u)) >> 29;
  const unsigned r = ((unsigned)e << 23) + m + up;  // a carry may raise the exponent
  return __uint_as_float((hi & 0x80000000u) | (zero ? 0u : r));
}
__device__ __forceinline__ double to_double_int(float f) {
  const unsigned b = __float_as_uint(f), a = b & 0x7FFFFFFFu;
  if (a - 1u < 0x007FFFFFu || a >= 0x7F800000u) return to_double_rare(f);  // subnormal, inf, nan
  const unsigned hi = a == 0 ? 0u : (a >> 3) + (896u << 20);
  return __hiloint2double((int)((b & 0x80000000u) | hi), (int)(b << 29));
}

// Mirror value of component v (0..4) of a state cell: density and energy as
// deltas from rho0 and E0 = P0/(K-1), momenta as they are; rounded once.
__device__ __forceinline__ float mirror_value(double x, int v, double rho0, double E0) {
  return to_float_int(v == 0 ? x - rho0 : (v == 4 ? x - E0 : x));
}
#endif  // __CUDACC__

// The two mirror buffers, the device flag naming the current one, and the
// reference state of a single case (batches take each cube's case).
// buf[0] == nullptr: no mirror (the FP64 path); kernels then skip it.
struct Mirror {
  float *buf[2] = {nullptr, nullptr};
  const int *parity = nullptr;  // device [1]: index of the current buffer ...
  int phase = 0;                // ... at the last launch of k_mirror_flip; 1: the other one now
  double rho0 = 0, E0 = 0;
};

#ifdef __CUDACC__
__device__ __forceinline__ int mirror_index(const Mirror &m) { return *m.parity ^ m.phase; }
// (a select, not m.buf[mirror_index(m)]: indexing a kernel argument's array with
// a run-time value would copy the argument to local memory)
__device__ __forceinline__ float *mirror_current(const Mirror &m) {
  return m.buf[0] ? (mirror_index(m) ? m.buf[1] : m.buf[0]) : nullptr;
}
#endif

}  // namespace bcmg
