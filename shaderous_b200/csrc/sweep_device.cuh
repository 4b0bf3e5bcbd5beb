// Device helpers shared by the uniform sweeps (sweep.cu, sweep_rows.cu): the step's clock, block
// maxima, unpacking; and the host's launch of a step after a step.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "hydro_math.cuh"
#include "sweep.h"

namespace shz {

__device__ __forceinline__ void unpack7(const float4 a, const float4 b, float* f) {
  f[0] = a.x;
  f[1] = a.y;
  f[2] = a.z;
  f[3] = a.w;
  f[4] = b.x;
  f[5] = b.y;
  f[6] = b.z;
}
__device__ __forceinline__ void unpack8(const float4 a, const float4 b, float* f) {
  unpack7(a, b, f);
  f[7] = b.w;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block maximum of a non-negative rate into *out (as the float's bits: non-negative floats
// order as unsigned integers). fmaxf drops NaN operands, so rate_guard carries a NaN rate as
// +inf, which orders above every finite rate and which the clock reports.
template <int NT>
__device__ __forceinline__ void block_max_to(float v, float* sRed, unsigned* out) {
  v = warp_max(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) sRed[warp] = v;
  __syncthreads();
  if (warp == 0) {
    constexpr int NW = (NT + 31) / 32;
    float m = lane < NW ? sRed[lane] : 0.f;
    m = warp_max(m);
    if (lane == 0) atomicMax(out, __float_as_uint(m));
  }
}

__device__ __forceinline__ float rate_guard(float r) { return (r == r) ? r : __int_as_float(0x7f800000); }

// A cell's state as the last step left it. A sweep may be resident while that step still writes the state
// (launch_after), so the arrays are not constant for the kernel's life and its reads of them must not
// be taken for such (ld.global.nc, which __ldg is, and plain reads of const __restrict__ pointers may
// become): a coherent load, and volatile, so that none is moved ahead of step_clock's wait.
__device__ __forceinline__ float4 ld_state(const float4* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// The clock of a step, formed by every CTA: dt from the rate maximum that the last sweep (or
// rate_kernel) left (clock.wgsl:38-147, in the reference's CPU form hydro.ts:382
// dt = min(cfl dx / rate, t_end - t)). A rate that is NaN or infinite marks the clock bad and holds it.
// The grid's first thread writes the clock advanced by the step, in float64, to the other of the
// clock's two copies, and empties the rate slot that the next sweep folds into: nothing that a CTA
// of this launch reads is written in it, so a launch repeated in place gives the same clock and state.
// The wait comes first: everything read from here on may be the step before's output; then the
// step after may be launched (it waits likewise for this grid to end).
struct StepDt {
  double dt;
  bool held;
};
__device__ __forceinline__ StepDt step_clock(const ClockArgs& K) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const DevClock c = *K.in;
  const float rate = __uint_as_float(*K.rate);
  const bool bad = c.bad || !(rate == rate) || isinf(rate);
  double dt = fmin(c.cfl_dx / fmax((double)rate, 1e-30), c.dt_max);
  if (c.t_end < HUGE_VAL) {
    const double rem = c.t_end - c.t;
    dt = rem <= 1e-12 * fabs(c.t_end) ? 0.0 : fmin(dt, rem);
  }
  if (bad) dt = 0.0;
  const bool held = !(dt > 0.0);
  if (threadIdx.x == 0 && (blockIdx.x | blockIdx.y | blockIdx.z) == 0) {
    DevClock o = c;
    o.bad = bad ? 1 : 0;
    o.dt = dt;
    o.held = held ? 1 : 0;
    if (!held) {
      o.t = c.t + dt;
      o.steps = c.steps + 1;
      o.last_dt = dt;
    }
    *K.out = o;
    *K.rate_next = 0u;
  }
  return {dt, held};
}

// A launch that may begin before the kernel ahead of it in the stream has ended (programmatic stream
// serialization); step_clock waits for that kernel before anything is read.
template <typename... KA, typename... A>
static cudaError_t launch_after(void (*k)(KA...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k, KA(a)...);
}

}  // namespace shz
