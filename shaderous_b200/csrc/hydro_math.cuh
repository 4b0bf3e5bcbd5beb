// What every pass of the hydro step shares: the kernels' parameters, the device clock, primitives and
// signal rate of a cell, the predictor's result and the boundary mapping. The scheme's arithmetic is in
// sweep_math.cuh (uniform sweeps) and block_math.cuh (block passes). Each function states the
// reference function it follows; the reference's CPU scheme is src/reference/hydro.ts, its shaders
// src/hydro/*.wgsl.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace shz {

enum Recon { R_MINMOD = 0, R_MC = 1, R_VANLEER = 2, R_KOREN = 3, R_PPM = 4 };

// Kernel parameters, passed by value.
struct KParams {
  double dx;  // cell size
  int n[3];
  int bc_lo[3], bc_hi[3];
  float gamma, gm1, inv_gm1, inv_gamma;
  float rho_floor, p_floor, e_floor;
  float eta_dual, shock_thresh, signal;
  int hll;
  double dv;  // cell volume dx^ndim in float64 (the float64 totals are scaled by it)
};

// The clock on the device (the reference's Clock, src/hydro/common.wgsl:84-96), advanced by
// each step (step_clock, clock_multi_kernel): t is the time of the state the sweep in flight produces.
struct DevClock {
  double t;
  double dt;
  double t_end;
  double dt_max;
  double cfl_dx;
  double last_dt;
  long long steps;
  long long max_steps;  // the clock holds once this many steps are taken (a batched request's length)
  int held;
  int bad;
};

// The per-cell result of the predictor (hydro.ts:272-322 predictRaw): the half-step state q,
// the shock flag and the first-order flag.
struct Pred {
  float q[6];
  float flag;
  bool fo;
};

// The shock detector's pressure jump along one axis (hydro.ts:300-303: |p+ - p-| / min(p+, p-)
// above the threshold), as its excess over the threshold: |p+ - p-| - threshold min(p+, p-), which
// is positive exactly where the ratio exceeds it (the pressures are floored, so positive), without
// the division. The largest over the axes decides.
__device__ __forceinline__ float jump_excess(float pm, float pp, float thresh) {
  return fabsf(pp - pm) - thresh * fminf(pp, pm);
}

// Primitives of one cell from its conserved state (hydro.ts:233-257 primitives; prim.wgsl:26-51):
// (rho, vx, vy, vz, p, s, cs), velocities multiplied by the boundary signs f.
__device__ __forceinline__ void prim_from_cons(const float4 a, const float4 b, const KParams& P, float fx, float fy,
                                               float fz, float* w) {
  const float rho = fmaxf(a.x, P.rho_floor);
  const float inv = 1.f / rho;
  float p = P.gm1 * b.y;
  if (!(p >= P.p_floor)) p = P.p_floor;
  w[0] = rho;
  w[1] = a.y * inv * fx;
  w[2] = a.z * inv * fy;
  w[3] = a.w * inv * fz;
  w[4] = p;
  w[5] = b.z * inv;
  w[6] = sqrtf(P.gamma * p * inv);
}

// The six primitives the stencil reads of a neighbour (rho, vx, vy, vz, p, s): the sound
// speed is needed only at the centre cell and is formed there (with_cs).
__device__ __forceinline__ void prim6_from_cons(const float4 a, const float4 b, const KParams& P, float fx, float fy,
                                                float fz, float* w) {
  const float rho = fmaxf(a.x, P.rho_floor);
  const float inv = 1.f / rho;
  float p = P.gm1 * b.y;
  if (!(p >= P.p_floor)) p = P.p_floor;
  w[0] = rho;
  w[1] = a.y * inv * fx;
  w[2] = a.z * inv * fy;
  w[3] = a.w * inv * fz;
  w[4] = p;
  w[5] = b.z * inv;
}
__device__ __forceinline__ void with_cs(float* w, const KParams& P) { w[6] = sqrtf(P.gamma * w[4] / w[0]); }

// The signal rate of a cell (hydro.ts:254): |vx| + |vy| + |vz| + signal * cs.
__device__ __forceinline__ float signal_rate(const float4 a, const float4 b, const KParams& P) {
  float w[7];
  prim_from_cons(a, b, P, 1.f, 1.f, 1.f, w);
  return fabsf(w[1]) + fabsf(w[2]) + fabsf(w[3]) + P.signal * w[6];
}

// hydro.ts:216-220 bcAxis: the source index of a possibly out-of-range index and the sign of
// the velocity along that axis. Indices beyond the reach of the scheme are clamped into range
// (they feed no output).
// Boundary codes: 0 periodic, 1 outflow, 2 reflect (the reference's), and 3 halo: a z face of one
// slab of a larger grid, whose ghost planes are stored beyond the slab and filled by the caller
// with the neighbouring slab's planes.
constexpr int BC_HALO = 3;
// Whether a face's ghosts take the adjacent inner cell's half step (outflow and reflect).
__host__ __device__ __forceinline__ bool bc_inner(int code) { return code == 1 || code == 2; }

__device__ __forceinline__ int bc_map(int i, int n, int lo, int hi, float& f) {
  f = 1.f;
  if (i < 0) {
    if (lo == 0) i = ((i % n) + n) % n;
    else if (lo == 1) i = 0;
    else { i = -1 - i; f = -1.f; }
  } else if (i >= n) {
    if (hi == 0) i = i % n;
    else if (hi == 1) i = n - 1;
    else { i = 2 * n - 1 - i; f = -1.f; }
  }
  return min(max(i, 0), n - 1);
}

}  // namespace shz
