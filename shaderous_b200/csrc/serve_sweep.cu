// The block sweep of served grids: every block of a batch lies on a uniform grid, so that a ghost is a
// same-level neighbour's cell or a boundary image, and no face is matched. The block sweep of the
// adaptive mesh (amr_sweep.cu) does the same with coarse and refined neighbours and per-block
// timesteps, in an arithmetic whose bits the meshes depend on (block_math.cuh). Here the uniform
// sweeps' arithmetic serves (sweep_math.cuh), and a block may be marched by several CTAs.
//
// A CTA takes `planes` planes of a block and marches them along z as the uniform sweep marches a
// column; the primitives, two ghost layers included, come from the atlas the assemble filled, three
// planes in shared memory, each staged by bulk copies (TMA) a plane ahead. Threads: 0 .. 255 the
// plane's cells, x fastest; then 16 a side: the ghosts below x, below y, above x, above y (the ring's
// corners feed no face). 10 warps at 96 registers: two CTAs per SM.
//
// Splitting a block costs two more planes a part, predicted only, and gives the same bits. It fills
// the SMs where a batch has few blocks: a march of 18 planes takes some 90 us however few blocks
// there are. A mix of six requests (99 blocks in 3D, 171 in 2D, 100 steps): 31.5 -> 23.3 ms, of which
// 15 are the steps (with the assemble's first pass split likewise).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "amr_device.cuh"
#include "launch_attr.h"
#include "sweep_math.cuh"
#include "tma.cuh"

namespace shz {
namespace gridsw {

using namespace amrk;

constexpr int SCELLS = BS * BS;        // threads of cells
constexpr int SNT = SCELLS + 4 * BS;   // 320 threads
constexpr int SWN = PAD * PAD;         // primitive texels per plane
constexpr int RING = 3;
constexpr int PLANE4 = 2 * SWN;        // float4 of a staged plane, w1 then w2
constexpr uint32_t PLANE_BYTES = SWN * sizeof(float4);
// in float4: the ring, x and y face states, x and y fluxes (also the half-step exchange), what a z
// boundary keeps, each thread's upper z face state, each cell's flux sums of the plane below
constexpr int S_RING = RING * PLANE4, S_FACE = 4 * SNT, S_FLUX = 4 * SNT, S_KEEP = 2 * SNT, S_ZUP = 2 * SNT, S_ACC = 2 * SCELLS;
constexpr size_t SMEM = (size_t)(S_RING + S_FACE + S_FLUX + S_KEEP + S_ZUP + S_ACC) * sizeof(float4);

// Eight floats a thread as two float4, entries tid and stride + tid.
__device__ __forceinline__ void put8(float4* a, int stride, int t, const float* v) {
  a[t] = make_float4(v[0], v[1], v[2], v[3]);
  a[stride + t] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void put7(float4* a, int stride, int t, const float* v) {
  a[t] = make_float4(v[0], v[1], v[2], v[3]);
  a[stride + t] = make_float4(v[4], v[5], v[6], 0.f);
}
__device__ __forceinline__ void get7(const float4* a, int stride, int t, float* v) {
  const float4 x = a[t], y = a[stride + t];
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  v[4] = y.x; v[5] = y.y; v[6] = y.z;
}
__device__ __forceinline__ void get8(const float4* a, int stride, int t, float* v) {
  get7(a, stride, t, v);
  v[7] = a[stride + t].w;
}
__device__ __forceinline__ void put_pred(float4* a, int stride, int t, const Pred& p) {
  a[t] = make_float4(p.q[0], p.q[1], p.q[2], p.q[3]);
  a[stride + t] = make_float4(p.q[4], p.q[5], p.flag, p.fo ? 1.f : 0.f);
}
__device__ __forceinline__ void get_pred(const float4* a, int stride, int t, Pred& p) {
  const float4 x = a[t], y = a[stride + t];
  p.q[0] = x.x; p.q[1] = x.y; p.q[2] = x.z; p.q[3] = x.w;
  p.q[4] = y.x; p.q[5] = y.y;
  p.flag = y.z;
  p.fo = y.w != 0.f;
}


// Texel (x, y) of a staged plane: its seven primitives (the sound speed as the atlas holds it).
__device__ __forceinline__ void read_w7(const float4* __restrict__ plane, int x, int y, float* w) {
  const int t = (y + NG) * PAD + (x + NG);
  const float4 a = plane[t], b = plane[SWN + t];
  w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
  w[4] = b.x; w[5] = b.y; w[6] = b.z;
}

template <int DIM, int R, bool ISEN>
__global__ void __maxnreg__(96)
    grid_sweep(const KParams* __restrict__ gp, const int* __restrict__ bt, const int* __restrict__ list, int n, int planes,
               const float4* __restrict__ u1, const float4* __restrict__ u2, const float4* __restrict__ w1,
               const float4* __restrict__ w2, float4* __restrict__ o1, float4* __restrict__ o2,
               const DevClock* __restrict__ clks, int* __restrict__ err) {
  extern __shared__ __align__(128) float4 smem[];
  float4* sW = smem;
  float4* sFace = sW + S_RING;
  float4* sFlux = sFace + S_FACE;
  float4* sKeep = sFlux + S_FLUX;
  float4* sZup = sKeep + S_KEEP;
  float4* sAcc = sZup + S_ZUP;
  __shared__ __align__(16) KParams sP;
  __shared__ __align__(8) uint64_t sBar[RING];
  const int tid = threadIdx.x;
  const bool tile_t = tid < SCELLS;
  const int side = tile_t ? -1 : (tid - SCELLS) / BS, along = tid % BS;  // ghosts: below x, below y, above x, above y
  const int lx = tile_t ? along : side == 0 ? -1 : side == 2 ? BS : along;
  const int ly = tile_t ? tid / BS : side == 1 ? -1 : side == 3 ? BS : along;
  const bool xface_t = tile_t || side == 2;  // solves the x face below lx
  const bool yface_t = tile_t || side == 3;
  // the threads of the texels below and above this one along x and y (those that solve or update)
  const int x_dn = lx == 0 ? SCELLS + ly : lx == BS ? ly * BS + BS - 1 : tid - 1;
  const int y_dn = ly == 0 ? SCELLS + BS + lx : ly == BS ? (BS - 1) * BS + lx : tid - BS;
  const int x_up = lx == BS - 1 ? SCELLS + 2 * BS + ly : tid + 1;
  const int y_up = ly == BS - 1 ? SCELLS + 3 * BS + lx : tid + BS;
  const int gface = side < 0 ? -1 : ((side & 1) << 1) + (side >> 1);
  const int g_in = gface == 0 ? ly * BS : gface == 1 ? ly * BS + BS - 1 : gface == 2 ? lx : (BS - 1) * BS + lx;
  auto ring = [&](int plane) -> float4* { return sW + (size_t)((plane + 3 * RING) % RING) * PLANE4; };
  // the phase each thread expects next of a slot's barrier (uniform across the CTA); copies in flight
  uint32_t phase = 0, pending = 0;
  if (tid == 0) {
    for (int s = 0; s < RING; s++) tma::mbar_init(&sBar[s], 1);
    tma::fence_mbar_init();
  }
  __syncthreads();

  const int parts = DIM == 3 ? BS / planes : 1;
  for (int i = blockIdx.x; i < n * parts; i += gridDim.x) {
    const int slot = __ldg(list + i / parts);
    const int z0 = DIM == 3 ? (i % parts) * planes : 0, z1 = DIM == 3 ? z0 + planes : 1;
    const int g = bt_at(bt, slot, GRID_WORD);
    const size_t base = (size_t)slot * BG<DIM>::CB;
    if (clks[g].held) {
      for (int t = z0 * SCELLS + tid; t < z1 * SCELLS; t += SNT) {
        o1[base + t] = __ldg(u1 + base + t);
        o2[base + t] = __ldg(u2 + base + t);
      }
      continue;
    }
    __syncthreads();  // the previous part's last reads of shared memory
    static_assert(sizeof(KParams) % 4 == 0, "KParams is copied as words");
    if (tid < (int)(sizeof(KParams) / 4))
      reinterpret_cast<int*>(&sP)[tid] = __ldg(reinterpret_cast<const int*>(gp + g) + tid);
    const KParams& P = sP;
    const double dt = clks[g].dt;
    const double dx = gp[g].dx;  // (served blocks are all at level 0)
    const float dtdx = (float)(dt / dx);
    const float h = (float)((0.5 * dt) / dx);
    const int gnb = gface >= 0 ? bt_at(bt, slot, 6 + gface) : 0;
    const bool g_bc = gface >= 0 && gnb <= -2;  // beyond the domain: the inner cell's half step
    const bool g_flip = g_bc && (-1 - gnb) == 2;
    bool xyg = false;
#pragma unroll
    for (int f = 0; f < 4; f++) xyg = xyg || bt_at(bt, slot, 6 + f) <= -2;
    const int zlo_nb = DIM == 3 ? bt_at(bt, slot, 10) : 0, zhi_nb = DIM == 3 ? bt_at(bt, slot, 11) : 0;

    float ph_prev = 0.f;
    // CTA-uniform: a predicted cell of plane j - 1 is shock-flagged; without one there or at plane j
    // the solver skips the HLL flux (the same bits)
    bool flagged_prev = true;
    auto issue = [&](int pl) {
      const int s = (pl + 3 * RING) % RING;
      if (tid == 0) {
        const size_t zb = (size_t)slot * BG<DIM>::WN + (DIM == 3 ? (size_t)(pl + NG) * SWN : 0);
        float4* dst = ring(pl);
        tma::fence_proxy_async();
        tma::mbar_expect_tx(&sBar[s], 2 * PLANE_BYTES);
        tma::bulk_g2s(dst, w1 + zb, PLANE_BYTES, &sBar[s]);
        tma::bulk_g2s(dst + SWN, w2 + zb, PLANE_BYTES, &sBar[s]);
      }
      pending |= 1u << s;
    };
    // Wait for plane pl; CTA-uniformly false if the copy did not complete in time.
    auto arrived = [&](int pl) -> bool {
      const int s = (pl + 3 * RING) % RING;
      const bool ok = tma::mbar_wait(&sBar[s], (phase >> s) & 1u, tma::WAIT_LIMIT);
      phase ^= 1u << s;
      pending &= ~(1u << s);
      return !__syncthreads_or(!ok);
    };
    // A copy that never completed: record it, let the others land (bounded), leave.
    auto give_up = [&]() {
      if (tid == 0 && err) atomicExch(err, tma::ERR_TMA_TIMEOUT);
      for (int s = 0; s < RING; s++)
        if (pending & (1u << s)) tma::mbar_wait(&sBar[s], (phase >> s) & 1u, tma::WAIT_LIMIT);
    };
    const int jb = DIM == 3 ? z0 - 1 : 0, je = DIM == 3 ? z1 : 0;
    if constexpr (DIM == 3) {
      issue(jb - 1);
      issue(jb);
      issue(jb + 1);
      if (!arrived(jb - 1) || !arrived(jb)) {
        give_up();
        return;
      }
    } else {
      issue(0);
    }
    for (int j = jb; j <= je; j++) {
      if (!arrived(DIM == 3 ? j + 1 : 0)) {
        give_up();
        return;
      }
      const float4* pj = ring(j);

      // the predictor at plane j
      float c[7];
      read_w7(pj, lx, ly, c);
      const uni::CellInv ci = uni::cell_inv(c);
      float su[DIM][6], sd[DIM][6];
      float conv, jump;
      {
        float m[7], p[7];
        read_w7(pj, lx - 1, ly, m);
        read_w7(pj, lx + 1, ly, p);
        uni::axis_edges<R, ISEN>(m, m, c, p, p, ci, P.inv_gamma, su[0], sd[0]);
        conv = p[1] - m[1];
        jump = jump_excess(m[4], p[4], P.shock_thresh);
        read_w7(pj, lx, ly - 1, m);
        read_w7(pj, lx, ly + 1, p);
        uni::axis_edges<R, ISEN>(m, m, c, p, p, ci, P.inv_gamma, su[1], sd[1]);
        conv += p[2] - m[2];
        jump = fmaxf(jump, jump_excess(m[4], p[4], P.shock_thresh));
        if constexpr (DIM == 3) {
          read_w7(ring(j - 1), lx, ly, m);
          read_w7(ring(j + 1), lx, ly, p);
          uni::axis_edges<R, ISEN>(m, m, c, p, p, ci, P.inv_gamma, su[2], sd[2]);
          conv += p[3] - m[3];
          jump = fmaxf(jump, jump_excess(m[4], p[4], P.shock_thresh));
        }
      }
      Pred pr;
      uni::hancock<DIM>(c, ci.r, conv, jump, su, sd, h, P, pr);

      const bool tile_plane = j >= z0 && j < z1;
      if (xyg && tile_plane) {
        // x and y boundary ghosts take the half step of the inner cell they map to
        put_pred(sFlux, SNT, tid, pr);
        __syncthreads();
        if (g_bc) {
          get_pred(sFlux, SNT, g_in, pr);
          if (g_flip && gface < 2) pr.q[1] = -pr.q[1];
          if (g_flip && gface >= 2) pr.q[2] = -pr.q[2];
        }
      }
      if constexpr (DIM == 3) {
        // z boundary ghosts: the lower one takes plane 0's half step with its own increments (kept
        // from plane -1); the upper one plane 15's (kept from plane 15). Each thread keeps and reads
        // back its own column: no barrier needed.
        if (j == -1 && zlo_nb <= -2) {
          sKeep[tid] = make_float4(su[2][0], su[2][1], su[2][2], su[2][3]);
          sKeep[SNT + tid] = make_float4(su[2][4], su[2][5], 0.f, 0.f);
        }
        if (j == 0 && z0 == 0 && zlo_nb <= -2) {
          Pred gq = pr;
          if (-1 - zlo_nb == 2) gq.q[3] = -gq.q[3];
          float inc[7], zf[7];
          get7(sKeep, SNT, tid, inc);
          uni::face_state(gq, inc, 1.f, zf);
          put7(sZup, SNT, tid, zf);
        }
        if (j == BS - 1 && z1 == BS && zhi_nb <= -2) put_pred(sKeep, SNT, tid, pr);
        if (j == BS && zhi_nb <= -2) {
          get_pred(sKeep, SNT, tid, pr);
          if (-1 - zhi_nb == 2) pr.q[3] = -pr.q[3];
        }
      }
      if (tile_plane) {
        float f[7];
        uni::face_state(pr, su[0], 1.f, f);
        put7(sFace, SNT, tid, f);
        uni::face_state(pr, su[1], 1.f, f);
        put7(sFace + 2 * SNT, SNT, tid, f);
      }
      const bool flagged = __syncthreads_or(pr.flag != 0.f);
      const bool hll_any = flagged || (DIM == 3 && flagged_prev);
      flagged_prev = flagged;
      // every thread is done with plane j - 1: its ring slot takes plane j + 2
      if (DIM == 3 && j + 2 <= je + 1) issue(j + 2);

      if (tile_plane) {
        if (xface_t) {
          float L[7], Rr[7], F[8];
          get7(sFace, SNT, x_dn, L);
          uni::face_state(pr, sd[0], -1.f, Rr);
          uni::riemann<0>(L, Rr, P, F, hll_any);
          put8(sFlux, SNT, tid, F);
        }
        if (yface_t) {
          float L[7], Rr[7], F[8];
          get7(sFace + 2 * SNT, SNT, y_dn, L);
          uni::face_state(pr, sd[1], -1.f, Rr);
          uni::riemann<1>(L, Rr, P, F, hll_any);
          put8(sFlux + 2 * SNT, SNT, tid, F);
        }
      }
      float Fz[8];
      if constexpr (DIM == 3) {
        if (tile_t && j >= z0) {
          // the z face below plane j
          float Rr[7], zf[7];
          uni::face_state(pr, sd[2], -1.f, Rr);
          get7(sZup, SNT, tid, zf);
          uni::riemann<2>(zf, Rr, P, Fz, hll_any);
        }
      }
      __syncthreads();

      if (tile_t) {
        float acc[8];
        if constexpr (DIM == 3) {
          if (j - 1 >= z0) {
            // plane j - 1 is complete: its upper z face is Fz
            get8(sAcc, SCELLS, tid, acc);
#pragma unroll
            for (int v = 0; v < 8; v++) acc[v] -= Fz[v];
            const size_t o = base + (size_t)(j - 1) * SCELLS + tid;
            float4 na, nb4;
            uni::update_cell(__ldg(u1 + o), __ldg(u2 + o), acc, ph_prev, dtdx, P, na, nb4);
            o1[o] = na;
            o2[o] = nb4;
          }
        }
        if (tile_plane) {
          float b[8];
          get8(sFlux, SNT, tid, acc);
          get8(sFlux, SNT, x_up, b);
#pragma unroll
          for (int v = 0; v < 8; v++) acc[v] -= b[v];
          get8(sFlux + 2 * SNT, SNT, tid, b);
#pragma unroll
          for (int v = 0; v < 8; v++) acc[v] += b[v];
          get8(sFlux + 2 * SNT, SNT, y_up, b);
#pragma unroll
          for (int v = 0; v < 8; v++) acc[v] -= b[v];
          ph_prev = pr.q[4];
          if constexpr (DIM == 3) {
#pragma unroll
            for (int v = 0; v < 8; v++) acc[v] += Fz[v];
            put8(sAcc, SCELLS, tid, acc);
          } else {
            const size_t o = base + tid;
            float4 na, nb4;
            uni::update_cell(__ldg(u1 + o), __ldg(u2 + o), acc, ph_prev, dtdx, P, na, nb4);
            o1[o] = na;
            o2[o] = nb4;
          }
        }
      }
      if constexpr (DIM == 3) {
        // the upper z face state of plane j (a lower boundary ghost's is set at plane 0)
        if (!(j == -1 && zlo_nb <= -2)) {
          float zf[7];
          uni::face_state(pr, su[2], 1.f, zf);
          put7(sZup, SNT, tid, zf);
        }
      }
    }
  }
}

template <int DIM, int R, bool ISEN>
cudaError_t launch(const AmrLaunch& L, const int* list, int n, int planes, int per_sm, const float4* u1, const float4* u2,
                   float4* o1, float4* o2, const DevClock* clks, cudaStream_t s) {
  auto k = grid_sweep<DIM, R, ISEN>;
  static LaunchAttr attr;
  const cudaError_t e = attr.set((const void*)k, SMEM, true);
  if (e != cudaSuccess) return e;
  k<<<grid_for(n * (DIM == 3 ? BS / planes : 1), per_sm), SNT, SMEM, s>>>(L.gp, L.bt, list, n, planes, u1, u2, L.w1, L.w2,
                                                                         o1, o2, clks, L.err);
  return cudaGetLastError();
}

// The planes of a block a CTA marches: the split whose parts fill the SMs best. A part of p planes
// takes about p + 4 plane times (two planes predicted only, the first copies); two parts run side by
// side on an SM, and one alone takes 0.65 of its time beside another.
int planes_of(int n) {
  double best = 0.0;
  int planes = BS;
  for (int p = BS; p >= 2; p /= 2) {
    const int per = (int)(((long long)n * (BS / p) + 147) / 148);
    const double cost = (p + 4) * (per / 2 + 0.65 * (per % 2));
    if (best == 0.0 || cost < best) {
      best = cost;
      planes = p;
    }
  }
  return planes;
}

}  // namespace gridsw

cudaError_t launch_grid_sweep(const AmrLaunch& L, const int* list, int n, const float4* u1, const float4* u2, float4* o1,
                              float4* o2, const DevClock* clks, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int planes = gridsw::planes_of(n);
  // (the grid is not timed here, the split decides more than it; a pinned block sweep's holds here too)
  tune::Choice c;
  const int per_sm = tune::pinned(tune::K_AMR_SWEEP, &c) && c.per_sm > 0 ? c.per_sm : 4;
  if (L.ndim == 3) {
    if (L.isen) { SHZ_RECON_SWITCH(L.recon, true, return (gridsw::launch<3, R, true>(L, list, n, planes, per_sm, u1, u2, o1, o2, clks, s))) }
    else { SHZ_RECON_SWITCH(L.recon, false, return (gridsw::launch<3, R, false>(L, list, n, planes, per_sm, u1, u2, o1, o2, clks, s))) }
  } else {
    if (L.isen) { SHZ_RECON_SWITCH(L.recon, true, return (gridsw::launch<2, R, true>(L, list, n, planes, per_sm, u1, u2, o1, o2, clks, s))) }
    else { SHZ_RECON_SWITCH(L.recon, false, return (gridsw::launch<2, R, false>(L, list, n, planes, per_sm, u1, u2, o1, o2, clks, s))) }
  }
  return cudaSuccess;
}

}  // namespace shz
