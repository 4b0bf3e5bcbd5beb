// The arithmetic of the uniform sweeps and of the served blocks' (sweep.cu, sweep_rows.cu,
// serve_sweep.cu): the scheme of block_math.cuh in the form of fewest instructions, which is what bounds
// those kernels. It rounds differently in places: limiters by
// sign-carrying minima instead of tests and selects, parabola edges as distances from the cell's
// value, one reciprocal shared by the divisions of a cell or of a face's side, the HLLC flux formed
// on the face's own side of the contact only. The adaptive mesh's passes keep block_math.cuh's form:
// refinement is decided by thresholds on what they compute, and another rounding makes another mesh.
// Measured against that form in the kernels of the time (one B200, ms a step): Taylor-Green 512^3 PPM
// 12.98 -> 9.23, Sedov 256^3 Koren 1.84 -> 1.46, Kelvin-Helmholtz 2048^2 Koren 0.271 -> 0.226, 1024^2 MC
// 0.0703 -> 0.0612; with what the kernels have gained since (cells in whole warps, the fitted depth,
// packed pairs) 8.70, 1.37, 0.198 and 0.0462. Errors against float64 (eight inputs each of 18 small cases):
// 0.79-1.09 times that form's for the state arrays, 0.96 in the mean.
#pragma once
#include "hydro_math.cuh"

#ifdef SHZ_PACKED_PAIRS
#define SHZ_UNI uni_packed
#else
#define SHZ_UNI uni
#endif

namespace shz {
namespace SHZ_UNI {

// The primitives are kept and read as the pairs (rho vx), (vy vz), (p s); what treats the six alike
// is written on the pairs. With SHZ_PACKED_PAIRS a pair's add, multiply or fma is one instruction of
// sm_100 (one issue slot for two operations of the same rate); else two.
#ifdef SHZ_PACKED_PAIRS
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 r;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n sub.rn.ftz.f32x2 z, x, y;\n mov.b64 {%0, %1}, z;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
#else
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
}
#endif
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 pair(const float* x, int i) { return make_float2(x[2 * i], x[2 * i + 1]); }
__device__ __forceinline__ void put2(float* x, int i, float2 v) {
  x[2 * i] = v.x;
  x[2 * i + 1] = v.y;
}

// min(|a|, |b|) with the sign of the product a b, in one instruction: positive where a and b have
// the same sign. The limiters take their test for an extremum from it: max(min_xs(a, b), 0) is the
// smaller of two differences of one sign, else 0, and min_xs(x, m) with m >= 0 gives x's sign to
// min(|x|, m). No comparison, select or sign copy is left (nor the product's underflow).
__device__ __forceinline__ float min_xs(float a, float b) {
  float d;
  asm("min.ftz.xorsign.abs.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float2 min_xs2(float2 a, float2 b) { return make_float2(min_xs(a.x, b.x), min_xs(a.y, b.y)); }
__device__ __forceinline__ float2 pos2(float2 a) { return make_float2(fmaxf(a.x, 0.f), fmaxf(a.y, 0.f)); }

// The limiters whose edge increment is the same slope at both faces (lim(a, b) == lim(b, a)).
template <int R>
__host__ __device__ constexpr bool symmetric_limiter() { return R == R_MINMOD || R == R_MC || R == R_VANLEER; }

// 1 / |0.01 scale|, the scale of Koren's smoothness measure (hydro.ts:29, 40-43 SMOOTH = 0.01); for
// a scale of 0 the measure's bound 1e-30 on the square.
constexpr float KOREN_K0 = 1e15f;
__device__ __forceinline__ float koren_k(float scale, float inv_scale) {
  return scale != 0.f ? 100.f * fabsf(inv_scale) : KOREN_K0;
}

// hydro.ts:30-46 LIMITERS, the symmetric ones on a pair: the edge increment from the differences on
// the two sides.
template <int R>
__device__ __forceinline__ float2 limit2(float2 a, float2 b) {
  static_assert(symmetric_limiter<R>(), "Koren's increments come as two (koren2)");
  if constexpr (R == R_MINMOD) {
    return min_xs2(a, pos2(min_xs2(a, b)));
  } else if constexpr (R == R_MC) {
    const float2 t = min_xs2(a, b);
    return min_xs2(mul2(add2(a, b), dup2(0.5f)), pos2(add2(t, t)));
  } else {
    const float2 q = mul2(a, b), s = add2(a, b), n = add2(q, q);
    return make_float2(q.x > 0.f ? n.x * (1.f / s.x) : 0.f, q.y > 0.f ? n.y * (1.f / s.y) : 0.f);
  }
}

// Koren's limited third-order increments of a pair, unlimited where the change is small against the
// quantity's scale (hydro.ts:35-45): lim(a, b) toward the upper face and lim(b, a) from the lower
// one. The smoothness measure (a^2 + b^2) / (0.01 scale)^2 and its weight are symmetric in the two
// differences and formed once; k = 1 / (0.01 scale) is the cell's, the same along every axis (the
// squares of a k and b k neither under- nor overflow where the measure decides). The two
// third-order increments share (a + b) / 3.
__device__ __forceinline__ void koren2(float2 a, float2 b, float2 k, float2& up, float2& dn) {
  const float2 third = dup2(1.f / 3.f);
  const float2 m = mul2(add2(a, b), third);
  const float2 fu = fma2(b, third, m), fd = fma2(a, third, m);
  const float2 t = min_xs2(a, b), r = pos2(add2(t, t));
  const float2 lu = min_xs2(fu, r), ld = min_xs2(fd, r);
  const float2 ak = mul2(a, k), bk = mul2(b, k);
  const float2 eta = fma2(ak, ak, mul2(bk, bk));
  const float2 w = make_float2(__saturatef(1.5f - eta.x), __saturatef(1.5f - eta.y));
  up = fma2(sub2(fu, lu), w, lu);
  dn = fma2(sub2(fd, ld), w, ld);
}

// The same for one quantity: lim(a, b) and lim(b, a) (k: Koren only).
template <int R>
__device__ __forceinline__ float limit(float a, float b) {
  if constexpr (R == R_MINMOD) {
    return min_xs(a, fmaxf(min_xs(a, b), 0.f));
  } else if constexpr (R == R_MC) {
    return min_xs(0.5f * (a + b), fmaxf(2.f * min_xs(a, b), 0.f));
  } else {
    static_assert(R == R_VANLEER, "Koren's increments come as two (limit_both)");
    return a * b > 0.f ? (2.f * a * b) * (1.f / (a + b)) : 0.f;
  }
}
template <int R>
__device__ __forceinline__ void limit_both(float a, float b, float k, float& up, float& dn) {
  if constexpr (symmetric_limiter<R>()) {
    up = limit<R>(a, b);
    dn = up;
  } else {
    const float m = (a + b) * (1.f / 3.f);
    const float fu = fmaf(b, 1.f / 3.f, m), fd = fmaf(a, 1.f / 3.f, m);
    const float r = fmaxf(2.f * min_xs(a, b), 0.f);
    const float lu = min_xs(fu, r), ld = min_xs(fd, r);
    const float ak = a * k, bk = b * k;
    const float w = __saturatef(1.5f - fmaf(ak, ak, bk * bk));
    up = fmaf(fu - lu, w, lu);
    dn = fmaf(fd - ld, w, ld);
  }
}

// What the edges of a cell need of its own primitives, the same along every axis: the reciprocals
// of the density, the pressure and the sound speed, and Koren's scales (hydro.ts:268-270: the
// density, the sound speed for velocities, the pressure, none for the scalar).
struct CellInv {
  float r, p, c;
  float kr, kc, kp;
};
__device__ __forceinline__ CellInv cell_inv(const float* c) {
  CellInv q;
  q.r = 1.f / c[0];
  q.p = 1.f / c[4];
  q.c = 1.f / fmaxf(c[6], 1e-30f);
  q.kr = koren_k(c[0], q.r);
  q.kc = c[6] != 0.f ? 100.f * (1.f / fabsf(c[6])) : KOREN_K0;
  q.kp = koren_k(c[4], q.p);
  return q;
}

// hydro.ts:65-83 isenInc and :260-265 isen, for both faces of a cell at once: moves the density
// increments toward the face (up) and from the lower face (dn) toward those along the adiabat,
// by the shared bound at most. m, c, p: (rho, vx, vy, vz, p, s, cs) of the lower neighbour, the
// cell and the upper neighbour; pu, pd: the cell's pressure increments at the two faces.
template <int R>
__device__ __forceinline__ void isen_blend(const float* m, const float* c, const float* p, const CellInv& q, float pu,
                                           float pd, float inv_gamma, float& up, float& dn) {
  const float rl = m[0], pl = m[4], rc = c[0], pc = c[4], rr = p[0], pr = p[4];
  // (hydro.ts:68: no increment unless all six are positive; the blend below is formed either way
  // and kept only then, a select rather than a branch)
  const bool ok = (fminf(fminf(rl, pl), fminf(rr, pr)) > 0.f) & (fminf(rc, pc) > 0.f);
  const float gi = inv_gamma;
  const float tl = fmaf(rl, powf(pc * (1.f / pl), gi), -rc);
  const float tr = fmaf(rr, powf(pc * (1.f / pr), gi), -rc);
  // the three fades: pressure jump / (0.2 p), distance from the adiabat / (0.01 rho), shear / (0.1 c)
  const float fade_s = __saturatef(fmaf(-fmaxf(fabsf(pl - pc), fabsf(pr - pc)), 5.f * q.p, 2.f));
  const float fade_a = __saturatef(fmaf(-fmaxf(fabsf(tl), fabsf(tr)), 100.f * q.r, 2.f));
  const float rx = p[1] - c[1], ry = p[2] - c[2], rz = p[3] - c[3];
  const float lx = c[1] - m[1], ly = c[2] - m[2], lz = c[3] - m[3];
  const float dv2 = fmaxf(fmaf(rx, rx, fmaf(ry, ry, rz * rz)), fmaf(lx, lx, fmaf(ly, ly, lz * lz)));
  const float fade_v = __saturatef(fmaf(-sqrtf(dv2), 10.f * q.c, 2.f));
  const float bound = fmaxf(0.25f * fminf(fabsf(rc - rl), fabsf(rr - rc)), 0.01f * rc * fade_s * fade_a * fade_v);
  float d_up, d_dn;
  limit_both<R>(-tl, tr, q.kr, d_up, d_dn);
  {
    const float pf = fmaxf(fmaf(0.5f, pu, pc), 1e-30f);
    const float rf = fminf(fmaxf(fmaf(0.5f, d_up, rc) * powf(pf * q.p, gi), fminf(rc, rr)), fmaxf(rc, rr));
    const float inc = 2.f * (rf - rc);
    up += ok ? fminf(fmaxf(inc - up, -bound), bound) : 0.f;
  }
  {
    const float pf = fmaxf(fmaf(-0.5f, pd, pc), 1e-30f);
    const float rf = fminf(fmaxf(fmaf(-0.5f, d_dn, rc) * powf(pf * q.p, gi), fminf(rc, rl)), fmaxf(rc, rl));
    const float inc = -2.f * (rf - rc);
    dn += ok ? fminf(fmaxf(inc - dn, -bound), bound) : 0.f;
  }
}

// Colella & Woodward (1984) parabola edges (their eqs. 1.6, 1.8 and 1.10) from five cells;
// no counterpart in the reference. The increments come in the reference's convention, twice the
// distance from the cell's value to its edge (hydro.ts:282-293), and so do the slopes here: twice
// the limited slope of eq. 1.8, min(|dl + dr|, 4 min(|dl|, |dr|)) with the differences' common sign.
__device__ __forceinline__ float2 ppm_slope2(float2 dl, float2 dr) {
  return min_xs2(add2(dl, dr), pos2(mul2(min_xs2(dl, dr), dup2(4.f))));
}
// The increments from the cell's two differences and the slopes at the cells below, at and above
// it (a march that has the slopes already gives them here). With R and L the doubled distances of
// the unlimited edges (eq. 1.6) from the cell's value, eq. 1.10 reads: none at an extremum
// (R L <= 0); an edge more than twice as far as the other is pulled in to twice its distance.
// In distances, rather than in edge values, the cell's value cancels exactly.
__device__ __forceinline__ void ppm_edges2(float2 dl, float2 dr, float2 sm, float2 s0, float2 sp, float2& su, float2& sd) {
  const float2 R = fma2(sub2(sp, s0), dup2(-1.f / 6.f), dr);
  const float2 L = fma2(sub2(s0, sm), dup2(1.f / 6.f), dl);
  const float2 t = pos2(min_xs2(R, L)), t2 = add2(t, t);
  su = min_xs2(R, t2);
  sd = min_xs2(L, t2);
}

// The edge increments of one cell along one axis (hydro.ts:282-293; the ghost form :347-356):
// su toward the upper face, sd from the lower face, for (rho, vx, vy, vz, p, s).
// m2, p2 (two cells away) are read by PPM only.
template <int R, bool ISEN>
__device__ __forceinline__ void axis_edges(const float* m2, const float* m, const float* c, const float* p, const float* p2,
                                           const CellInv& q, float inv_gamma, float* su, float* sd) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const float2 cc = pair(c, i), dl = sub2(cc, pair(m, i)), dr = sub2(pair(p, i), cc);
    float2 u, d;
    if constexpr (R == R_PPM) {
      const float2 d1 = sub2(pair(m, i), pair(m2, i)), d4 = sub2(pair(p2, i), pair(p, i));
      ppm_edges2(dl, dr, ppm_slope2(d1, dl), ppm_slope2(dl, dr), ppm_slope2(dr, d4), u, d);
    } else if constexpr (R == R_KOREN) {
      koren2(dl, dr, i == 0 ? make_float2(q.kr, q.kc) : i == 1 ? dup2(q.kc) : make_float2(q.kp, KOREN_K0), u, d);
    } else {
      u = limit2<R>(dl, dr);
      d = u;
    }
    put2(su, i, u);
    put2(sd, i, d);
  }
  if constexpr (ISEN && R != R_PPM) isen_blend<R>(m, c, p, q, su[4], sd[4], inv_gamma, su[0], sd[0]);
}

// hydro.ts:360-375 side, rotated so that index 1 is normal to the face; then
// hydro.ts:102-159 riemannFlux. L and R are (rho, vx, vy, vz, p, s, shock flag). The flux comes
// back in the lab frame: (m, mx, my, mz, e, ei, s, vn).
// The side of the contact the face lies on (the upwind side where both waves run one way) is chosen
// first, by selects, so that a warp whose faces fall in different regions runs one path, and the
// state and flux are formed for that side only. The star state moves its transverse velocities
// with the mass flux, so those two momentum fluxes are the mass flux times the side's velocities.
// hll_any: false when the caller knows that neither side of any face it solves is shock-flagged
// (a CTA-uniform fact, so the branch does not diverge). The HLL flux, which needs both sides, then
// has weight 0 and is skipped; a face of weight 0 takes the HLLC flux as it is either way.
template <int AXIS>
__device__ __forceinline__ void riemann(const float* L, const float* R, const KParams& P, float* F,
                                        bool hll_any = true) {
  constexpr int A0 = 1 + AXIS, A1 = 1 + (AXIS + 1) % 3, A2 = 1 + (AXIS + 2) % 3;
  const float lr = fmaxf(L[0], P.rho_floor), rr = fmaxf(R[0], P.rho_floor);
  const float lp = fmaxf(L[4], P.p_floor), rp = fmaxf(R[4], P.p_floor);
  const float lu = L[A0], ru = R[A0];
  const float ilr = 1.f / lr, irr = 1.f / rr;
  const float lh = lp * ilr, rh = rp * irr;  // p / rho
  const float lc = sqrtf(P.gamma * lh), rc = sqrtf(P.gamma * rh);
  const float sl = fminf(lu - lc, ru - rc);
  const float sr = fmaxf(lu + lc, ru + rc);
  const float ql = lr * (sl - lu);
  const float qr = rr * (sr - ru);
  // the contact speed
  const float sm = fmaf(-ru, qr, fmaf(lu, ql, rp - lp)) * (1.f / (ql - qr));
  const bool supl = sl >= 0.f, supr = sr <= 0.f;
  const bool sup = supl | supr;
  const bool left = supl | (!supr & (sm >= 0.f));
  const float sK = left ? sl : sr, qK = left ? ql : qr, rK = left ? lr : rr, uK = left ? lu : ru;
  const float vK = left ? L[A1] : R[A1], wK = left ? L[A2] : R[A2], pK = left ? lp : rp;
  const float kin = 0.5f * fmaf(uK, uK, fmaf(vK, vK, wK * wK));
  const float hK = (left ? lh : rh) * P.inv_gm1;  // the side's specific internal energy
  const float eK = rK * (hK + kin);
  const float mK = rK * uK;
  const float fK = fmaf(mK, uK, pK), feK = (eK + pK) * uK;
  // HLLC star state
  const float g = 1.f / (sK - sm), du = sm - uK;
  const float f = qK * g;
  const float es = fmaf(f, fmaf(du, sm, hK + kin), du * (pK * g));
  const float cm = fmaf(sK, f - rK, mK);
  const float c0 = fmaf(sK, fmaf(f, sm, -mK), fK);
  const float ce = fmaf(sK, es - eK, feK);
  // supersonic faces take the upwind side's flux
  float m = sup ? mK : cm, p0 = sup ? fK : c0, e = sup ? feK : ce;
  const float vn = sup ? uK : sm;
  float p1 = m * vK, p2 = m * wK;
  if (hll_any || P.hll) {
    const float w_hll = P.hll ? 1.f : fmaxf(L[6], R[6]);
    const float lv = L[A1], lw = L[A2], rv = R[A1], rw = R[A2];
    const float inv = 1.f / (sr - sl);
    const float slsr = sl * sr;
    const float el = lr * fmaf(lh, P.inv_gm1, 0.5f * fmaf(lu, lu, fmaf(lv, lv, lw * lw)));
    const float er = rr * fmaf(rh, P.inv_gm1, 0.5f * fmaf(ru, ru, fmaf(rv, rv, rw * rw)));
    const float ml = lr * lu, mr = rr * ru;
    const float hm = (sr * ml - sl * mr + slsr * (rr - lr)) * inv;
    const float h0 = (sr * fmaf(ml, lu, lp) - sl * fmaf(mr, ru, rp) + slsr * (mr - ml)) * inv;
    const float h1 = (sr * (ml * lv) - sl * (mr * rv) + slsr * (rr * rv - lr * lv)) * inv;
    const float h2 = (sr * (ml * lw) - sl * (mr * rw) + slsr * (rr * rw - lr * lw)) * inv;
    const float he = (sr * ((el + lp) * lu) - sl * ((er + rp) * ru) + slsr * (er - el)) * inv;
    // a face of weight 0 keeps the HLLC flux exactly, as where the HLL one was skipped: the
    // result does not depend on which faces share a CTA (c + (h - c) * 0 can turn -0 into +0)
    const bool blend = !sup & (w_hll != 0.f);
    m = blend ? fmaf(hm - m, w_hll, m) : m;
    p0 = blend ? fmaf(h0 - p0, w_hll, p0) : p0;
    p1 = blend ? fmaf(h1 - p1, w_hll, p1) : p1;
    p2 = blend ? fmaf(h2 - p2, w_hll, p2) : p2;
    e = blend ? fmaf(he - e, w_hll, e) : e;
  }
  const bool up = m >= 0.f;
  F[0] = m;
  F[A0] = p0;
  F[A1] = p1;
  F[A2] = p2;
  F[4] = e;
  F[5] = m * ((up ? lh : rh) * P.inv_gm1);
  F[6] = m * (up ? L[5] : R[5]);
  F[7] = vn;
}

// hydro.ts:294-321: slopes -> shock flag -> Hancock half step -> positivity fallback, given the
// edge increments su/sd per active axis, the convergence, and the largest jump_excess over the axes.
// inv_rho: 1 / c[0].
template <int DIM>
__device__ __forceinline__ void hancock(const float* c, float inv_rho, float conv, float jump, const float (*su)[6],
                                        const float (*sd)[6], float h, const KParams& P, Pred& out) {
  float big = 0.f, fall = 0.f, dv = 0.f;  // (fall, dv and gradp doubled, as the increments are)
  float gradp[3] = {0.f, 0.f, 0.f};
  float2 adv[3];
#pragma unroll
  for (int a = 0; a < DIM; a++) {
    big = fmaxf(big, fmaxf(fabsf(su[a][4]), fabsf(sd[a][4])));
    fall = fminf(fall, fminf(su[a][0], -sd[a][0]));
    const float2 va = dup2(0.5f * c[1 + a]);
    float sum[6];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const float2 t = add2(pair(su[a], i), pair(sd[a], i));
      put2(sum, i, t);
      adv[i] = a == 0 ? mul2(va, t) : fma2(va, t, adv[i]);
    }
    dv = a == 0 ? sum[1] : dv + sum[1 + a];
    gradp[a] = sum[4];
  }
  out.flag = ((conv < 0.f) & (jump > 0.f)) ? 1.f : 0.f;
  const float rho = c[0], cs = c[6];
  const float hi = 0.5f * inv_rho, hdv = 0.5f * dv;
  const float2 mh = dup2(-h);
  float qh[6];
  put2(qh, 0, fma2(mh, make_float2(fmaf(rho, hdv, adv[0].x), fmaf(gradp[0], hi, adv[0].y)), pair(c, 0)));
  put2(qh, 1, fma2(mh, DIM == 3 ? fma2(make_float2(gradp[1], gradp[2]), dup2(hi), adv[1])
                                : make_float2(fmaf(gradp[1], hi, adv[1].x), adv[1].y), pair(c, 1)));
  put2(qh, 2, fma2(mh, make_float2(fmaf(rho * cs * cs, hdv, adv[2].x), adv[2].y), pair(c, 2)));
  const float rmin = fmaf(0.5f, fall, qh[0]);
  const float pmin = fmaf(-0.5f, big, qh[4]);
  out.fo = !((rmin > 0.f) & (pmin > 0.f));
#pragma unroll
  for (int v = 0; v < 6; v++) out.q[v] = out.fo ? c[v] : qh[v];
}

// Face state q + 0.5 sgn inc (q alone when first order: the increments are zeroed), with the
// cell's shock flag (hydro.ts:362 side's f(n)).
__device__ __forceinline__ void face_state(const Pred& pr, const float* inc, float sgn, float* f) {
  const float2 k = dup2(pr.fo ? 0.f : 0.5f * sgn);
#pragma unroll
  for (int i = 0; i < 3; i++) put2(f, i, fma2(k, pair(inc, i), pair(pr.q, i)));
  f[6] = pr.flag;
}

// The update of one cell (hydro.ts:422-446): conservative update, dual-energy switch and floors.
// acc = (dm, dmx, dmy, dmz, de, dei, ds, dvn) summed with the reference's signs; ph = the
// cell's half-step pressure.
__device__ __forceinline__ void update_cell(const float4 a, const float4 b, const float* acc, float ph, float dtdx,
                                            const KParams& P, float4& na, float4& nb) {
  const float2 d = dup2(dtdx);
  const float2 ra = fma2(d, pair(acc, 0), make_float2(a.x, a.y)), rb = fma2(d, pair(acc, 1), make_float2(a.z, a.w));
  const float2 en = fma2(d, make_float2(acc[4], fmaf(fmaxf(ph, P.p_floor), acc[7], acc[5])), make_float2(b.x, b.y));
  const float rho = fmaxf(ra.x, P.rho_floor);
  const float mx = ra.y, my = rb.x, mz = rb.y;
  float E = en.x, eint = en.y;
  const float ke = (0.5f * fmaf(mx, mx, fmaf(my, my, mz * mz))) * (1.f / rho);
  const float eth = E - ke;
  const float emin = P.e_floor;
  // the dual-energy switch by selects (a warp whose cells choose differently runs one path)
  const bool from_total = (eth > P.eta_dual * E) & (eth >= emin);
  const float eadv = (eint >= emin) ? eint : emin;
  eint = from_total ? eth : eadv;
  E = from_total ? E : ke + eadv;
  na = make_float4(rho, mx, my, mz);
  nb = make_float4(E, eint, fmaf(dtdx, acc[6], b.z), b.w);
}

}  // namespace SHZ_UNI
}  // namespace shz
