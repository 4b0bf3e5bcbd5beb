// The adaptive grid's arithmetic of one cell and one face (amr_*.cu): limiters, the density along the
// adiabat, the Hancock step, face states, the HLLC/HLL flux and the update. The sweeps of uniform grids
// and of served blocks have the same scheme in sweep_math.cuh, in a form of fewer instructions that
// rounds differently in places. This form keeps its rounding: refinement is
// decided by thresholds on what it computes, so that another rounding gives another mesh (on a mesh
// of 6,000 blocks, one block's decision within a dozen checks).
#pragma once
#include "hydro_math.cuh"

namespace shz {

// (Bitwise & and | rather than && and ||: no short-circuit, so no branch; the same values.)
__device__ __forceinline__ bool same_sign(float a, float b) { return ((a > 0.f) & (b > 0.f)) | ((a < 0.f) & (b < 0.f)); }

// hydro.ts:30-46 LIMITERS: the edge increment from the differences (far, near) and the
// quantity's natural scale (Koren only). The product test a*b > 0 is taken by signs, which is
// the same test without float32 underflow (as limiters/koren.wgsl:46-48 does).
template <int R>
__device__ __forceinline__ float limit(float a, float b, float scale) {
  if constexpr (R == R_MINMOD) {
    return same_sign(a, b) ? copysignf(fminf(fabsf(a), fabsf(b)), a) : 0.f;
  } else if constexpr (R == R_MC) {
    return same_sign(a, b) ? copysignf(fminf(fminf(2.f * fabsf(a), 2.f * fabsf(b)), 0.5f * fabsf(a + b)), a) : 0.f;
  } else if constexpr (R == R_VANLEER) {
    return same_sign(a, b) ? (2.f * a * b) / (a + b) : 0.f;
  } else {
    // Koren's limited third-order increment, unlimited where the change is small against the
    // scale (hydro.ts:35-45; SMOOTH = 0.01).
    const float far = a, near = b;
    const float fr = (far + 2.f * near) * (1.f / 3.f);
    const float lim = same_sign(far, near)
        ? copysignf(fminf(fminf(2.f * fabsf(far), 2.f * fabsf(near)), fabsf(fr)), near) : 0.f;
    const float s = 0.01f * scale;
    const float s2 = s * s;
    const bool as_is = ((s2 >= 1e-30f) & (s2 < 1e30f)) | (s == 0.f);
    // both forms, one kept (a select rather than a branch)
    const float eta_as_is = (far * far + near * near) / fmaxf(s2, 1e-30f);
    const float k = 1.f / fabsf(s);
    const float eta_scaled = (far * k) * (far * k) + (near * k) * (near * k);
    const float eta = as_is ? eta_as_is : eta_scaled;
    const float w = fminf(fmaxf(1.5f - eta, 0.f), 1.f);
    return lim + (fr - lim) * w;
  }
}

// Both of a cell's edge increments at once, lim(a, b) toward the upper face and lim(b, a) from the
// lower one. Koren's smoothness measure (far^2 + near^2) / scale^2 and its weight are symmetric in
// the two differences, as the reference computes them in float64: formed once for the pair (a
// single rounding order, where forming it per call let a fused multiply-add round the two orders
// apart), as are the sign test and the twice-the-smaller bound. Other limiters: two calls.
template <int R>
__device__ __forceinline__ void limit_pair(float a, float b, float scale, float& up, float& dn) {
  if constexpr (R != R_KOREN) {
    up = limit<R>(a, b, scale);
    dn = limit<R>(b, a, scale);
  } else {
    const float fu = (a + 2.f * b) * (1.f / 3.f), fd = (b + 2.f * a) * (1.f / 3.f);
    const bool same = same_sign(a, b);
    const float m2 = fminf(2.f * fabsf(a), 2.f * fabsf(b));
    const float lu = same ? copysignf(fminf(m2, fabsf(fu)), b) : 0.f;
    const float ld = same ? copysignf(fminf(m2, fabsf(fd)), a) : 0.f;
    const float s = 0.01f * scale;
    const float s2 = s * s;
    const bool as_is = ((s2 >= 1e-30f) & (s2 < 1e30f)) | (s == 0.f);
    const float eta_as_is = (a * a + b * b) / fmaxf(s2, 1e-30f);
    const float k = 1.f / fabsf(s);
    const float eta_scaled = (a * k) * (a * k) + (b * k) * (b * k);
    const float eta = as_is ? eta_as_is : eta_scaled;
    const float w = fminf(fmaxf(1.5f - eta, 0.f), 1.f);
    up = lu + (fu - lu) * w;
    dn = ld + (fd - ld) * w;
  }
}

// The limiters whose edge increment is the same slope at both faces (lim(a, b) == lim(b, a)).
template <int R>
__host__ __device__ constexpr bool symmetric_limiter() { return R == R_MINMOD || R == R_MC || R == R_VANLEER; }

// hydro.ts:65-83 isenInc and :260-265 isen, for both faces of a cell at once: moves the density
// increments toward the face (up) and from the lower face (dn) toward those along the adiabat,
// by the shared bound at most. m, c, p: (rho, vx, vy, vz, p, s, cs) of the lower neighbour, the
// cell and the upper neighbour; pu, pd: the cell's pressure increments at the two faces.
template <int R>
__device__ __forceinline__ void isen_blend(const float* m, const float* c, const float* p, float pu, float pd,
                                           float inv_gamma, float& up, float& dn) {
  const float rl = m[0], pl = m[4], rc = c[0], pc = c[4], rr = p[0], pr = p[4];
  // (hydro.ts:68: no increment unless all six are positive; the blend below is formed either way
  // and kept only then, a select rather than a branch)
  const bool ok = (rl > 0.f) & (pl > 0.f) & (rc > 0.f) & (pc > 0.f) & (rr > 0.f) & (pr > 0.f);
  const float gi = inv_gamma;
  const float tl = rl * powf(pc / pl, gi) - rc;
  const float tr = rr * powf(pc / pr, gi) - rc;
  const float fade_s = fminf(fmaxf(2.f - fmaxf(fabsf(pl - pc), fabsf(pr - pc)) / (0.2f * pc), 0.f), 1.f);
  const float fade_a = fminf(fmaxf(2.f - fmaxf(fabsf(tl), fabsf(tr)) / (0.01f * rc), 0.f), 1.f);
  const float dvr = sqrtf((p[1] - c[1]) * (p[1] - c[1]) + (p[2] - c[2]) * (p[2] - c[2]) + (p[3] - c[3]) * (p[3] - c[3]));
  const float dvl = sqrtf((c[1] - m[1]) * (c[1] - m[1]) + (c[2] - m[2]) * (c[2] - m[2]) + (c[3] - m[3]) * (c[3] - m[3]));
  const float fade_v = fminf(fmaxf(2.f - fmaxf(dvr, dvl) / (0.1f * fmaxf(c[6], 1e-30f)), 0.f), 1.f);
  const float bound = fmaxf(0.25f * fminf(fabsf(rc - rl), fabsf(rr - rc)), 0.01f * rc * fade_s * fade_a * fade_v);
  float d_up, d_dn;
  limit_pair<R>(-tl, tr, rc, d_up, d_dn);
  {
    const float d = d_up;
    const float pf = pc + 0.5f * pu;
    const float rf = fminf(fmaxf((rc + 0.5f * d) * powf(fmaxf(pf, 1e-30f) / pc, gi), fminf(rc, rr)), fmaxf(rc, rr));
    const float inc = 2.f * (rf - rc);
    up += ok ? fminf(fmaxf(inc - up, -bound), bound) : 0.f;
  }
  {
    const float d = d_dn;
    const float pf = pc - 0.5f * pd;
    const float rf = fminf(fmaxf((rc - 0.5f * d) * powf(fmaxf(pf, 1e-30f) / pc, gi), fminf(rc, rl)), fmaxf(rc, rl));
    const float inc = -2.f * (rf - rc);
    dn += ok ? fminf(fmaxf(inc - dn, -bound), bound) : 0.f;
  }
}

// The edge increments of one cell along one axis (hydro.ts:282-293; the ghost form :347-356):
// su toward the upper face, sd from the lower face, for (rho, vx, vy, vz, p, s).
template <int R, bool ISEN>
__device__ __forceinline__ void axis_edges(const float* m, const float* c, const float* p, float inv_gamma, float* su,
                                           float* sd) {
  // hydro.ts:268-270 scales: density, sound speed for velocities, pressure, none for s.
  const float sc[6] = {c[0], c[6], c[6], c[6], c[4], 0.f};
#pragma unroll
  for (int v = 0; v < 6; v++) {
    if constexpr (symmetric_limiter<R>()) {
      su[v] = limit<R>(c[v] - m[v], p[v] - c[v], sc[v]);
      sd[v] = su[v];
    } else {
      limit_pair<R>(c[v] - m[v], p[v] - c[v], sc[v], su[v], sd[v]);
    }
  }
  if constexpr (ISEN) isen_blend<R>(m, c, p, su[4], sd[4], inv_gamma, su[0], sd[0]);
}

// hydro.ts:360-375 side, rotated so that index 1 is normal to the face; then
// hydro.ts:102-159 riemannFlux. L and R are (rho, vx, vy, vz, p, s, shock flag). The flux comes
// back in the lab frame: (m, mx, my, mz, e, ei, s, vn).
// The three regions (left-supersonic, right-supersonic, star) and the star side are chosen by
// selects rather than branches, so that a warp whose faces fall in different regions runs one
// path; the values computed for the regions not chosen are discarded.
// hll_any: false when the caller knows that neither side of any face it solves is shock-flagged
// (a CTA-uniform fact, so the branch does not diverge). The HLL flux then has weight 0 and is
// skipped; a face of weight 0 takes the HLLC flux as it is either way.
template <int AXIS>
__device__ __forceinline__ void riemann(const float* L, const float* R, const KParams& P, float* F,
                                        bool hll_any = true) {
  constexpr int A0 = 1 + AXIS, A1 = 1 + (AXIS + 1) % 3, A2 = 1 + (AXIS + 2) % 3;
  const float lr = fmaxf(L[0], P.rho_floor), rr = fmaxf(R[0], P.rho_floor);
  const float lp = fmaxf(L[4], P.p_floor), rp = fmaxf(R[4], P.p_floor);
  const float lu = L[A0], lv = L[A1], lw = L[A2];
  const float ru = R[A0], rv = R[A1], rw = R[A2];
  const float lc = sqrtf(P.gamma * lp / lr), rc = sqrtf(P.gamma * rp / rr);
  const float lei = lp * P.inv_gm1, rei = rp * P.inv_gm1;
  const float w_hll = P.hll ? 1.f : fmaxf(L[6], R[6]);

  const float sl = fminf(lu - lc, ru - rc);
  const float sr = fmaxf(lu + lc, ru + rc);
  const float el = lei + 0.5f * lr * (lu * lu + lv * lv + lw * lw);
  const float er = rei + 0.5f * rr * (ru * ru + rv * rv + rw * rw);
  const float ml0 = lr * lu, ml1 = lr * lv, ml2 = lr * lw;
  const float mr0 = rr * ru, mr1 = rr * rv, mr2 = rr * rw;
  const float fpl0 = ml0 * lu + lp, fpl1 = ml1 * lu, fpl2 = ml2 * lu;
  const float fpr0 = mr0 * ru + rp, fpr1 = mr1 * ru, fpr2 = mr2 * ru;
  const float fel = (el + lp) * lu, fer = (er + rp) * ru;

  // HLL state flux and the contact speed
  const float ql = lr * (sl - lu);
  const float qr = rr * (sr - ru);
  const float sm = (rp - lp + lu * ql - ru * qr) / (ql - qr);
  // HLLC star state on the side of the contact the face lies on
  const bool left = sm >= 0.f;
  const float sK = left ? sl : sr, qK = left ? ql : qr, rK = left ? lr : rr, uK = left ? lu : ru;
  const float vK = left ? lv : rv, wK = left ? lw : rw, pK = left ? lp : rp, eK = left ? el : er;
  const float mK0 = left ? ml0 : mr0, mK1 = left ? ml1 : mr1, mK2 = left ? ml2 : mr2;
  const float fK0 = left ? fpl0 : fpr0, fK1 = left ? fpl1 : fpr1, fK2 = left ? fpl2 : fpr2, feK = left ? fel : fer;
  const float f = qK / (sK - sm);
  const float es = f * (eK / rK + (sm - uK) * (sm + pK / qK));
  const float cm = mK0 + sK * (f - rK);
  const float c0 = fK0 + sK * (f * sm - mK0);
  const float c1 = fK1 + sK * (f * vK - mK1);
  const float c2 = fK2 + sK * (f * wK - mK2);
  const float ce = feK + sK * (es - eK);
  float m = cm, p0 = c0, p1 = c1, p2 = c2, e = ce;
  if (hll_any || P.hll) {
    const float inv = 1.f / (sr - sl);
    const float slsr = sl * sr;
    const float hm = (sr * ml0 - sl * mr0 + slsr * (rr - lr)) * inv;
    const float hp0 = (sr * fpl0 - sl * fpr0 + slsr * (mr0 - ml0)) * inv;
    const float hp1 = (sr * fpl1 - sl * fpr1 + slsr * (mr1 - ml1)) * inv;
    const float hp2 = (sr * fpl2 - sl * fpr2 + slsr * (mr2 - ml2)) * inv;
    const float he = (sr * fel - sl * fer + slsr * (er - el)) * inv;
    // a face of weight 0 keeps the HLLC flux exactly, as where the HLL one was skipped: the
    // result does not depend on which faces share a CTA (c + (h - c) * 0 can turn -0 into +0)
    const bool blend = w_hll != 0.f;
    m = blend ? cm + (hm - cm) * w_hll : cm;
    p0 = blend ? c0 + (hp0 - c0) * w_hll : c0;
    p1 = blend ? c1 + (hp1 - c1) * w_hll : c1;
    p2 = blend ? c2 + (hp2 - c2) * w_hll : c2;
    e = blend ? ce + (he - ce) * w_hll : ce;
  }
  float vn = sm;
  // supersonic faces take the upwind side's flux
  const bool supl = sl >= 0.f, supr = sr <= 0.f;
  m = supl ? ml0 : (supr ? mr0 : m);
  p0 = supl ? fpl0 : (supr ? fpr0 : p0);
  p1 = supl ? fpl1 : (supr ? fpr1 : p1);
  p2 = supl ? fpl2 : (supr ? fpr2 : p2);
  e = supl ? fel : (supr ? fer : e);
  vn = supl ? lu : (supr ? ru : vn);
  const bool up = m >= 0.f;
  F[0] = m;
  F[A0] = p0;
  F[A1] = p1;
  F[A2] = p2;
  F[4] = e;
  F[5] = m * ((up ? lei : rei) / (up ? lr : rr));
  F[6] = m * (up ? L[5] : R[5]);
  F[7] = vn;
}

// hydro.ts:294-321: slopes -> shock flag -> Hancock half step -> positivity fallback, given the
// edge increments su/sd per active axis, the convergence, and the largest jump_excess over the
// axes; with the half-step slopes of some axes masked out (hydro/predictor.wgsl
// `mask`): a ghost next to a coarser block at the rim of its face has no transverse neighbours,
// so its slopes along those axes do not drive the half step. The positivity check still sees
// every increment, as in the reference.
template <int DIM>
__device__ __forceinline__ void hancock_masked(const float* c, float conv, float jump, const float (*su)[6],
                                               const float (*sd)[6], const float* mask, float h, const KParams& P,
                                               Pred& out) {
  float big = 0.f, fall = 0.f, dv = 0.f;
  float adv[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  float gradp[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int a = 0; a < DIM; a++) {
    big = fmaxf(big, fmaxf(fabsf(su[a][4]), fabsf(sd[a][4])));
    fall = fminf(fall, fminf(0.5f * su[a][0], -0.5f * sd[a][0]));
    const float va = c[1 + a];
    const float k = 0.5f * mask[a];
#pragma unroll
    for (int v = 0; v < 6; v++) adv[v] += va * (k * (su[a][v] + sd[a][v]));
    dv += k * (su[a][1 + a] + sd[a][1 + a]);
    gradp[a] = k * (su[a][4] + sd[a][4]);
  }
  out.flag = ((conv < 0.f) & (jump > 0.f)) ? 1.f : 0.f;
  const float rho = c[0], cs = c[6];
  const float inv_rho = 1.f / rho;
  float qh[6];
  qh[0] = rho - h * (adv[0] + rho * dv);
#pragma unroll
  for (int d = 0; d < 3; d++) qh[1 + d] = c[1 + d] - h * (adv[1 + d] + gradp[d] * inv_rho);
  qh[4] = c[4] - h * (adv[4] + rho * cs * cs * dv);
  qh[5] = c[5] - h * adv[5];
  const float rmin = qh[0] + fall;
  const float pmin = qh[4] - 0.5f * big;
  out.fo = !((rmin > 0.f) & (pmin > 0.f));
#pragma unroll
  for (int v = 0; v < 6; v++) out.q[v] = out.fo ? c[v] : qh[v];
}

// Face state q + 0.5 sgn inc (q alone when first order: the increments are zeroed), with the
// cell's shock flag (hydro.ts:362 side's f(n)).
__device__ __forceinline__ void face_state(const Pred& pr, const float* inc, float sgn, float* f) {
  const float k = pr.fo ? 0.f : 0.5f * sgn;
#pragma unroll
  for (int v = 0; v < 6; v++) f[v] = pr.q[v] + k * inc[v];
  f[6] = pr.flag;
}

// The update of one cell (hydro.ts:422-446): conservative update, dual-energy switch and floors.
// acc = (dm, dmx, dmy, dmz, de, dei, ds, dvn) summed with the reference's signs; ph = the
// cell's half-step pressure.
__device__ __forceinline__ void update_cell(const float4 a, const float4 b, const float* acc, float ph, float dtdx,
                                            const KParams& P, float4& na, float4& nb) {
  const float rho = fmaxf(a.x + dtdx * acc[0], P.rho_floor);
  const float mx = a.y + dtdx * acc[1], my = a.z + dtdx * acc[2], mz = a.w + dtdx * acc[3];
  float E = b.x + dtdx * acc[4];
  float eint = b.y + dtdx * (acc[5] + fmaxf(ph, P.p_floor) * acc[7]);
  const float ke = (0.5f * (mx * mx + my * my + mz * mz)) / rho;
  const float eth = E - ke;
  const float emin = P.e_floor;
  // the dual-energy switch by selects (a warp whose cells choose differently runs one path)
  const bool from_total = (eth > P.eta_dual * E) & (eth >= emin);
  const float eadv = (eint >= emin) ? eint : emin;
  eint = from_total ? eth : eadv;
  E = from_total ? E : ke + eadv;
  na = make_float4(rho, mx, my, mz);
  nb = make_float4(E, eint, b.z + dtdx * acc[6], b.w);
}

}  // namespace shz
