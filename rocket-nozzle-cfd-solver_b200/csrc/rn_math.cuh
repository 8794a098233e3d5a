// rn_math.cuh -- per-cell and per-face arithmetic of the time step, sm_100a.
//
// Every function states the reference shader lines it computes
// (source/solver.js, source/spray.js). The kernels in rn_step.cu fuse these
// into tiles; the arithmetic and its operation order are the reference's, so
// that in the exact variant (IEEE division and square root, multiply-add
// contraction off) the fused kernels give the same float32 results as the
// pass-by-pass restatement wherever the math library functions (pow, exp, log,
// sin, cos) agree.
// GLSL max/min are IEEE maxNum/minNum (fmaxf/fminf), what NVIDIA GPUs execute.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "rn.h"

#define RN_DEV __device__ __forceinline__

namespace rn {

constexpr float RHO_MIN = 1e-7f;   // solver.js:27
constexpr float P_MIN = 1e-7f;     // solver.js:28

struct Grid {
  int Nx, Nr;
  const uint8_t* __restrict__ mask;   // Nx*Nr, nonzero = solid
  const float4* __restrict__ geoA;    // (Nx+1)*(Nr+1): (V, Am, Ax west, Ar south), negative area -> first order
  const float4* __restrict__ geoG;    // Nx*Nr: group (V, Am, Wx, Wr)
  const float4* __restrict__ geoM;    // Nx*Nr: (host dx, host dy, slave mask, turbulence length)
};

struct Prim { float4 w, s; };        // w = (rho, u, v, p), s = (Z, F, G, O)   solver.js:29
struct Flux { float4 F, Y; float O; };   // face flux: F(4), (FZ, FF, u_f G_f, u_f), FO

// Division of the time-step arithmetic. The fast variant (RN_FAST) multiplies
// by the hardware's approximate reciprocal (one instruction, within 2 ulp for
// divisors of magnitude 2^-126 .. 2^126, which every divisor here is: densities,
// pressures, wave speeds, face areas and volumes, all floored well above
// 2^-126 and far below 2^126); the exact variant divides as IEEE does.
#ifdef RN_FAST
RN_DEV float rcp(float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return r;
}
#endif
RN_DEV float fdiv(float a, float b) {
#ifdef RN_FAST
  return a * rcp(b);
#else
  return a / b;
#endif
}
// Several quotients over one divisor b: over(b)(a) == fdiv(a, b). The fast
// variant forms the reciprocal once and multiplies (fdiv there is a times the
// hardware reciprocal of b); the exact variant divides each time.
struct Over {
  float b, r;
  RN_DEV float operator()(float a) const {
#ifdef RN_FAST
    return a * r;
#else
    return a / b;
#endif
  }
};
RN_DEV Over over(float b) {
  Over o;
  o.b = b;
#ifdef RN_FAST
  o.r = rcp(b);
#else
  o.r = 0.0f;
#endif
  return o;
}

// Pairs of lanes through Blackwell's packed FP32 instructions (two IEEE
// round-to-nearest operations per instruction, each lane rounding as the
// scalar operation does). madd2 is a*b + c: one fused multiply-add per lane in
// the fast variant, a multiply then an add (scalar) in the exact one.
RN_DEV float2 lo2(float4 v) { return make_float2(v.x, v.y); }
RN_DEV float2 hi2(float4 v) { return make_float2(v.z, v.w); }
RN_DEV float4 cat4(float2 l, float2 h) { return make_float4(l.x, l.y, h.x, h.y); }
RN_DEV float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
// b * (-1) is exact, so this is a - b rounded once: one packed instruction
// where a packed add of -b would negate b's lanes first
RN_DEV float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
RN_DEV float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
RN_DEV float2 madd2(float2 a, float2 b, float2 c) {
#ifdef RN_FAST
  return __ffma2_rn(a, b, c);
#else
  // scalar lanes: a packed multiply followed by a packed add may be fused,
  // which the exact variant must not do (it is built with -fmad=false)
  return make_float2(c.x + a.x * b.x, c.y + a.y * b.y);
#endif
}
RN_DEV float4 diff4(float4 a, float4 b) { return cat4(sub2(lo2(a), lo2(b)), sub2(hi2(a), hi2(b))); }

RN_DEV float clampf(float x, float a, float b) { return fminf(fmaxf(x, a), b); }
RN_DEV float mixf(float x, float y, float a) { return x * (1.0f - a) + y * a; }
RN_DEV float smoothstepf(float e0, float e1, float x) {
  float t = clampf(fdiv(x - e0, e1 - e0), 0.0f, 1.0f);
  return t * t * (3.0f - 2.0f * t);
}
RN_DEV float len2(float a, float b) { return sqrtf(a * a + b * b); }
RN_DEV int iround(float v) { return __float2int_rn(v); }

RN_DEV bool solid_at(const Grid& g, int i, int j) { return g.mask[j * g.Nx + i] != 0; }

// toPrim (solver.js:33-39)
RN_DEV Prim to_prim(float4 a, float4 b) {
  Prim q;
  float rho = fmaxf(a.x, RHO_MIN);
  const Over per_rho = over(rho);
  float vx = per_rho(a.y), vy = per_rho(a.z);
  float G = fmaxf(b.z, 0.5f);
  float p = fmaxf(fdiv(a.w - 0.5f * rho * (vx * vx + vy * vy), G), P_MIN);
  q.w = make_float4(rho, vx, vy, p);
  q.s = make_float4(__saturatef(per_rho(b.x)), __saturatef(per_rho(b.y)), G, __saturatef(per_rho(b.w)));
  return q;
}
// soundSpeed (solver.js:40)
RN_DEV float sound_speed(const Prim& q) { return sqrtf(fdiv((1.0f + fdiv(1.0f, q.s.z)) * q.w.w, q.w.x)); }

// CFL wave speed of one fluid cell (FS_REDUCE1, solver.js:376-379)
RN_DEV float wave_speed(float4 a, float4 b) {
  Prim q = to_prim(a, b);
  return fabsf(q.w.y) + fabsf(q.w.z) + 2.0f * sound_speed(q);
}

// Cells of the grid as ghost_prim_c reads them: solid flag and raw state of
// in-grid cell (i, j). GlobalCells reads the planes in global memory; the
// stage kernels read the tile they staged in shared memory (rn_step.cu).
struct GlobalCells {
  const Grid& g;
  const float4* __restrict__ A;
  const float4* __restrict__ B;
  RN_DEV bool solid(int i, int j) const { return g.mask[j * g.Nx + i] != 0; }
  RN_DEV float4 a(int i, int j) const { return A[j * g.Nx + i]; }
  RN_DEV float4 b(int i, int j) const { return B[j * g.Nx + i]; }
};

// W of a wall cell: rho = -1 marks it. Its pressure is a NaN, so that the shock
// sensor's minima and maxima (minNum/maxNum) pass over it; nothing else reads it.
RN_DEV float4 wall_prim() { return make_float4(-1.0f, 0.0f, 0.0f, __int_as_float(0x7fffffff)); }

// Padded primitive cell (i, j), i in [-2, Nx+1], j in [-2, Nr+1] (FS_PRIM,
// solver.js:56-126). Wall cells come back as W = wall_prim(), Wb = 0.
// t is the time the inlet ramp reads (t_old in stage 1, t_new in stage 2).
// Every cell it reads lies within 2 cells of (i, j), inside the grid.
template <class C>
RN_DEV void ghost_prim_c(int Nx, int Nr, const C& cells, int i, int j, float t, const rn_params& P, float4& W,
                         float4& Wb) {
  bool mir = j < 0;
  if (mir) j = -j - 1;
  Prim q;
  q.w = make_float4(P.amb[0], P.amb[1], P.amb[2], P.amb[3]);
  q.s = make_float4(0.0f, 0.0f, P.inlet[3], 0.0f);
  bool wall = false;
  if (i < 0) {
    if (j < Nr && cells.solid(0, j)) wall = true;
    else if (float(j) + 0.5f < P.RcCells && P.inj) wall = true;
    else if (float(j) + 0.5f < P.RcCells) {
      float f = P.ramp > 0.0f ? smoothstepf(0.0f, P.ramp, t) : 1.0f;
      float P0 = mixf(P.pStart, P.res[0], f);
      float T0 = P.res[1], R = P.res[2], G = P.inlet[2], gg = 1.0f + 1.0f / G;
      float4 a = cells.a(0, j);
      float ubar = fmaxf(cells.b(0, j).w, 0.0f);
      float c0 = sqrtf(gg * R * T0);
      float ui = clampf(a.y / fmaxf(a.x, RHO_MIN), 0.0f, 0.5f * c0);
      float ut = ubar * smoothstepf(1.0f, 2.0f, P0 / fmaxf(P.pStart, 1e-6f));
      float u = mixf(ui, ut, P.inlet[1]);
      float T = T0 - u * u * (gg - 1.0f) / (2.0f * gg * R);
      float p = P0 * powf(T / T0, gg * G);
      q.w = make_float4(p / (R * T), u, 0.0f, p);
      q.s = make_float4(1.0f, 1.0f, G, 0.0f);
    }
  } else if (j >= Nr) {
    int ci = min(i, Nx - 1), cj = Nr - 1;
    if (!cells.solid(ci, cj)) {
      Prim tq = to_prim(cells.a(ci, cj), cells.b(ci, cj));
      float cs = sound_speed(tq);
      if (tq.w.z >= cs) q = tq;
      else if (tq.w.z > 0.0f) { q = tq; q.w.w = P.amb[3]; }
    }
  } else if (i >= Nx) {
    int ci = Nx - 1, cj = j;
    if (!cells.solid(ci, cj)) {
      Prim tq = to_prim(cells.a(ci, cj), cells.b(ci, cj));
      float cs = sound_speed(tq);
      if (tq.w.y >= cs) q = tq;
      else if (tq.w.y > 0.0f) { q = tq; q.w.w = P.amb[3]; }
      else q.w.y = fmaxf(q.w.y, 0.0f);
    }
  } else {
    // the state is loaded with the mask (not after it), so the two loads overlap
    const float4 a = cells.a(i, j), b = cells.b(i, j);
    if (cells.solid(i, j)) wall = true;
    else q = to_prim(a, b);
  }
  if (wall) {
    W = wall_prim();
    Wb = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    return;
  }
  if (mir) q.w.z = -q.w.z;
  W = q.w;
  Wb = q.s;
}
RN_DEV void ghost_prim(const Grid& g, const float4* __restrict__ A, const float4* __restrict__ B, int i, int j,
                       float t, const rn_params& P, float4& W, float4& Wb) {
  ghost_prim_c(g.Nx, g.Nr, GlobalCells{g, A, B}, i, j, t, P, W, Wb);
}

// Interior cell as the padded texture holds it (wall flag or toPrim).
RN_DEV void interior_prim(const Grid& g, const float4* __restrict__ A, const float4* __restrict__ B, int i, int j,
                          float4& W, float4& Wb) {
  if (solid_at(g, i, j)) {
    W = wall_prim();
    Wb = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  } else {
    Prim q = to_prim(A[j * g.Nx + i], B[j * g.Nx + i]);
    W = q.w;
    Wb = q.s;
  }
}

// ---------------------------------------------------------------------------
// Inviscid face flux: MUSCL van Leer + HLLC blended to HLL (makeFluxShader,
// solver.js:133-259).
//
// Half the limited slope of a cell from its differences a (to the cell behind)
// and b (to the cell ahead): ab / (a + b) where ab > 0, else 0. The reference's
// limiter is 2 max(ab, 0) / mix(den, 1, step(|den|, 1e-30)), den = a + b, and
// its face values are w +- 0.5 times it. For ab <= 0 the quotient is a zero
// carrying den's sign, so the division is skipped.
RN_DEV float2 half_slope2(float2 a, float2 b) {
  const float2 ab = mul2(a, b), den = add2(a, b);
#ifdef RN_FAST
  // ab > 0 means a and b of one sign, so |den| = |a| + |b| >= 2 sqrt(ab) >
  // 1e-30: the guard never applies
  const float2 r = make_float2(rcp(den.x), rcp(den.y));
  return mul2(ab, make_float2(ab.x > 0.0f ? r.x : 0.0f, ab.y > 0.0f ? r.y : 0.0f));
#else
  const float2 d = make_float2((1e-30f < fabsf(den.x)) ? den.x : 1.0f, (1e-30f < fabsf(den.y)) ? den.y : 1.0f);
  return make_float2(ab.x > 0.0f ? 0.5f * (2.0f * ab.x / d.x) : copysignf(0.0f, d.x),
                     ab.y > 0.0f ? 0.5f * (2.0f * ab.y / d.y) : copysignf(0.0f, d.y));
#endif
}
// One side's face value: w + h or w - h of the primitives, and of the scalars
// with their bounds (fractions in 0..1, G in 0.5..100).
struct Side { float4 w, s; };
template <bool PLUS>
RN_DEV Side side_of(float4 w, float4 b, float4 h, float4 g) {
  Side o;
  if constexpr (PLUS) {
    o.w = cat4(add2(lo2(w), lo2(h)), add2(hi2(w), hi2(h)));
    o.s = make_float4(__saturatef(b.x + g.x), __saturatef(b.y + g.y), clampf(b.z + g.z, 0.5f, 100.0f),
                      __saturatef(b.w + g.w));
  } else {
    o.w = diff4(w, h);
    o.s = make_float4(__saturatef(b.x - g.x), __saturatef(b.y - g.y), clampf(b.z - g.z, 0.5f, 100.0f),
                      __saturatef(b.w - g.w));
  }
  return o;
}
RN_DEV float4 half_slope4(float4 a, float4 b) {
  return cat4(half_slope2(lo2(a), lo2(b)), half_slope2(hi2(a), hi2(b)));
}
// |a - b| / min(a, b), a not NaN; 0 where b is NaN (a wall cell).
RN_DEV float jump_ratio(float a, float b) {
  const float lo = fminf(a, b);
  return fdiv(fmaxf(a, b) - lo, lo);
}

#ifdef RN_FAST
// HLLC of the fast variant (makeFluxShader's formulas, solver.js:211-251, with
// the star flux in its closed form). The reference forms F_K + S_K (U*_K - U_K)
// per component from the two sides' full flux vectors; with
//   a = rho_K (S_K - u_K), k = a / (S_K - S*), p* = p_K + a (S* - u_K)
// that is the upwind form  mass k S*, momentum (k S*) S* + p*, transverse
// (k S*) v_K, energy S* (E* + p*), species (k S*) Y_K: the same flux in about
// half the operations and without the cancellation of the difference. A
// supersonic face is the same expressions with u_K, p_K, E_K in place of the
// star state, so no branch separates the three cases. E / rho and the
// enthalpy come from p / rho, the Roe weights from one square root of the
// density ratio. The HLL blend of the shock sensor needs both sides' flux
// vectors and runs on the faces that have it only. With the packed limiter and
// the range test of the sensor: stage 1 of a plain 2048x768 grid 54.0 -> 44.4
// warp instructions per cell, 106.7 -> 93.4 us; the step of a plain 4096x1536
// grid 0.776 -> 0.679 ms, of the viscous plume 512x192 24.6 -> 22.9 us. Error
// against a 64-bit run of the scheme unchanged.
RN_DEV Flux hllc(const Side& L, const Side& R, float hllw) {
  const float4 WLw = L.w, WLs = L.s, WRw = R.w, WRs = R.s;
  const float rL = WLw.x, uL = WLw.y, vL = WLw.z, pL = WLw.w, GL = WLs.z;
  const float rR = WRw.x, uR = WRw.y, vR = WRw.z, pR = WRw.w, GR = WRs.z;
  const float irL = rcp(rL), irR = rcp(rR);
  const float gL = pL * irL, gR = pR * irR;                       // p / rho
  const float cL = sqrtf(gL + fdiv(gL, GL)), cR = sqrtf(gR + fdiv(gR, GR));
  const float eL = gL * GL + 0.5f * (uL * uL + vL * vL);          // E / rho
  const float eR = gR * GR + 0.5f * (uR * uR + vR * vR);
  // Roe weights sqrt(rho_K) / (sqrt(rho_L) + sqrt(rho_R))
  const float q = sqrtf(rR * irL), wL = rcp(1.0f + q), wR = q * wL;
  const float uT = wL * uL + wR * uR, vT = wL * vL + wR * vR, GT = wL * GL + wR * GR;
  const float HT = wL * (eL + gL) + wR * (eR + gR);
  const float cT = sqrtf(fmaxf(fdiv(HT - 0.5f * (uT * uT + vT * vT), GT), 1e-12f));
  const float SL = fminf(uL - cL, uT - cT), SR = fmaxf(uR + cR, uT + cT);
  const float aL = rL * (SL - uL), aR = rR * (SR - uR);
  const float Ss = fdiv(pR - pL + uL * aL - uR * aR, aL - aR);
  const bool left = SL >= 0.0f || (SR > 0.0f && Ss >= 0.0f);
  const float rK = left ? rL : rR, uK = left ? uL : uR, vK = left ? vL : vR, pK = left ? pL : pR;
  const float eK = left ? eL : eR, SK = left ? SL : SR, aK = left ? aL : aR, GK = left ? GL : GR;
  const bool super = left ? SL >= 0.0f : SR <= 0.0f;
  const float dU = Ss - uK, iS = rcp(SK - Ss), kk = aK * iS, d = dU * iS;
  const float Us = super ? uK : Ss;
  const float m = super ? rK * uK : kk * Ss;
  const float pp = super ? pK : pK + aK * dU;
  const float EE = super ? rK * eK : kk * (eK + dU * Ss) + d * pK;
  const float uf = super ? uK : uK + SK * d;
  float F0 = m, F1 = m * Us + pp, F2 = m * vK, F3 = Us * (EE + pp);
  float Y0 = m * (left ? WLs.x : WRs.x), Y1 = m * (left ? WLs.y : WRs.y), Y2 = m * (left ? WLs.w : WRs.w);
  if (hllw != 0.0f && !super) {
    const float inv = rcp(SR - SL), SLR = SL * SR * inv, fl = SR * inv, fr = SL * inv;
    const float mL = rL * uL, mR = rR * uR, EL = rL * eL, ER = rR * eR;
    const float xL = fl * mL - SLR * rL, xR = fr * mR - SLR * rR;  // shares of the advected quantities
    F0 = mixf(F0, fl * mL - fr * mR + SLR * (rR - rL), hllw);
    F1 = mixf(F1, fl * (mL * uL + pL) - fr * (mR * uR + pR) + SLR * (mR - mL), hllw);
    F2 = mixf(F2, vL * xL - vR * xR, hllw);
    F3 = mixf(F3, fl * uL * (EL + pL) - fr * uR * (ER + pR) + SLR * (ER - EL), hllw);
    Y0 = mixf(Y0, WLs.x * xL - WRs.x * xR, hllw);
    Y1 = mixf(Y1, WLs.y * xL - WRs.y * xR, hllw);
    Y2 = mixf(Y2, WLs.w * xL - WRs.w * xR, hllw);
  }
  Flux out;
  out.F = make_float4(F0, F1, F2, F3);
  out.Y = make_float4(Y0, Y1, uf * GK, uf);
  out.O = Y2;
  return out;
}
#else
RN_DEV Flux hllc(const Side& L, const Side& R, float hllw) {
  const float4 WLw = L.w, WLs = L.s, WRw = R.w, WRs = R.s;
  // HLLC (solver.js:211-251)
  float GL = WLs.z, GR = WRs.z;
  float rL = WLw.x, uL = WLw.y, vL = WLw.z, pL = WLw.w;
  float rR = WRw.x, uR = WRw.y, vR = WRw.z, pR = WRw.w;
  const Over per_rL = over(rL), per_rR = over(rR);
  float cL = sqrtf(per_rL((1.0f + fdiv(1.0f, GL)) * pL)), cR = sqrtf(per_rR((1.0f + fdiv(1.0f, GR)) * pR));
  float EL = pL * GL + 0.5f * rL * (uL * uL + vL * vL);
  float ER = pR * GR + 0.5f * rR * (uR * uR + vR * vR);
  float sL = sqrtf(rL), sR = sqrtf(rR);
  const Over per_s = over(sL + sR);
  float uT = per_s(sL * uL + sR * uR);
  float HT = per_s(per_rL(sL * (EL + pL)) + per_rR(sR * (ER + pR)));
  float vT = per_s(sL * vL + sR * vR);
  float GT = per_s(sL * GL + sR * GR);
  float cT = sqrtf(fmaxf(fdiv(HT - 0.5f * (uT * uT + vT * vT), GT), 1e-12f));
  float SL = fminf(uL - cL, uT - cT);
  float SR = fmaxf(uR + cR, uT + cT);
  float mL = rL * uL, mR = rR * uR;
  float FL0 = mL, FL1 = mL * uL + pL, FL2 = mL * vL, FL3 = uL * (EL + pL);
  float FR0 = mR, FR1 = mR * uR + pR, FR2 = mR * vR, FR3 = uR * (ER + pR);
  float YL0 = mL * WLs.x, YL1 = mL * WLs.y, YL2 = mL * WLs.w;
  float YR0 = mR * WRs.x, YR1 = mR * WRs.y, YR2 = mR * WRs.w;
  float F0, F1, F2, F3, Y0, Y1, Y2, uf, Gf;
  if (SL >= 0.0f) { F0 = FL0; F1 = FL1; F2 = FL2; F3 = FL3; Y0 = YL0; Y1 = YL1; Y2 = YL2; uf = uL; Gf = GL; }
  else if (SR <= 0.0f) { F0 = FR0; F1 = FR1; F2 = FR2; F3 = FR3; Y0 = YR0; Y1 = YR1; Y2 = YR2; uf = uR; Gf = GR; }
  else {
    float Ss = fdiv(pR - pL + mL * (SL - uL) - mR * (SR - uR), rL * (SL - uL) - rR * (SR - uR));
    bool left = Ss >= 0.0f;
    float rK = left ? rL : rR, uK = left ? uL : uR, vK = left ? vL : vR, pK = left ? pL : pR;
    float EK = left ? EL : ER, SK = left ? SL : SR;
    float YK0 = left ? WLs.x : WRs.x, YK1 = left ? WLs.y : WRs.y, YK2 = left ? WLs.w : WRs.w;
    float FK0 = left ? FL0 : FR0, FK1 = left ? FL1 : FR1, FK2 = left ? FL2 : FR2, FK3 = left ? FL3 : FR3;
    float FYK0 = left ? YL0 : YR0, FYK1 = left ? YL1 : YR1, FYK2 = left ? YL2 : YR2;
    float UK1 = left ? mL : mR, UK2 = rK * vK;
    const Over per_dS = over(SK - Ss);
    float kk = per_dS(rK * (SK - uK));
    float Us0 = kk * 1.0f, Us1 = kk * Ss, Us2 = kk * vK, Us3 = kk * (fdiv(EK, rK) + (Ss - uK) * (Ss + fdiv(pK, rK * (SK - uK))));
    float C0 = FK0 + SK * (Us0 - rK), C1 = FK1 + SK * (Us1 - UK1), C2 = FK2 + SK * (Us2 - UK2), C3 = FK3 + SK * (Us3 - EK);
    float CY0 = FYK0 + SK * (kk * YK0 - rK * YK0), CY1 = FYK1 + SK * (kk * YK1 - rK * YK1);
    float CY2 = FYK2 + SK * (kk * YK2 - rK * YK2);
    if (hllw != 0.0f) {
      float inv = fdiv(1.0f, SR - SL);
      float SLR = SL * SR;
      float H0 = (SR * FL0 - SL * FR0 + SLR * (rR - rL)) * inv;
      float H1 = (SR * FL1 - SL * FR1 + SLR * (mR - mL)) * inv;
      float H2 = (SR * FL2 - SL * FR2 + SLR * (rR * vR - rL * vL)) * inv;
      float H3 = (SR * FL3 - SL * FR3 + SLR * (ER - EL)) * inv;
      float HY0 = (SR * YL0 - SL * YR0 + SLR * (rR * WRs.x - rL * WLs.x)) * inv;
      float HY1 = (SR * YL1 - SL * YR1 + SLR * (rR * WRs.y - rL * WLs.y)) * inv;
      float HY2 = (SR * YL2 - SL * YR2 + SLR * (rR * WRs.w - rL * WLs.w)) * inv;
      F0 = mixf(C0, H0, hllw); F1 = mixf(C1, H1, hllw); F2 = mixf(C2, H2, hllw); F3 = mixf(C3, H3, hllw);
      Y0 = mixf(CY0, HY0, hllw); Y1 = mixf(CY1, HY1, hllw); Y2 = mixf(CY2, HY2, hllw);
    } else {
      // mix(Fc, Fhll, 0) = Fc + 0 Fhll: the HLL flux only decides the sign of
      // a zero component, so it is not computed where the sensor is quiet
      F0 = C0; F1 = C1; F2 = C2; F3 = C3;
      Y0 = CY0; Y1 = CY1; Y2 = CY2;
    }
    uf = uK + SK * (per_dS(SK - uK) - 1.0f);
    Gf = left ? GL : GR;
  }
  Flux out;
  out.F = make_float4(F0, F1, F2, F3);
  out.Y = make_float4(Y0, Y1, uf * Gf, uf);
  out.O = Y2;
  return out;
}
#endif

// The shock sensor's blend weight of a face from the pressures of its two
// cells and of their transverse neighbours (NaN where a neighbour is a wall:
// minNum/maxNum return the other operand, so the sensor takes the cell's own
// pressure there). Smooth pressure gives 0 exactly: when the six cells' range
// times hllBlend is clearly below 0.15 (the smoothstep's start) of their least,
// so is every jump ratio. The margin (0.1 against 0.15) dwarfs rounding.
RN_DEV float hll_weight(float p1, float pa1, float pb1, float p2, float pa2, float pb2, float hb) {
  const float lo = fminf(fminf(fminf(pa1, pb1), p1), fminf(fminf(pa2, pb2), p2));
  const float hi = fmaxf(fmaxf(fmaxf(pa1, pb1), p1), fmaxf(fmaxf(pa2, pb2), p2));
  if ((hi - lo) * hb < 0.1f * lo || !(hb > 0.0f)) return 0.0f;
  const float jm = fmaxf(fmaxf(jump_ratio(p1, pa1), jump_ratio(p1, pb1)), fmaxf(jump_ratio(p2, pa2), jump_ratio(p2, pb2)));
  return smoothstepf(0.15f, 0.6f, jm * hb);
}

// Flux of the face between cells 1 and 2 of a line of four cells 0..3. DIR_R
// selects the r-direction (normal velocity in .z): one instance of the code
// serves both directions, since a second copy costs more in instruction-cache
// misses than the direction's selects cost in instructions. The reconstruction
// works component by component, so only the two face states are turned into the
// face-normal frame. pa1, pb1, pa2, pb2: pressures of the transverse
// neighbours of cells 1 and 2. A negative area makes the face first order (next
// to a cut cell). Walls and first-order faces are branches that most warps
// skip, not selects that every face pays.
RN_DEV Flux face_flux(bool DIR_R, float area, float4 w0, float4 b0, float4 w1, float4 b1, float4 w2, float4 b2,
                      float4 w3, float4 b3, float pa1, float pb1, float pa2, float pb2, const rn_params& P) {
  const bool s1 = w1.x < 0.0f, s2 = w2.x < 0.0f;
  float hllw = 0.0f;
  Side L, R;
  bool ok = false;
  if (!(s1 || s2)) {
    hllw = hll_weight(w1.w, pa1, pb1, w2.w, pa2, pb2, P.hllBlend);
    if (P.order2 && area > 0.0f) {
      float4 d01 = diff4(w1, w0), d12 = diff4(w2, w1), d23 = diff4(w3, w2);
      float4 e01 = diff4(b1, b0), e12 = diff4(b2, b1), e23 = diff4(b3, b2);
      const bool s0 = w0.x < 0.0f, s3 = w3.x < 0.0f;
      if (__builtin_expect(s0 || s3, 0)) {
        // a wall neighbour is the cell's own reflection: the difference is
        // twice the normal velocity, nothing else
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s0) {
          d01 = DIR_R ? make_float4(0.f, 0.f, w1.z + w1.z, 0.f) : make_float4(0.f, w1.y + w1.y, 0.f, 0.f);
          e01 = z;
        }
        if (s3) {
          d23 = DIR_R ? make_float4(0.f, 0.f, -w2.z - w2.z, 0.f) : make_float4(0.f, -w2.y - w2.y, 0.f, 0.f);
          e23 = z;
        }
      }
      L = side_of<true>(w1, b1, half_slope4(d01, d12), half_slope4(e01, e12));
      R = side_of<false>(w2, b2, half_slope4(d12, d23), half_slope4(e12, e23));
      ok = L.w.x > 0.0f && L.w.w > 0.0f && R.w.x > 0.0f && R.w.w > 0.0f;
    }
  }
  if (__builtin_expect(!ok, 0)) {                // first order, or a wall on one side
    if (s1 && s2) {
      Flux none;
      none.F = make_float4(0.f, 0.f, 0.f, 0.f);
      none.Y = none.F;
      none.O = 0.0f;
      return none;
    }
    L.w = s1 ? w2 : w1; L.s = s1 ? b2 : b1;
    R.w = s2 ? w1 : w2; R.s = s2 ? b1 : b2;
    if (s1) { if (DIR_R) L.w.z = -L.w.z; else L.w.y = -L.w.y; }
    if (s2) { if (DIR_R) R.w.z = -R.w.z; else R.w.y = -R.w.y; }
  }
  if (DIR_R) {   // face-normal frame: normal velocity in .y
    float t;
    t = L.w.y; L.w.y = L.w.z; L.w.z = t;
    t = R.w.y; R.w.y = R.w.z; R.w.z = t;
  }
  Flux out = hllc(L, R, hllw);
  if (DIR_R) { float t = out.F.y; out.F.y = out.F.z; out.F.z = t; }   // rotate momentum back to (x, r)
  return out;
}

// wallPressure (solver.js:301-306): slip-wall pressure from the reflected Riemann problem
RN_DEV float wall_pressure(const Prim& q, float un) {
  float g = 1.0f + fdiv(1.0f, q.s.z), p = q.w.w, rho = q.w.x, c = sqrtf(fdiv(g * p, rho));
  if (un > 0.0f) {
    float a = 0.25f * (g + 1.0f) * un;
    return p + rho * un * (a + sqrtf(a * a + c * c));
  }
  float f = fmaxf(1.0f + fdiv(0.5f * (g - 1.0f) * un, c), 0.0f);
  return p * powf(f, fdiv(2.0f * g, g - 1.0f));
}

// member flux accumulation of one group member (memberFlux, solver.js:287-299)
RN_DEV void sub4(float4& L, float ae, float4 fe, float aw, float4 fw) {
  L.x -= ae * fe.x - aw * fw.x;
  L.y -= ae * fe.y - aw * fw.y;
  L.z -= ae * fe.z - aw * fw.z;
  L.w -= ae * fe.w - aw * fw.w;
}

// L of a cell whose x-faces have area ax and whose south and north faces have
// areas as_ and as_ + 1 (an uncut cell), after sub4's of both directions from
// L = 0. The fast variant takes sub4's products and sums in lane pairs: ten
// packed operations where sub4 takes 24 scalar ones. Each product a f is rounded
// and its partner fused, as sub4's are: forming the differences fe - fw and
// fn - fs first takes as many operations, but then G's update, the difference of
// its flux and G times the velocity's, came out 1.38 times as far from a 64-bit
// run (128x48 grids, 120 steps: 1.09e-6 against 7.9e-7).
RN_DEV float4 box4(float ax, float as_, float4 fw, float4 fe, float4 fs, float4 fn) {
#ifdef RN_FAST
  const float2 xw = make_float2(ax, ax), xe = make_float2(-ax, -ax);
  const float2 rs = make_float2(-as_, -as_), rn = make_float2(as_ + 1.0f, as_ + 1.0f);
  const float2 xl = madd2(xe, lo2(fe), mul2(xw, lo2(fw))), xh = madd2(xe, hi2(fe), mul2(xw, hi2(fw)));
  const float2 rl = madd2(rn, lo2(fn), mul2(rs, lo2(fs))), rh = madd2(rn, hi2(fn), mul2(rs, hi2(fs)));
  return cat4(sub2(xl, rl), sub2(xh, rh));
#else
  float4 L = make_float4(0.f, 0.f, 0.f, 0.f);
  sub4(L, ax, fe, ax, fw);
  sub4(L, as_ + 1.0f, fn, as_, fs);
  return L;
#endif
}

// GLSL_GAS (solver.js:445-450)
RN_DEV float sutherland(float TK, const rn_params& P) { return fdiv(P.gas[3] * 1.458e-6f * TK * sqrtf(TK), TK + 110.4f); }
RN_DEV float rmix(float4 s, const rn_params& P) {
  return (1.0f - s.x) * P.gas[0] + s.y * P.Rs[0] + s.w * P.Rs[1] + fmaxf(s.x - s.y - s.w, 0.0f) * P.Rs[2];
}

// FS_VCELL (solver.js:458-488) for one cell from its padded W/Wb and neighbours.
// CENTRAL (fast variant): where all four neighbours are fluid, all but a few
// cells along walls, the mean of the two one-sided differences is formed as the
// central one.
template <bool CENTRAL = false>
RN_DEV void vcell(float4 w0, float4 sc, float4 wE, float4 wW, float4 wN, float4 wS, int i, int j, float l, float dt,
                  const rn_params& P, float4& T1, float4& T2) {
  T1 = make_float4(0.f, 0.f, 0.f, 0.f);
  T2 = T1;
  if (w0.x < 0.0f) return;
  float ux, vx, ur, vr;
#ifdef RN_FAST
  if (CENTRAL && fminf(fminf(wE.x, wW.x), fminf(wN.x, wS.x)) > 0.0f) {
    ux = 0.5f * (wE.y - wW.y);
    vx = 0.5f * (wE.z - wW.z);
    ur = 0.5f * (wN.y - wS.y);
    vr = 0.5f * (wN.z - wS.z);
  } else
#endif
  {
    float fE = wE.x < 0.0f ? 0.0f : 1.0f, fW = wW.x < 0.0f ? 0.0f : 1.0f;
    float fN = wN.x < 0.0f ? 0.0f : 1.0f, fS = wS.x < 0.0f ? 0.0f : 1.0f;
    float dxn = fmaxf(fE + fW, 1.0f), drn = fmaxf(fN + fS, 1.0f);
    const Over per_dx = over(dxn), per_dr = over(drn);
    ux = per_dx(fE * (wE.y - w0.y) + fW * (w0.y - wW.y));
    vx = per_dx(fE * (wE.z - w0.z) + fW * (w0.z - wW.z));
    ur = per_dr(fN * (wN.y - w0.y) + fS * (w0.y - wS.y));
    vr = per_dr(fN * (wN.z - w0.z) + fS * (w0.z - wS.z));
  }
  float r = float(j) + 0.5f, vor = fdiv(w0.z, r);
  float div = ux + vr + vor;
  float S2 = 2.0f * (ux * ux + vr * vr + vor * vor) + (ur + vx) * (ur + vx) - 0.6666667f * div * div;
  float om = vx - ur;
  float sens = fdiv(om * om, om * om + div * div + 1e-8f);
  float Smag = sqrtf(fmaxf(S2, 0.0f)) * sens;
  float rho = w0.x, p = w0.w;
  float Rm = rmix(sc, P);
  float mu = sutherland(fdiv(p, rho * Rm) * P.gas[2], P);
  float mut = rho * l * l * Smag;
  if (float(i) < P.chamberNu[1]) mut = fmaxf(mut, rho * P.chamberNu[0]);
  T1 = make_float4(ux, ur, vx, vr);
  T2 = make_float4(fminf(mu + mut, fdiv(0.08f * rho, fmaxf(dt, 1e-9f))), fdiv((sc.z + 1.0f) * p, rho), Smag, mu);
}

// makeViscFluxShader (solver.js:499-536) for one face. (w1, s1, t1, m1) is
// the cell behind the face, (w2, s2, t2, m2) the cell the face belongs to; j
// is the face's row; DIR_R selects the r-direction (one instance for both).
RN_DEV void visc_flux(bool DIR_R, float4 w1, float4 s1, float4 t1, float4 m1, float4 w2, float4 s2, float4 t2,
                      float4 m2, int j, float4& F, float4& FY) {
  float mu = 0.5f * (m1.x + m2.x);
  float uf = 0.5f * (w1.y + w2.y), vf = 0.5f * (w1.z + w2.z);
  float ttx = 0.5f * (t1.x + t2.x), tty = 0.5f * (t1.y + t2.y), ttz = 0.5f * (t1.z + t2.z), ttw = 0.5f * (t1.w + t2.w);
  float r, ux, vx, ur, vr;
  if (DIR_R) { r = fmaxf(float(j), 0.5f); ux = ttx; vx = ttz; ur = w2.y - w1.y; vr = w2.z - w1.z; }
  else { r = float(j) + 0.5f; ux = w2.y - w1.y; vx = w2.z - w1.z; ur = tty; vr = ttw; }
  float div = ux + vr + fdiv(vf, r);
  float txr = mu * (ur + vx);
  float k = mu * 1.25f;
  if (DIR_R) {
    float trr = mu * (2.0f * vr - 0.6666667f * div);
    F = make_float4(-k * (s2.w - s1.w), -txr, -trr, -(uf * txr + vf * trr) - k * (m2.y - m1.y));
  } else {
    float txx = mu * (2.0f * ux - 0.6666667f * div);
    F = make_float4(-k * (s2.w - s1.w), -txx, -txr, -(uf * txx + vf * txr) - k * (m2.y - m1.y));
  }
  FY = make_float4(-k * (s2.x - s1.x), -k * (s2.y - s1.y), -k * (s2.z - s1.z), 0.0f);
}

}  // namespace rn
