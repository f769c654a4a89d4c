// batch_march2.cuh -- the plain and diffusive families of the served FP32
// step with two columns per lane and packed binary32 arithmetic.
//
// Same work decomposition as batch_march.cuh, but a warp owns a strip of 64
// padded columns (60 interior columns plus the 2-column halo on each side) and
// lane l holds columns 2l and 2l + 1 as the two halves of float2 registers.
// Both columns run the same instructions, so every binary32 add, multiply and
// multiply-add of the step is issued once for the pair (sm_100 packed
// FADD2 / FMUL2 / FFMA2: the one-column body is bound by instruction issue,
// not by the FMA pipe); selects, comparisons, min / max, reciprocals and
// square roots stay per column.  The pair also halves the warp shuffles per
// cell (a column's left or right neighbour is in the same lane half the
// time), the 64-bit loads and stores halve the memory instructions, and the
// halo is 4 of 64 columns instead of 4 of 32.
//
// Physics and update order are those of the one-column kernel (States.h:32-43,
// RiemannSolvers.h:7-128, Update.h:93-174 with constant gravity,
// ThermalConduction.h:36-73 with constant conductivity, Viscosity.h:27-119):
// HLL or HLLC, PCM or PLM.  Each face is solved once; a face that two bands
// share is solved by both, in code whose every operation is an explicitly
// rounded intrinsic or an exact instruction, so both get the same bits and
// the step stays exactly conservative across lanes, strips and bands.
#pragma once

#include "batch_march.cuh"

namespace fv2d {
namespace bm2 {

using bm::SimView;
using bm::WarpSim;

constexpr int STRIP = 60;  // interior columns per warp

typedef float2 f2;
struct b2 {
  bool x, y;
};

__device__ __forceinline__ f2 F2(float a) { return make_float2(a, a); }
__device__ __forceinline__ f2 operator+(f2 a, f2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ f2 operator*(f2 a, f2 b) { return __fmul2_rn(a, b); }
// a - b = b * (-1) + a: one rounding, one packed instruction
__device__ __forceinline__ f2 operator-(f2 a, f2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ f2 rcp2(f2 a) { return make_float2(__fdividef(1.f, a.x), __fdividef(1.f, a.y)); }
__device__ __forceinline__ f2 sqrt2(f2 a) { return make_float2(sqrtf(a.x), sqrtf(a.y)); }
__device__ __forceinline__ f2 min2(f2 a, f2 b) { return make_float2(fminf(a.x, b.x), fminf(a.y, b.y)); }
__device__ __forceinline__ f2 max2(f2 a, f2 b) { return make_float2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }
__device__ __forceinline__ f2 sel2(b2 c, f2 a, f2 b) { return make_float2(c.x ? a.x : b.x, c.y ? a.y : b.y); }
__device__ __forceinline__ b2 gt0(f2 a) { return b2{a.x > 0.f, a.y > 0.f}; }
__device__ __forceinline__ b2 ge0(f2 a) { return b2{a.x >= 0.f, a.y >= 0.f}; }
__device__ __forceinline__ b2 le0(f2 a) { return b2{a.x <= 0.f, a.y <= 0.f}; }

typedef S4<f2> Q2;

__device__ __forceinline__ Q2 sub(const Q2 &a, const Q2 &b) { return Q2{a.r - b.r, a.u - b.u, a.v - b.v, a.p - b.p}; }
__device__ __forceinline__ Q2 zero() { return Q2{F2(0.f), F2(0.f), F2(0.f), F2(0.f)}; }
__device__ __forceinline__ Q2 swap_uv(const Q2 &q) { return Q2{q.r, q.v, q.u, q.p}; }

// Neighbours along x of the pair (columns 2l, 2l + 1): the left one is
// (column 2l - 1 from lane l - 1, column 2l), the right one (column 2l + 1,
// column 2l + 2 from lane l + 1).
__device__ __forceinline__ f2 left(f2 a) { return make_float2(__shfl_up_sync(0xffffffffu, a.y, 1), a.x); }
__device__ __forceinline__ f2 right(f2 a) { return make_float2(a.y, __shfl_down_sync(0xffffffffu, a.x, 1)); }
__device__ __forceinline__ Q2 left(const Q2 &q) { return Q2{left(q.r), left(q.u), left(q.v), left(q.p)}; }
__device__ __forceinline__ Q2 right(const Q2 &q) { return Q2{right(q.r), right(q.u), right(q.v), right(q.p)}; }

// minmod (Update.h:77-85) of each column's left and right differences as the
// median of the two and zero: four minima and maxima a column, where the
// product's sign took two comparisons, two selects and the product (and missed
// opposite signs whose product underflows)
__device__ __forceinline__ f2 minmod2(f2 dl, f2 dr) {
  return max2(min2(dl, dr), min2(max2(dl, dr), F2(0.f)));
}
__device__ __forceinline__ Q2 slope(const Q2 &dl, const Q2 &dr) {
  return Q2{minmod2(dl.r, dr.r), minmod2(dl.u, dr.u), minmod2(dl.v, dr.v), minmod2(dl.p, dr.p)};
}
// q + half * s (Update.h:25)
__device__ __forceinline__ Q2 face(const Q2 &q, const Q2 &s, f2 half) {
  return Q2{fma2(half, s.r, q.r), fma2(half, s.u, q.u), fma2(half, s.v, q.v), fma2(half, s.p, q.p)};
}

struct Gas2 {
  f2 gamma, entho, half;
};

// RiemannSolvers.h:7-51, every candidate evaluated and selected in the
// reference's branch order, per column.
__device__ __forceinline__ void hll(const Q2 &qL, const Q2 &qR, Q2 &f, f2 &pout, const Gas2 &g) {
  const f2 rrL = rcp2(qL.r), rrR = rcp2(qR.r);
  const f2 aL = sqrt2(qL.p * g.gamma * rrL);
  const f2 aR = sqrt2(qR.p * g.gamma * rrR);
  const f2 SL = min2(qL.u - aL, qR.u - aR);
  const f2 SR = max2(qL.u + aL, qR.u + aR);
  const f2 peL = qL.p * g.entho, peR = qR.p * g.entho;
  const f2 EL = peL + (g.half * qL.r) * fma2(qL.u, qL.u, qL.v * qL.v);
  const f2 ER = peR + (g.half * qR.r) * fma2(qR.u, qR.u, qR.v * qR.v);
  const f2 ruL = qL.r * qL.u, ruR = qR.r * qR.u;
  const Q2 FL{ruL, fma2(ruL, qL.u, qL.p), ruL * qL.v, (qL.p + EL) * qL.u};
  const Q2 FR{ruR, fma2(ruR, qR.u, qR.p), ruR * qR.v, (qR.p + ER) * qR.u};
  const f2 mvL = qL.r * qL.v, mvR = qR.r * qR.v;
  const f2 uEL = fma2(g.half * fma2(ruL, ruL, mvL * mvL), rrL, peL);
  const f2 uER = fma2(g.half * fma2(ruR, ruR, mvR * mvR), rrR, peR);
  const f2 SLSR = SL * SR;
  const f2 rden = rcp2(SR - SL);
  Q2 FM;
  FM.r = fma2(SLSR, qR.r - qL.r, SR * FL.r - SL * FR.r) * rden;
  FM.u = fma2(SLSR, ruR - ruL, SR * FL.u - SL * FR.u) * rden;
  FM.v = fma2(SLSR, mvR - mvL, SR * FL.v - SL * FR.v) * rden;
  FM.p = fma2(SLSR, uER - uEL, SR * FL.p - SL * FR.p) * rden;
  const f2 pM = g.half * (qL.p + qR.p);
  const b2 lf = ge0(SL), rt0 = le0(SR);
  const b2 rt{!lf.x && rt0.x, !lf.y && rt0.y};
  f.r = sel2(lf, FL.r, sel2(rt, FR.r, FM.r));
  f.u = sel2(lf, FL.u, sel2(rt, FR.u, FM.u));
  f.v = sel2(lf, FL.v, sel2(rt, FR.v, FM.v));
  f.p = sel2(lf, FL.p, sel2(rt, FR.p, FM.p));
  pout = sel2(lf, qL.p, sel2(rt, qR.p, pM));
}

// RiemannSolvers.h:53-128: the star state of the side the reference would
// reach (u* > 0 -> left), then the final state in its branch order.  The side
// K is picked once (SL > 0 takes the left state whatever u* is), so every
// select below serves the star state and the flux (18 of them instead of 32),
// the total energy is formed for that side only, and the larger sound speed is
// the root of the larger square.
__device__ __forceinline__ void hllc(const Q2 &qL, const Q2 &qR, Q2 &f, f2 &pout, const Gas2 &g) {
  const f2 rL = qL.r, uL = qL.u, vL = qL.v, pL = qL.p;
  const f2 rR = qR.r, uR = qR.u, vR = qR.v, pR = qR.p;
  const f2 cmax = sqrt2(max2(pL * g.gamma * rcp2(rL), pR * g.gamma * rcp2(rR)));
  const f2 SL = min2(uL, uR) - cmax;
  const f2 SR = max2(uL, uR) + cmax;
  const f2 rcL = rL * (uL - SL);
  const f2 rcR = rR * (SR - uR);
  const f2 rd = rcp2(rcR + rcL);
  const f2 uS = (fma2(rcR, uR, rcL * uL) + (pL - pR)) * rd;
  const f2 pS = fma2(rcL * rcR, uL - uR, fma2(rcR, pL, rcL * pR)) * rd;
  const b2 bL = gt0(SL), sR = gt0(SR), sideL = gt0(uS);
  const b2 left{bL.x || sideL.x, bL.y || sideL.y};
  const b2 star{!bL.x && (sideL.x || sR.x), !bL.y && (sideL.y || sR.y)};
  const f2 rK = sel2(left, rL, rR);
  const f2 uK = sel2(left, uL, uR);
  const f2 sv = sel2(left, vL, vR);
  const f2 pK = sel2(left, pL, pR);
  const f2 SK = sel2(left, SL, SR);
  const f2 EK = fma2(g.half * rK, fma2(uK, uK, sv * sv), pK * g.entho);
  const f2 rd2 = rcp2(SK - uS);
  const f2 SKu = SK - uK;
  const f2 rS = (rK * SKu) * rd2;
  const f2 ES = fma2(pS, uS, SKu * EK - pK * uK) * rd2;
  const f2 sr = sel2(star, rS, rK);
  const f2 su = sel2(star, uS, uK);
  const f2 sp = sel2(star, pS, pK);
  const f2 E = sel2(star, ES, EK);
  pout = sp;
  f.r = sr * su;
  f.u = fma2(f.r, su, sp);
  f.v = f.r * sv;
  f.p = (E + sp) * su;
}

template <int RS>
__device__ __forceinline__ Q2 solve(const Q2 &qL, const Q2 &qR, const Gas2 &g, f2 &pout) {
  Q2 f;
  if constexpr (RS == RS_HLL)
    hll(qL, qR, f, pout, g);
  else
    hllc(qL, qR, f, pout, g);
  return f;
}

// pressure_of for the pair (batch_common.cuh), and its low-Mach recovery per column
__device__ __forceinline__ f2 pressure2(f2 dE, float bg_e, f2 r, f2 u, f2 v, float gm1) {
  const f2 ek = (F2(0.5f) * r) * fma2(u, u, v * v);
  return ((dE - ek) + F2(bg_e)) * F2(gm1);
}
__device__ __forceinline__ f2 pressure2_lowmach(f2 dE, float bg_e, f2 r, f2 u, f2 v, float gm1) {
  return make_float2(pressure_of(dE.x, bg_e, r.x, u.x, v.x, gm1, 1), pressure_of(dE.y, bg_e, r.y, u.y, v.y, gm1, 1));
}

// consToPrim of a stored offset pair (States.h:32-43) with the negative reset
// of checkNegatives (SimInfo.h:618-627) where the reference's Q carries it
__device__ __forceinline__ Q2 to_prim(const f2 u[4], const SimView &S) {
  f2 r = u[0] + F2(S.bg_r);
  const f2 rr = rcp2(r);
  const f2 uu = u[1] * rr, vv = u[2] * rr;
  f2 p = pressure2(u[3], S.bg_e, r, uu, vv, S.gm1);
  if (S.lowmach || fminf(fminf(r.x, r.y), fminf(p.x, p.y)) < 0.f) {
    if (S.lowmach) p = pressure2_lowmach(u[3], S.bg_e, r, uu, vv, S.gm1);
    if (!S.avg) {
      if (r.x < 0.f) r.x = 1e-8f;
      if (r.y < 0.f) r.y = 1e-8f;
      if (p.x < 0.f) p.x = 1e-8f;
      if (p.y < 0.f) p.y = 1e-8f;
    }
  }
  return Q2{r, uu, vv, p};
}

}  // namespace bm2

// What the row loop of a work item is compiled for: an Euler step without
// gravity, or anything (gravity, RK2 stages, the low-Mach recovery, decided as it
// runs).  The tests of those cases cut the loop's blocks where the compiler would
// interleave the update with the Riemann solves: KH 2048^2 x 200 13.9 ms with
// them, 13.2 without, HLL 1400^2 x 100 4.35 and 4.11.  The diffusive body is
// compiled in the second form only: its longer blocks spill without the cuts (RT
// 1024 x 3072 x 100 8.16 ms, 8.68 without).
enum { FORM_FREE = 0, FORM_ANY = 1 };

// One work item of the two-column march.  TCV: the diffusive family's body
// (constant conduction and viscosity); the plain body carries neither.
template <int RS, int RECON, bool TCV, int FORM>
__device__ __forceinline__ void march2_item(const BatchArgs &a, const WorkItem item, const bm::WarpSim &W,
                                            const int lane) {
  using namespace bm2;
  constexpr bool SLOPES = RECON != BR_PCM;
  SimView S;
  {
    float *U[2] = {bm::sim_get<float *, offsetof(SimDev, U)>(W), bm::sim_get<float *, offsetof(SimDev, U) + 8>(W)};
    const StageBuffers B = stage_buffers(U, FV2D_SIM(W, cur), FV2D_SIM(W, ts), FV2D_SIM(W, stage));
    S.src = B.src;
    S.dst = B.dst;
    S.avg = FORM == FORM_ANY && B.avg;
    S.last = FORM != FORM_ANY || B.last;
  }
  S.PL = FV2D_SIM(W, plane);
  S.Nx = FV2D_SIM(W, Nx);
  S.Ny = FV2D_SIM(W, Ny);
  S.P = FV2D_SIM(W, pitch);
  S.dt = (float)FV2D_SIM(W, dt);
  S.gamma = FV2D_SIM(W, gamma);
  S.gm1 = FV2D_SIM(W, gm1);
  S.inv_dx = FV2D_SIM(W, inv_dx);
  S.inv_dy = FV2D_SIM(W, inv_dy);
  S.gx = FV2D_SIM(W, gx);
  S.gy = FV2D_SIM(W, gy);
  S.kappa = FV2D_SIM(W, kappa);
  S.mu = FV2D_SIM(W, mu);
  S.bg_r = FV2D_SIM(W, bg_r);
  S.bg_e = FV2D_SIM(W, bg_e);
  S.bcx = FV2D_SIM(W, bcx);
  S.bcy = FV2D_SIM(W, bcy);
  S.grav = FORM == FORM_ANY ? FV2D_SIM(W, grav) : 0;
  S.tc = FV2D_SIM(W, tc);
  S.visc = FV2D_SIM(W, visc);
  S.lowmach = FORM == FORM_ANY ? FV2D_SIM(W, lowmach) : 0;
  const Gas2 gas{F2(S.gamma), F2(FV2D_SIM(W, entho)), F2(0.5f)};
  const int ntiles = FV2D_SIM(W, ntx) * FV2D_SIM(W, nty);
  const int Nx = S.Nx, Ny = S.Ny;
  const int gxl = item.tx * STRIP + 2 * lane;  // padded column of the pair's first half (even)
  // the pair a lane loads: its own (gxl + 1 < pitch: it lies in the row), or,
  // past the row's end, its last one, which never reaches an output column
  const int gld = min(gxl, (Nx + 3) & ~1);
  const bool out0 = lane >= 1 && lane < 31 && gxl - 2 < Nx;  // columns 2..61 of the strip are interior
  const bool out1 = out0 && gxl - 1 < Nx;
  const bm::XGhosts xg = out0 ? bm::x_ghosts(gxl - 2, out1, Nx, S.bcx) : bm::XGhosts{0u};
  const int band = FV2D_SIM(W, band);
  const int j0 = item.ty * band, jend = min(j0 + band, Ny);
  const f2 dtdx = F2(S.dt * S.inv_dx), dtdy = F2(S.dt * S.inv_dy);

  auto load = [&](int L, f2 u[4]) {  // padded row L, columns gxl and gxl + 1
    const long long g = (long long)L * S.P + gld;
#pragma unroll
    for (int k = 0; k < 4; ++k) u[k] = __ldg(reinterpret_cast<const float2 *>(S.src + k * S.PL + g));
  };
  const Q2 z = zero();
  auto yslope = [&](const Q2 &dl, const Q2 &dr) {
    if constexpr (SLOPES) return slope(dl, dr);
    else return z;
  };
  auto ydiff = [&](const Q2 &lo, const Q2 &hi) {
    if constexpr (SLOPES) return sub(hi, lo);
    else return z;
  };
  // x slope of a row: each column's left difference, the right one from the
  // next column
  auto xslope = [&](const Q2 &c) {
    if constexpr (SLOPES) {
      const Q2 dl = sub(c, left(c));
      return slope(dl, right(dl));
    } else {
      return z;
    }
  };
  const f2 hp5 = F2(0.5f), hm5 = F2(-0.5f);

  // The row loop of batch_march.cuh, with its four window-fill iterations
  // peeled into a prologue so that the main loop's y-face and x-face solves,
  // which are independent, share one block the compiler can interleave.
  // The prologue's rows are loaded together: row by row, each of its short
  // iterations waited for memory (KH 512^2 1.52 against 1.45 ms per 100 steps).
  // Iteration L loads padded row L and (from L = j0 + 4 on) updates row
  // C = L - 2.  Both copies of the row entry and of the y face are the same
  // functions of the same operands, and every operation in them is an explicit
  // packed intrinsic or an exact instruction (nothing is left for the compiler
  // to contract), so a face that two bands share gets bit-identical fluxes from
  // the prologue of one and the main loop of the other: the step stays exactly
  // conservative.
  // The loop is bound by instruction issue and by the latency of its chain at 16
  // warps per SM, so rare work (negative or NaN cells, the low-Mach recovery)
  // leaves it through one branch at each end, HLLC picks its side once and loads
  // need no column test: KH 2048^2 x 200, PLM + HLLC, 17.1 | 14.9 ms.
  // The window carries the primitives of rows L - 2 and L - 1 (q0, qp), the
  // y slope of row L - 2, the y flux of face C - 1/2 and the prefetched next
  // row; the conservative row C is read again at its update (an L1 hit: it
  // was loaded two iterations earlier).
  Q2 q0 = z, qp = z, h0 = z, Gm = z;
  f2 Unext[4];
  float lmax = 0.f;
  unsigned nneg = 0, nnan = 0;
  // primitives of the new row L and the y slope of row L - 1
  auto enter = [&](const f2 Un[4], Q2 &qn, Q2 &hp) {
    qn = to_prim(Un, S);
    hp = yslope(ydiff(q0, qp), ydiff(qp, qn));
  };
  // y face between rows L - 2 and L - 1
  auto yface = [&](const Q2 &hp) {
    f2 pout;
    return swap_uv(solve<RS>(swap_uv(face(q0, h0, hp5)), swap_uv(face(qp, hp, hm5)), gas, pout));
  };
  // Conduction (constant conductivity, ThermalConduction.h:36-73) and viscosity
  // (Viscosity.h:27-119): a face's heat flux and viscous terms are formed once,
  // those of an x face in the column on its right, those of a y face when the
  // march crosses it, as the cells of a face share them in the reference up to
  // the sign.  The window carries the temperature, the x span of the velocities
  // and the y face terms of row C, and row C - 1's velocities: half the
  // arithmetic, a third of the shuffles and none of the loads and conversions of
  // forming the four faces of each cell from its 3 x 3 neighbours (RT 1024 x
  // 3072, HLL, ms per 100 steps: 9.38 | 8.14; the one-column march 8.9).
  struct V2 {
    f2 u, v;
  };
  struct T2 {
    f2 u, v, e;
  };
  f2 T0 = F2(0.f), Hm = F2(0.f);
  V2 E0{F2(0.f), F2(0.f)}, um = E0;
  T2 Ym{F2(0.f), F2(0.f), F2(0.f)};
  auto temperature = [&](const Q2 &q) { return q.p * rcp2(q.r); };
  auto yheat = [&](f2 Ta, f2 Tb) { return F2(S.kappa * S.inv_dy) * (Tb - Ta); };
  auto xspan = [&](const Q2 &q) { return V2{right(q.u) - left(q.u), right(q.v) - left(q.v)}; };
  // mu times (tau_nn, tau_nt, tau . velocity) of a face from the velocities'
  // normal and transverse derivatives and their means
  auto stress = [&](f2 dndn, f2 dtdn, f2 dndt, f2 dtdt, f2 qn, f2 qt) {
    const f2 tnn = fma2(F2(4.f / 3.f), dndn, F2(-2.f / 3.f) * dtdt), tnt = dtdn + dndt;
    const f2 mu = F2(S.mu);
    return T2{mu * tnn, mu * tnt, mu * fma2(tnn, qn, tnt * qt)};
  };
  auto yvisc = [&](const V2 &Ea, const V2 &Eb) {  // between q0's row and qp's
    const f2 d = F2(S.inv_dy), c = F2(0.25f * S.inv_dx);
    const T2 t = stress(d * (qp.v - q0.v), d * (qp.u - q0.u), c * (Eb.v + Ea.v), c * (Eb.u + Ea.u), hp5 * (qp.v + q0.v),
                        hp5 * (qp.u + q0.u));
    return T2{t.v, t.u, t.e};
  };
  auto xvisc = [&]() {  // between the columns of q0's row
    const f2 d = F2(S.inv_dx), c = F2(0.25f * S.inv_dy);
    const V2 D{qp.u - um.u, qp.v - um.v}, Dw{left(D.u), left(D.v)};
    const f2 uw = left(q0.u), vw = left(q0.v);
    return stress(d * (q0.u - uw), d * (q0.v - vw), c * (D.u + Dw.u), c * (D.v + Dw.v), hp5 * (q0.u + uw),
                  hp5 * (q0.v + vw));
  };
  // jend >= j0 + 1: rows j0 to j0 + 4 are in the band's window
  f2 Ufill[4][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) load(j0 + k, Ufill[k]);
  load(j0 + 4, Unext);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int L = j0 + k;
    Q2 qn, hp;
    enter(Ufill[k], qn, hp);
    if (L == j0 + 3) Gm = yface(hp);
    if constexpr (TCV) {  // row j0 + 1's, then those of the face below it
      if (L >= j0 + 2 && S.tc) {
        const f2 Tp = temperature(qp);
        Hm = yheat(T0, Tp);
        T0 = Tp;
      }
      if (L >= j0 + 2 && S.visc) {
        const V2 Ep = xspan(qp);
        Ym = yvisc(E0, Ep);
        E0 = Ep;
        um = V2{q0.u, q0.v};
      }
    }
    q0 = qp;
    qp = qn;
    h0 = hp;
  }
  for (int L = j0 + 4; L < jend + 4; ++L) {
    const int C = L - 2;
    const int j = C - 2;
    f2 U0[4];
    load(C, U0);
    const f2 Un[4] = {Unext[0], Unext[1], Unext[2], Unext[3]};
    if (L + 1 < jend + 4) load(L + 1, Unext);
    Q2 qn, hp;
    enter(Un, qn, hp);
    const Q2 Gp = yface(hp);  // face between rows C and C + 1
    {
      // x faces of row C: the pair solves faces 2l - 1/2 and 2l + 1/2
      const Q2 hx = xslope(q0);
      f2 poutX;
      const Q2 Fw = solve<RS>(left(face(q0, hx, hp5)), face(q0, hx, hm5), gas, poutX);
      const Q2 Fe = right(Fw);

      // update in the reference's order: x flux, x gravity, y flux, y
      // gravity, conduction, viscosity (Update.h:114-168, 176-191)
      f2 un[4];
      un[0] = fma2(Fw.r - Fe.r, dtdx, U0[0]);
      un[1] = fma2(Fw.u - Fe.u, dtdx, U0[1]);
      un[2] = fma2(Fw.v - Fe.v, dtdx, U0[2]);
      un[3] = fma2(Fw.p - Fe.p, dtdx, U0[3]);
      const f2 dt2 = F2(S.dt);
      if (S.grav) {
        un[2] = fma2(dt2 * q0.r, F2(S.gx), un[2]);
        un[3] = fma2(dt2 * (hp5 * (Fw.r + Fe.r)), F2(S.gx), un[3]);
      }
      un[0] = fma2(Gm.r - Gp.r, dtdy, un[0]);
      un[1] = fma2(Gm.u - Gp.u, dtdy, un[1]);
      un[2] = fma2(Gm.v - Gp.v, dtdy, un[2]);
      un[3] = fma2(Gm.p - Gp.p, dtdy, un[3]);
      if (S.grav) {
        un[2] = fma2(dt2 * q0.r, F2(S.gy), un[2]);
        un[3] = fma2(dt2 * (hp5 * (Gm.r + Gp.r)), F2(S.gy), un[3]);
      }
      if constexpr (TCV) {
        if (S.tc) {
          const f2 Tp = temperature(qp);
          const f2 Hp = yheat(T0, Tp);
          const f2 Hw = F2(S.kappa * S.inv_dx) * (T0 - left(T0));  // x faces as above: the pair's west ones
          un[3] = un[3] + fma2(dtdx, right(Hw) - Hw, dtdy * (Hp - Hm));
          T0 = Tp;
          Hm = Hp;
        }
        if (S.visc) {
          const V2 Ep = xspan(qp);
          const T2 Yp = yvisc(E0, Ep);
          const T2 Xw = xvisc();
          const f2 f1 = (right(Xw.u) - Xw.u) + (Yp.u - Ym.u);
          const f2 f2_ = (right(Xw.v) - Xw.v) + (Yp.v - Ym.v);
          const f2 f3 = (right(Xw.e) - Xw.e) + (Yp.e - Ym.e);
          un[1] = fma2(f1, dt2, un[1]);
          un[2] = fma2(f2_, dt2, un[2]);
          un[3] = fma2(f3, dt2, un[3]);
          E0 = Ep;
          Ym = Yp;
          um = V2{q0.u, q0.v};
        }
      }

      if (out0) {
        const long long g = (long long)C * S.P + gxl;
        if (S.avg) {  // SSP-RK2: 0.5 (U^n + U**) (Update.h:214-220), offsets alike
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float *d = S.dst + k * S.PL + g;
            const f2 o = out1 ? *reinterpret_cast<const float2 *>(d) : make_float2(d[0], 0.f);
            un[k] = hp5 * (o + un[k]);
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float *d = S.dst + k * S.PL + g;
          if (out1)
            *reinterpret_cast<float2 *>(d) = un[k];
          else
            d[0] = un[k].x;
        }
        if (S.last) {
          // primitive state of the new cells for the next dt; the negative
          // and NaN guards leave the common path through one test
          const f2 r = un[0] + F2(S.bg_r);
          const f2 rr = rcp2(r);
          const f2 u = un[1] * rr, v = un[2] * rr;
          f2 p = pressure2(un[3], S.bg_e, r, u, v, S.gm1);
          f2 cs2 = p * F2(S.gamma) * rr;
          // a NaN of any field reaches the pressure
          if (S.lowmach || !(min_nan(min_nan(r.x, p.x), min_nan(r.y, p.y)) >= 0.f)) {
            if (S.lowmach) p = pressure2_lowmach(un[3], S.bg_e, r, u, v, S.gm1);
            auto guard = [&](float rh, float ph, float rrh, float &c2) {
              nnan += is_nan_f(ph);
              nneg += (rh < 0.f) + (ph < 0.f);
              c2 = (ph < 0.f ? 1e-8f : ph) * S.gamma * (rh < 0.f ? __fdividef(1.f, 1e-8f) : rrh);
            };
            guard(r.x, p.x, rr.x, cs2.x);
            if (out1) guard(r.y, p.y, rr.y, cs2.y);
          }
          const f2 cs = sqrt2(cs2);
          const f2 cu = make_float2(cs.x + fabsf(u.x), cs.y + fabsf(u.y));
          const f2 cv = make_float2(cs.x + fabsf(v.x), cs.y + fabsf(v.y));
          const f2 ih = fma2(cu, F2(S.inv_dx), cv * F2(S.inv_dy));
          lmax = fmaxf(lmax, fmaxf(ih.x, out1 ? ih.y : 0.f));  // NaN never enters
        } else {
          nnan += is_nan_f(min_nan(min_nan(un[0].x, un[1].x), min_nan(un[2].x, un[3].x)));
          if (out1) nnan += is_nan_f(min_nan(min_nan(un[0].y, un[1].y), min_nan(un[2].y, un[3].y)));
        }
        // ghost copies (BoundaryConditions.h:82-147, inverse map): the pair's
        // row, then, for rows whose ghosts copy it, each of those rows
        const bool ey = j < 2 || j >= Ny - 2;
        if (ey || xg.any()) {
#pragma unroll 1
          for (int t = ey ? 0 : 4; t < 5; ++t) {
            int ty = j;
            bool flip = false;
            if (t < 4) {
              ty = t < 2 ? t - 2 : Ny + t - 2;
              if (ghost_source(ty, Ny, S.bcy, &flip) != j) continue;
            }
            float *row = S.dst + (long long)(ty + 2) * S.P;
#pragma unroll
            for (int k = 0; k < 4; ++k, row += S.PL) {
              f2 x = un[k];
              if (k == 2 && flip) x = make_float2(-x.x, -x.y);
              if (t < 4) {
                if (out1) *reinterpret_cast<float2 *>(row + gxl) = x;
                else row[gxl] = x.x;
              }
              if (k == 1 && S.bcx == 1) x = make_float2(-x.x, -x.y);  // reflecting
              if (xg.any()) row[xg.a()] = xg.ha() ? x.y : x.x;
              if (xg.two()) row[xg.b()] = xg.hb() ? x.y : x.x;
            }
          }
        }
      }
    }

    // advance the window
    q0 = qp;
    qp = qn;
    h0 = hp;
    Gm = Gp;
  }

  // item reductions and the per-simulation commit
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
  const unsigned wn = __reduce_add_sync(0xffffffffu, nneg);
  const unsigned wnan = __reduce_add_sync(0xffffffffu, nnan);
  if (lane == 0) {
    SimDev *Gw = a.sims + item.sim;
    if (S.last) atomicMax(&Gw->acc_bits, __float_as_uint(lmax));
    if (wn) atomicAdd(&Gw->negatives, (unsigned long long)wn);
    if (wnan) atomicAdd(&Gw->nan_cells, wnan);
    __threadfence();
    const unsigned t = atomicAdd(&Gw->ticket, 1u);
    if (t == (unsigned)ntiles - 1u) commit_stage(Gw);
  }
}

template <bool TCV, int FORM>
__device__ __forceinline__ void march2_form(const BatchArgs &a, const WorkItem item, const bm::WarpSim &W,
                                            const int lane) {
  const bool plm = FV2D_SIM(W, recon) == BR_PLM;
  if (FV2D_SIM(W, rs) == RS_HLL) {
    if (plm)
      march2_item<RS_HLL, BR_PLM, TCV, FORM>(a, item, W, lane);
    else
      march2_item<RS_HLL, BR_PCM, TCV, FORM>(a, item, W, lane);
  } else {
    if (plm)
      march2_item<RS_HLLC, BR_PLM, TCV, FORM>(a, item, W, lane);
    else
      march2_item<RS_HLLC, BR_PCM, TCV, FORM>(a, item, W, lane);
  }
}

// The plain (TCV false) or diffusive (TCV true) family with two columns per
// lane: HLL / HLLC x PCM / PLM.  A request of the other family never enters
// (the service keeps the families in separate lanes); if one did, it would
// fail rather than run without its conduction and viscosity.
template <int NT, int MINB, bool TCV>
__global__ void __launch_bounds__(NT, MINB) batch_march2_kernel(const BatchArgs a) {
  const int lane = threadIdx.x & 31;
  const int nwarps = gridDim.x * (NT / 32);
  const int nw = *a.n_work;
  for (int w = blockIdx.x * (NT / 32) + (threadIdx.x >> 5); w < nw; w += nwarps) {
    const WorkItem item = a.work[w];
    const bm::WarpSim W = bm::load_sim(a.sims + item.sim, lane);
    if (FV2D_SIM(W, status) != SIM_ACTIVE) continue;
    if (!TCV && (FV2D_SIM(W, tc) || FV2D_SIM(W, visc))) {
      if (lane == 0) {  // fail the request through its commit, like a wait that gave up
        SimDev *Gw = a.sims + item.sim;
        atomicOr(&Gw->dev_err, (unsigned)BATCH_ERR_FAMILY);
        __threadfence();
        const unsigned t = atomicAdd(&Gw->ticket, 1u);
        if (t == (unsigned)(FV2D_SIM(W, ntx) * FV2D_SIM(W, nty)) - 1u) commit_stage(Gw);
      }
      __syncwarp();
      continue;
    }
    if (TCV || FV2D_SIM(W, ts) != 0 || FV2D_SIM(W, lowmach) || FV2D_SIM(W, grav))
      march2_form<TCV, FORM_ANY>(a, item, W, lane);
    else
      march2_form<TCV, TCV ? FORM_ANY : FORM_FREE>(a, item, W, lane);
    __syncwarp();
  }
}

}  // namespace fv2d
