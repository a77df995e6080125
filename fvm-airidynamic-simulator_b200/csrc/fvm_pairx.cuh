// fvm_pairx.cuh -- what a stage-kernel thread evaluates per step, in packed
// FP32x2 arithmetic: the two x-faces (same column, rows r and r+1), the two
// y-faces (r-2 | r-1) and (r-1 | r), and the update of rows r-2 and r-1.
//
// sm_100 issues two FP32 adds, multiplies or FMAs per instruction
// (__fadd2_rn / __fmul2_rn / __ffma2_rn) at the same FMA throughput as the
// scalar forms, so packing saves issue slots, which is what the stage kernels
// are bound by.  The primitive ring stores each row pair interleaved, {rho_r,
// rho_r+1, u_r, u_r+1} and {v_r, v_r+1, p_r, p_r+1}, so one shared-memory
// vector load yields both rows' operands as aligned register pairs and no
// register moves are needed; lane .x is row r, lane .y row r+1.  The y-faces'
// upper cells straddle two row pairs and are paired from those loads.
// Square roots, reciprocals, min/max and the wave-fan selections stay per
// lane.
//
// The faces are those of the reference's computeFluxesKernel
// (src/solver.cu:1502-1598 / :1601-1682) with its HLLC (:1112-1223 /
// :1315-1430) or AUSM+, the update that of updateKernel (:1736-1875), with
// explicit fused multiply-adds and one approximate reciprocal per shared
// divisor, so results can differ from the reference's in the last bits.  The
// x-face ring stores each row pair interleaved as well, so the update's flux
// differences come out of vector loads as register pairs.
#pragma once
#include "fvm_math.cuh"

namespace fvm {

using f2 = float2;

__device__ __forceinline__ f2 mk2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ f2 splat(float a) { return make_float2(a, a); }
__device__ __forceinline__ f2 p_add(f2 a, f2 b) { return __fadd2_rn(a, b); }
// a - b as a + b*(-1): one rounding, the value of a subtraction
__device__ __forceinline__ f2 p_sub(f2 a, f2 b) { return __ffma2_rn(b, splat(-1.0f), a); }
__device__ __forceinline__ f2 p_mul(f2 a, f2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ f2 p_fma(f2 a, f2 b, f2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ f2 p_min(f2 a, f2 b) { return mk2(fminf(a.x, b.x), fminf(a.y, b.y)); }
__device__ __forceinline__ f2 p_max(f2 a, f2 b) { return mk2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }
__device__ __forceinline__ f2 p_max(f2 a, float b) { return mk2(fmaxf(a.x, b), fmaxf(a.y, b)); }
__device__ __forceinline__ f2 p_sqrt(f2 a) { return mk2(sqrtf(a.x), sqrtf(a.y)); }
// per-lane approximate reciprocal, shared by quotients with one divisor
__device__ __forceinline__ f2 p_rcp(f2 a) { return mk2(rcp_approx(a.x), rcp_approx(a.y)); }
// division a / b in the fast approximate form the scalar path uses
// (__fdividef: a times the approximate reciprocal of b, flushed to zero for
// |b| > 2^126), with the two products packed into one instruction
__device__ __forceinline__ f2 p_div(f2 a, f2 b) { return p_mul(a, p_rcp(b)); }
// per-lane approximate reciprocal square root
__device__ __forceinline__ f2 p_rsqrt(f2 a) { return mk2(rsqrtf(a.x), rsqrtf(a.y)); }
__device__ __forceinline__ f2 p_sel(bool cx, bool cy, f2 a, f2 b) { return mk2(cx ? a.x : b.x, cy ? a.y : b.y); }

// Half the limited slope per lane, (q_i+1/2 - q_i) of the reconstruction:
// minmod (src/solver.cu:110-150) or the van Leer harmonic mean.  The limiters'
// own factors absorb the half: 0.25 (sign + sign) min, and ab / (a + b).
template <int LIM>
__device__ __forceinline__ f2 p_half_slope(f2 qm1, f2 q0, f2 qp1) {
    const f2 dL = p_sub(q0, qm1), dR = p_sub(qp1, q0);
    if (LIM == 0) {
        const f2 s = p_add(mk2(copysignf(0.25f, dL.x), copysignf(0.25f, dL.y)),
                           mk2(copysignf(0.25f, dR.x), copysignf(0.25f, dR.y)));
        return p_mul(s, mk2(fminf(fabsf(dL.x), fabsf(dR.x)), fminf(fabsf(dL.y), fabsf(dR.y))));
    } else {
        const f2 ab = p_mul(dL, dR);
        const f2 q = p_div(ab, p_add(dL, dR));
        return mk2(ab.x > 0.0f ? q.x : 0.0f, ab.y > 0.0f ? q.y : 0.0f);
    }
}

// Primitive states of one column for a row pair: lane .x row r, lane .y row r+1.
struct PairPrim {
    f2 rho, u, v, p;
};
__device__ __forceinline__ PairPrim pair_prim(const float4 &A, const float4 &B) {
    return PairPrim{mk2(A.x, A.y), mk2(A.z, A.w), mk2(B.x, B.y), mk2(B.z, B.w)};
}

// Half limited slopes of a cell pair in the face frame: normal and tangential
// velocity components (x-faces: u, v; y-faces: v, u).
struct PairSl {
    f2 rho, n, t, p;
};

// HLLC flux of a face pair with Roe-averaged Davis wave speeds (src/solver.cu:
// 1112-1223 / :1315-1430) from the reconstructed states, the reference's
// expressions; F[0..3] = mass, x-, y-momentum, energy, F[4] = the upwinded
// rho_e flux.
template <bool XDIR>
__device__ __forceinline__ void hllc_pair(const f2 &rL, const f2 &nL, const f2 &tL, const f2 &pL, const f2 &rR,
                                          const f2 &nR, const f2 &tR, const f2 &pR, f2 F[5]) {
    const f2 hp = splat(0.5f);
    // E = p/(gamma-1) + rho*(u^2 + v^2)/2, the x component squared first
    const f2 igm1 = splat(1.0f / (GAMMA - 1.0f));
    const f2 eL = p_mul(pL, igm1), eR = p_mul(pR, igm1);
    const f2 qL = XDIR ? p_fma(nL, nL, p_mul(tL, tL)) : p_fma(tL, tL, p_mul(nL, nL));
    const f2 qR = XDIR ? p_fma(nR, nR, p_mul(tR, tR)) : p_fma(tR, tR, p_mul(nR, nR));
    const f2 EL = p_fma(p_mul(hp, rL), qL, eL);
    const f2 ER = p_fma(p_mul(hp, rR), qR, eR);

    // ---- HLLC with Roe-averaged Davis wave speeds; quotients that share a
    // divisor (1/rho of each side, the Roe weight sum, the star-state
    // denominator) multiply by one reciprocal
    // one reciprocal square root per side gives sqrt(rho) = rho / sqrt(rho)
    // and 1/rho = (1/sqrt(rho))^2
    const f2 rqL = p_rsqrt(rL), rqR = p_rsqrt(rR);
    const f2 sqL = p_mul(rL, rqL), sqR = p_mul(rR, rqR);
    const f2 irL = p_mul(rqL, rqL), irR = p_mul(rqR, rqR);
    const f2 cL = p_sqrt(p_mul(p_mul(splat(GAMMA), pL), irL));
    const f2 cR = p_sqrt(p_mul(p_mul(splat(GAMMA), pR), irR));
    // (the densities are >= MIN_DENSITY, so the reference's 1e-10 in this
    // divisor is below half its last bit: left out, bit for bit the same)
    const f2 iden = p_rcp(p_add(sqL, sqR));
    const f2 un_roe = p_mul(p_fma(sqL, nL, p_mul(sqR, nR)), iden);
    const f2 ut_roe = p_mul(p_fma(sqL, tL, p_mul(sqR, tR)), iden);
    const f2 HL = p_mul(p_add(EL, pL), irL), HR = p_mul(p_add(ER, pR), irR);
    const f2 H_roe = p_mul(p_fma(sqL, HL, p_mul(sqR, HR)), iden);
    const f2 q_roe = XDIR ? p_fma(un_roe, un_roe, p_mul(ut_roe, ut_roe)) : p_fma(ut_roe, ut_roe, p_mul(un_roe, un_roe));
    const f2 c2 = p_mul(splat(GAMMA - 1.0f), p_fma(splat(-0.5f), q_roe, H_roe));
    const f2 c_avg = p_mul(hp, p_add(cL, cR));
    const f2 c_roe = mk2(c2.x > 0.0f ? sqrtf(c2.x) : c_avg.x, c2.y > 0.0f ? sqrtf(c2.y) : c_avg.y);
    f2 SL = p_min(p_sub(nL, cL), p_sub(un_roe, c_roe));
    f2 SR = p_max(p_add(nR, cR), p_add(un_roe, c_roe));
    const f2 delta = p_mul(splat(ENTROPY_FIX), p_max(cL, cR));
    SL = mk2(fabsf(SL.x) < delta.x ? -delta.x : SL.x, fabsf(SL.y) < delta.y ? -delta.y : SL.y);
    SR = mk2(fabsf(SR.x) < delta.x ? delta.x : SR.x, fabsf(SR.y) < delta.y ? delta.y : SR.y);
    const f2 aL = p_sub(SL, nL), aR = p_sub(SR, nR);
    const f2 mL = p_mul(rL, aL), mR = p_mul(rR, aR);
    // m_L - m_R < 0 always (S_L <= u_L - c_L, S_R >= u_R + c_R), so the
    // reference's floor of its magnitude is a minimum
    const f2 ds = p_sub(mL, mR);
    const f2 sds = mk2(fminf(ds.x, -1e-10f), fminf(ds.y, -1e-10f));
    const f2 Ss = p_div(p_sub(p_fma(mL, nL, p_sub(pR, pL)), p_mul(mR, nR)), sds);
    // upwind side K of the wave fan: the left state if all waves or the contact
    // move right, else the right one (the reference branches four ways)
    const bool supL0 = SL.x >= 0.0f, supL1 = SL.y >= 0.0f;
    const bool supR0 = !supL0 && SR.x <= 0.0f, supR1 = !supL1 && SR.y <= 0.0f;
    const bool useL0 = supL0 || (!supR0 && Ss.x >= 0.0f), useL1 = supL1 || (!supR1 && Ss.y >= 0.0f);
    const f2 rK = p_sel(useL0, useL1, rL, rR), nK = p_sel(useL0, useL1, nL, nR), tK = p_sel(useL0, useL1, tL, tR);
    const f2 pK = p_sel(useL0, useL1, pL, pR), EK = p_sel(useL0, useL1, EL, ER), SK = p_sel(useL0, useL1, SL, SR);
    const f2 d = p_sub(SK, nK);   // SK - unK
    const f2 rkd = p_mul(rK, d);  // rK (SK - unK): the same product as mL / mR
    const f2 fK0 = p_mul(rK, nK);
    const f2 fK1 = p_fma(fK0, nK, pK);
    const f2 fK2 = XDIR ? p_mul(fK0, tK) : p_mul(p_mul(rK, tK), nK);  // (rho u) v either way
    const f2 fK3 = p_mul(p_add(EK, pK), nK);
    // |S_K - S*| floored at 1e-10 with its sign (the reference's
    // `cd >= 0 ? 1e-10 : -1e-10`; S_K is never zero after the entropy fix,
    // so the difference is never -0)
    f2 cd = p_sub(SK, Ss);
    cd = mk2(copysignf(fmaxf(fabsf(cd.x), 1e-10f), cd.x), copysignf(fmaxf(fabsf(cd.y), 1e-10f), cd.y));
    const f2 icd = p_rcp(cd);
    const f2 rs = p_max(p_mul(rkd, icd), MIN_DENSITY);
    const f2 ps = p_max(p_fma(rkd, p_sub(Ss, nK), pK), MIN_PRESSURE);
    const f2 Es = p_mul(p_sub(p_fma(EK, d, p_mul(ps, Ss)), p_mul(pK, nK)), icd);
    // star region: F = F_K + S_K (U*_K - U_K); supersonic: F = F_K, written
    // as F_K + 0 * (U*_K - U_K) (there the wave fan keeps |ds| >= rho c, so
    // the star quantities are finite and the product is exactly zero)
    const bool st0 = !(supL0 || supR0), st1 = !(supL1 || supR1);
    const f2 SKs = p_sel(st0, st1, SK, splat(0.0f));
    F[0] = p_fma(SKs, p_sub(rs, rK), fK0);
    F[XDIR ? 1 : 2] = p_fma(SKs, p_sub(p_mul(rs, Ss), fK0), fK1);
    F[XDIR ? 2 : 1] = p_fma(SKs, p_mul(p_sub(rs, rK), tK), fK2);
    F[3] = p_fma(SKs, p_sub(Es, EK), fK3);
    // upwinded internal-energy flux
    const f2 uf = p_add(nL, nR);  // sign of 0.5 (unL + unR)
    F[4] = p_sel(uf.x >= 0.0f, uf.y >= 0.0f, p_mul(eL, nL), p_mul(eR, nR));
}

// Mach numbers clamped to [-1, 1]; a NaN stays one, so that the update of a
// cell with a non-finite neighbour still sees a non-finite flux and rolls back.
__device__ __forceinline__ f2 mach_clamped(f2 M) {
    return mk2(fabsf(M.x) >= 1.0f ? copysignf(1.0f, M.x) : M.x, fabsf(M.y) >= 1.0f ? copysignf(1.0f, M.y) : M.y);
}

// AUSM+ flux of a face pair (Liou 1996, J. Comput. Phys. 129:364-382; no
// reference counterpart): interface sound speed from the critical sound
// speeds, split Mach numbers of degree 4 (beta = 1/8), split pressures of
// degree 5 (alpha = 3/16).  The split polynomials are evaluated at the Mach
// number clamped to [-1, 1], where they end in exactly 0 and 1; the split Mach
// number of a supersonic side adds what was clamped off (exact: M - 1 and
// 1 + (M - 1) do not round for M >= 1).  The upwind sum keeps both sides (one
// mass flux is zero): packed multiplies instead of selects.  Measured on the
// 2048x1024 vortex street, stage 1 / stage 2: 62.3 / 62.5 us with one scalar
// evaluation per lane, 53.2 / 53.1 us packed.
template <bool XDIR>
__device__ __forceinline__ void ausm_plus_pair(const f2 &rL, const f2 &nL, const f2 &tL, const f2 &pL, const f2 &rR,
                                               const f2 &nR, const f2 &tR, const f2 &pR, f2 F[5]) {
    const f2 half = splat(0.5f), one = splat(1.0f), quarter = splat(0.25f), eighth = splat(0.125f);
    const f2 igm1 = splat(1.0f / (GAMMA - 1.0f));
    const f2 eL = p_mul(pL, igm1), eR = p_mul(pR, igm1);
    const f2 qL = XDIR ? p_fma(nL, nL, p_mul(tL, tL)) : p_fma(tL, tL, p_mul(nL, nL));
    const f2 qR = XDIR ? p_fma(nR, nR, p_mul(tR, tR)) : p_fma(tR, tR, p_mul(nR, nR));
    const f2 HL = p_mul(p_add(p_fma(p_mul(half, rL), qL, eL), pL), p_rcp(rL));
    const f2 HR = p_mul(p_add(p_fma(p_mul(half, rR), qR, eR), pR), p_rcp(rR));
    const f2 kcrit = splat(2.0f * (GAMMA - 1.0f) / (GAMMA + 1.0f));
    const f2 sL = p_sqrt(p_mul(kcrit, HL)), sR = p_sqrt(p_mul(kcrit, HR));
    const f2 c = p_min(p_div(p_mul(sL, sL), p_max(sL, nL)), p_div(p_mul(sR, sR), p_max(sR, mk2(-nR.x, -nR.y))));
    const f2 ic = p_rcp(c);
    const f2 ML = p_mul(nL, ic), MR = p_mul(nR, ic);
    const f2 cl = mach_clamped(ML), cr = mach_clamped(MR);
    // M+ = (M+1)^2/4 + (M^2-1)^2/8, P+ = (M+1)^2 (2-M)/4 + 3/16 M (M^2-1)^2
    const f2 al = p_add(cl, one), bl = p_fma(cl, cl, splat(-1.0f));
    const f2 al4 = p_mul(quarter, al);
    const f2 mp = p_add(p_fma(al4, al, p_mul(p_mul(eighth, bl), bl)), p_max(p_sub(ML, one), 0.0f));
    const f2 pp = p_fma(p_mul(al4, al), p_fma(cl, splat(-1.0f), splat(2.0f)),
                        p_mul(p_mul(p_mul(splat(0.1875f), cl), bl), bl));
    // M- = -(M-1)^2/4 - (M^2-1)^2/8, P- = (M-1)^2 (2+M)/4 - 3/16 M (M^2-1)^2
    const f2 ar = p_sub(cr, one), br = p_fma(cr, cr, splat(-1.0f));
    const f2 ar4 = p_mul(quarter, ar);
    const f2 mm = p_sub(p_min(p_add(MR, one), splat(0.0f)), p_fma(ar4, ar, p_mul(p_mul(eighth, br), br)));
    const f2 pm = p_fma(p_mul(ar4, ar), p_add(cr, splat(2.0f)), p_mul(p_mul(p_mul(splat(-0.1875f), cr), br), br));
    const f2 m12 = p_add(mp, mm);
    const f2 p12 = p_fma(pm, pR, p_mul(pp, pL));
    // mass fluxes taken from the left and from the right cell
    const f2 hc = p_mul(half, c), am = mk2(fabsf(m12.x), fabsf(m12.y));
    const f2 fl = p_mul(p_mul(hc, p_add(m12, am)), rL), fr = p_mul(p_mul(hc, p_sub(m12, am)), rR);
    F[0] = p_add(fl, fr);
    F[XDIR ? 1 : 2] = p_add(p_fma(fl, nL, p_mul(fr, nR)), p12);
    F[XDIR ? 2 : 1] = p_fma(fl, tL, p_mul(fr, tR));
    F[3] = p_fma(fl, HL, p_mul(fr, HR));
    // upwinded internal-energy flux
    const f2 uf = p_add(nL, nR);  // sign of 0.5 (unL + unR)
    F[4] = p_sel(uf.x >= 0.0f, uf.y >= 0.0f, p_mul(eL, nL), p_mul(eR, nR));
}

// Two faces between cells a | b (lane .x: face 0, lane .y: face 1) from the
// cells' primitives and half limited slopes sa, sb (face frame); F = {mass,
// x-momentum, y-momentum, energy, rho_e}, each a lane pair.  `m` holds the
// mask bytes of the two faces' owner cells, lane .x in bits 0-7, lane .y in
// bits 8-15.  First-order faces (a wall at the outer stencil cells, a density
// below LOW_DENSITY) and wall faces are rare and touch few warps, so they sit
// behind branches; with selects on every face the ALU pipe, which no packed
// form relieves, was the stage kernels' busiest.  With the update's rollback
// and cap and the boundary conditions behind branches too: stage 1 / stage 2
// 695 / 696 -> 647 / 672 us at 8192x4096 (van Leer, HLLC).
template <bool XDIR, int SCHEME>
__device__ __forceinline__ void face_pair_core(uint32_t m, const PairPrim &a, const PairSl &sa, const PairPrim &b,
                                               const PairSl &sb, f2 F[5]) {
    constexpr uint32_t V = XDIR ? MB_XV : MB_YV, N = XDIR ? MB_XN : MB_YN;
    PairSl la = sa, lb = sb;
    if ((m & (N * 0x0101u)) != 0u ||
        fminf(fminf(a.rho.x, a.rho.y), fminf(b.rho.x, b.rho.y)) < LOW_DENSITY) {
        const bool fo0 = (m & N) != 0u || a.rho.x < LOW_DENSITY || b.rho.x < LOW_DENSITY;
        const bool fo1 = (m & (N << 8)) != 0u || a.rho.y < LOW_DENSITY || b.rho.y < LOW_DENSITY;
        const f2 om = mk2(fo0 ? 0.0f : 1.0f, fo1 ? 0.0f : 1.0f);  // order mask
        la = PairSl{p_mul(sa.rho, om), p_mul(sa.n, om), p_mul(sa.t, om), p_mul(sa.p, om)};
        lb = PairSl{p_mul(sb.rho, om), p_mul(sb.n, om), p_mul(sb.t, om), p_mul(sb.p, om)};
    }
    const f2 an = XDIR ? a.u : a.v, at = XDIR ? a.v : a.u;
    const f2 bn = XDIR ? b.u : b.v, bt = XDIR ? b.v : b.u;
    // MUSCL: left = a + slope_a/2, right = b - slope_b/2
    const f2 rL = p_max(p_add(a.rho, la.rho), MIN_DENSITY);
    const f2 nL = p_add(an, la.n);
    const f2 tL = p_add(at, la.t);
    const f2 pL = p_max(p_add(a.p, la.p), MIN_PRESSURE);
    const f2 rR = p_max(p_sub(b.rho, lb.rho), MIN_DENSITY);
    const f2 nR = p_sub(bn, lb.n);
    const f2 tR = p_sub(bt, lb.t);
    const f2 pR = p_max(p_sub(b.p, lb.p), MIN_PRESSURE);

    if (SCHEME == 0)
        hllc_pair<XDIR>(rL, nL, tL, pL, rR, nR, tR, pR, F);
    else
        ausm_plus_pair<XDIR>(rL, nL, tL, pL, rR, nR, tR, pR, F);
    // wall faces: no mass/energy flux, normal momentum flux = pressure of the left/bottom cell
    if ((m & (V * 0x0101u)) != V * 0x0101u) {
        const bool v0 = (m & V) != 0u, v1 = (m & (V << 8)) != 0u;
        const f2 zero = splat(0.0f);
        F[0] = p_sel(v0, v1, F[0], zero);
        F[1] = p_sel(v0, v1, F[1], XDIR ? a.p : zero);
        F[2] = p_sel(v0, v1, F[2], XDIR ? zero : a.p);
        F[3] = p_sel(v0, v1, F[3], zero);
        F[4] = p_sel(v0, v1, F[4], zero);
    }
}

// Half limited x-slopes of a row pair from the slope ring's interleaved entries
// {rho_r, rho_r+1, u_r, u_r+1}, {v_r, v_r+1, p_r, p_r+1} (x-face frame).
__device__ __forceinline__ PairSl pair_sl(const float4 &A, const float4 &B) {
    return PairSl{mk2(A.x, A.y), mk2(A.z, A.w), mk2(B.x, B.y), mk2(B.z, B.w)};
}

// The two y-faces a stage-kernel thread evaluates per step, (r-2 | r-1) in
// lane .x and (r-1 | r) in lane .y, from the primitives of rows
// (r-2, r-1) = lo, (r-1, r) = mid and (r, r+1) = hi of one column and the
// y-slopes of row r-2 (carried from the previous step; `sy_lo` in, the slopes
// of row r out for the next step).
template <int SCHEME, int LIM>
__device__ __forceinline__ void face_pair_y(uint32_t m, const PairPrim &lo, const PairPrim &mid,
                                            const PairPrim &hi, float sy_lo[4], f2 F[5]) {
    // half slopes of rows (r-1, r): limited(row-1, row, row+1), face frame (v normal, u tangential)
    const PairSl sm{p_half_slope<LIM>(lo.rho, mid.rho, hi.rho), p_half_slope<LIM>(lo.v, mid.v, hi.v),
                    p_half_slope<LIM>(lo.u, mid.u, hi.u), p_half_slope<LIM>(lo.p, mid.p, hi.p)};
    // slopes of rows (r-2, r-1)
    const PairSl sl{mk2(sy_lo[0], sm.rho.x), mk2(sy_lo[1], sm.n.x), mk2(sy_lo[2], sm.t.x), mk2(sy_lo[3], sm.p.x)};
    face_pair_core<false, SCHEME>(m, lo, sl, mid, sm, F);
    sy_lo[0] = sm.rho.y;
    sy_lo[1] = sm.n.y;
    sy_lo[2] = sm.t.y;
    sy_lo[3] = sm.p.y;
}

// Face velocities of the rho_e source for two faces (lanes): mass flux over
// the mean of the two cells' clamped densities (src/solver.cu:1772-1794).
__device__ __forceinline__ f2 p_face_velocity(f2 mass, f2 rho_a, f2 rho_b) {
    const f2 mean = p_mul(splat(0.5f), p_add(p_max(rho_a, MIN_DENSITY), p_max(rho_b, MIN_DENSITY)));
    return p_mul(mass, p_rcp(mean));
}

// Rollback of one updated cell (src/solver.cu:1812-1824): a non-finite or
// too small density takes the old one (clamped), a non-finite momentum or
// energy the old value, a non-finite or too small rho_e the old rho_e.  The
// density is >= MIN_DENSITY afterwards, so the reference's second clamp to
// MIN_DENSITY changes nothing and is left out.
__device__ __forceinline__ void rollback_lane(float &rho, float &ru, float &rv, float &E, float &re, float U0, float U1,
                                              float U2, float U3, float U4) {
    if (!isfinite(rho) || rho < MIN_DENSITY) rho = fmaxf(U0, MIN_DENSITY);
    if (!isfinite(ru)) ru = U1;
    if (!isfinite(rv)) rv = U2;
    if (!isfinite(E)) E = U3;
    if (!isfinite(re) || re < MIN_PRESSURE / (GAMMA - 1.0f)) re = U4;
}

// |u| > MAX_VEL (compared in squares): velocity rescaled to MAX_VEL, momenta
// and |u|^2 recomputed (src/solver.cu:1827-1839).
__device__ __forceinline__ void velocity_cap_lane(float rho, float &u, float &v, float &ru, float &rv, float &q) {
    if (q > MAX_VEL * MAX_VEL) {
        const float scale = MAX_VEL / sqrtf(q);
        u *= scale;
        v *= scale;
        ru = rho * u;
        rv = rho * v;
        q = u * u + v * v;
    }
}

// updateKernel body (src/solver.cu:1736-1875) for the two cells of one
// column in rows j (lane .x) and j+1 (lane .y), not walls: U - (dt/dx) dX -
// (dt/dy) dY with dX = F(i+1/2) - F(i-1/2), dY = F(j+1/2) - F(j-1/2) per
// field; the reference zeroes a flux difference across a domain edge
// (i = 0 or nx-1 for x, j = 0 or ny-1 for y), done here by zeroing its
// coefficient.  The rho_e source -p div(v) (interior cells) takes du =
// u(i+1/2) - u(i-1/2) and dv = v(j+1/2) - v(j-1/2) of the face velocities
// and p_c, the cells' primitive pressures.  Then the rollback, the velocity
// cap and the dual-energy resync with e in [rho R T_min, rho R T_max]/(gamma-1).
__device__ __forceinline__ void update_pair(const f2 U[5], const f2 dX[5], const f2 dY[5], f2 du, f2 dv, f2 p_c,
                                            bool edge_x, bool edge_y0, bool edge_y1, const UpdateArgs &a,
                                            f2 out[5]) {
    const f2 ncx = splat(edge_x ? -0.0f : -(a.dt * a.inv_dx));
    const f2 ncy = mk2(edge_y0 ? -0.0f : -(a.dt * a.inv_dy), edge_y1 ? -0.0f : -(a.dt * a.inv_dy));
    f2 n[5];
#pragma unroll
    for (int k = 0; k < 5; k++) n[k] = p_fma(ncy, dY[k], p_fma(ncx, dX[k], U[k]));
    const f2 div_v = p_fma(du, splat(a.inv_dx), p_mul(dv, splat(a.inv_dy)));
    const f2 n4s = p_fma(p_mul(p_c, div_v), splat(-a.dt), n[4]);
    n[4] = p_sel(!edge_x && !edge_y0, !edge_x && !edge_y1, n4s, n[4]);
    f2 inv_rho = p_rcp(n[0]);
    f2 u = p_mul(n[1], inv_rho), v = p_mul(n[2], inv_rho);
    f2 q = p_fma(u, u, p_mul(v, v));
    // the rollback and the velocity cap change a cell only when one of the five
    // new values is not finite (their sum is then not finite either), a floor
    // is undercut or |u| exceeds the cap: one test per cell, the work behind it
    const f2 sum = p_add(p_add(p_add(n[0], n[1]), p_add(n[2], n[3])), n[4]);
    constexpr float re_min = MIN_PRESSURE / (GAMMA - 1.0f);
    const bool fine = isfinite(sum.x) && isfinite(sum.y) && n[0].x >= MIN_DENSITY && n[0].y >= MIN_DENSITY &&
                      n[4].x >= re_min && n[4].y >= re_min && q.x <= MAX_VEL * MAX_VEL && q.y <= MAX_VEL * MAX_VEL;
    if (!fine) {
        rollback_lane(n[0].x, n[1].x, n[2].x, n[3].x, n[4].x, U[0].x, U[1].x, U[2].x, U[3].x, U[4].x);
        rollback_lane(n[0].y, n[1].y, n[2].y, n[3].y, n[4].y, U[0].y, U[1].y, U[2].y, U[3].y, U[4].y);
        inv_rho = p_rcp(n[0]);
        u = p_mul(n[1], inv_rho);
        v = p_mul(n[2], inv_rho);
        q = p_fma(u, u, p_mul(v, v));
        velocity_cap_lane(n[0].x, u.x, v.x, n[1].x, n[2].x, q.x);
        velocity_cap_lane(n[0].y, u.y, v.y, n[1].y, n[2].y, q.y);
    }
    const f2 rho = n[0], E = n[3], re = n[4];
    const f2 ke = p_mul(p_mul(splat(0.5f), rho), q);
    const f2 e_from_E = p_sub(E, ke);
    const f2 thr = p_mul(splat(ETA_THRESHOLD), E);  // dual-energy switch rho_e < 1e-3 E, E > 0
    f2 e = p_sel(E.x > 0.0f && re.x < thr.x, E.y > 0.0f && re.y < thr.y, re, e_from_E);
    e = p_min(p_max(e, p_mul(rho, splat(kEminPerRho))), p_mul(rho, splat(kEmaxPerRho)));
    out[0] = rho;
    out[1] = n[1];
    out[2] = n[2];
    out[3] = p_add(e, ke);
    out[4] = e;
}

// wave_speed of the primitives of two conserved states (prim_from_cons, then
// src/solver.cu:2729-2739), for the fused CFL reduction.
__device__ __forceinline__ f2 pair_wave_speed(const f2 U[5]) {
    const f2 r = p_max(U[0], MIN_DENSITY);
    const f2 inv = p_rcp(r);
    const f2 u = p_mul(U[1], inv), v = p_mul(U[2], inv);
    const f2 q = p_fma(u, u, p_mul(v, v));
    const f2 e_from_E = p_fma(p_mul(splat(-0.5f), r), q, U[3]);
    const f2 e = p_sel(dual_energy_low(U[4].x, U[3].x), dual_energy_low(U[4].y, U[3].y), U[4], e_from_E);
    const f2 p = p_max(p_mul(splat(GAMMA - 1.0f), e), MIN_PRESSURE);
    const f2 c2 = p_mul(p_mul(splat(GAMMA), p), p_rcp(p_add(U[0], splat(1e-10f))));
    return p_add(p_sqrt(q), p_sqrt(c2));
}

// How many of two conserved states, of those counted (c0, c1), have a NaN or
// infinite field (their sum is then not finite; finite states are far below
// the float range).
__device__ __forceinline__ unsigned pair_nonfinite(const f2 U[5], bool c0, bool c1) {
    const f2 s = p_add(p_add(p_add(U[0], U[1]), p_add(U[2], U[3])), U[4]);
    unsigned n = 0u;
    if (!(isfinite(s.x) && isfinite(s.y)))
        n = (c0 && !isfinite(s.x) ? 1u : 0u) + (c1 && !isfinite(s.y) ? 1u : 0u);
    return n;
}

// Divergence terms of the viscous half step for one interior fluid cell
// (src/solver.cu:2437-2510): rhs = {d(tau_xx)/dx + d(tau_xy)/dy,
// d(tau_xy)/dx + d(tau_yy)/dy, -div q + div(tau . v), -div q + Phi}, central
// differences of the per-cell quantities stress_heat_work_sel produced, with
// the x and y parts of each derivative pair in one FP32x2 lane pair:
// (dtau_xx/dx, dtau_xy/dx), (dtau_xy/dy, dtau_yy/dy), (dqx/dx, dqy/dy),
// (dwork_x/dx, dwork_y/dy).  {txx, txy, qx, wx} of the east / west
// neighbours, {tyy, txy, qy, wy} of the north / south ones, Phi of the cell.
struct ViscX {
    float txx, txy, qx, wx;
};
struct ViscY {
    float tyy, txy, qy, wy;
};
__device__ __forceinline__ void viscous_rhs_w(const ViscX &E, const ViscX &W, const ViscY &N, const ViscY &S, float phi,
                                              const ViscArgs &va, float rhs[4]) {
    const f2 i2x = splat(va.inv_2dx), i2y = splat(va.inv_2dy), i2xy = mk2(va.inv_2dx, va.inv_2dy);
    const f2 dtx = p_mul(p_sub(mk2(E.txx, E.txy), mk2(W.txx, W.txy)), i2x);  // (dtau_xx_dx, dtau_xy_dx)
    const f2 dty = p_mul(p_sub(mk2(N.txy, N.tyy), mk2(S.txy, S.tyy)), i2y);  // (dtau_xy_dy, dtau_yy_dy)
    const f2 dq = p_mul(p_sub(mk2(E.qx, N.qy), mk2(W.qx, S.qy)), i2xy);      // (dqx_dx, dqy_dy)
    const f2 dw = p_mul(p_sub(mk2(E.wx, N.wy), mk2(W.wx, S.wy)), i2xy);      // (dwork_dx, dwork_dy)
    const f2 r01 = p_add(dtx, dty);
    rhs[0] = r01.x;
    rhs[1] = r01.y;
    rhs[2] = -dq.x - dq.y + dw.x + dw.y;
    rhs[3] = -dq.x - dq.y + phi;
}

}  // namespace fvm
