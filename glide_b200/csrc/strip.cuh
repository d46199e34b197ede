// strip.cuh -- the linearised operator of one level, marched in strips.
//
// A warp owns a strip of columns, one lane per column, and walks down the rows
// of its chunk.  Every array value is loaded once per strip (coalesced, one row
// ahead of its use) and lives in registers; horizontal neighbours come from
// shuffles, vertical ones are carried from row to row.  Each derived quantity
// -- a vertex shear, a cell viscosity, a normal stress, a face flux -- is
// evaluated once, by the lane that owns it, and handed to the two or four rows
// it enters.  No shared memory, no block barrier, no staging.
//
// The 16 x 16 tile form this replaces evaluated every face flux and most
// stresses twice (the transposed product 17 whole rows per cell), read each
// value from shared memory up to nine times and issued about 1050 instructions
// per owned cell for the Jacobian product; the march issues about 540.  What
// bounds it now is the dependent chain of a row step (loads one row ahead, 16
// shuffles, one cube root) at 16 to 20 warps per SM.  Measured at 2048^2: J e in
// binary32 139 -> 93 us, J^T lambda 264 -> 93 us, in binary64 243 -> 135 and 500 ->
// 134 us; a smoother sweep (product and block solve) in binary32 225 -> 182 us, of
// the adjoint 393 -> 168 us, where its bytes alone take 78 and 103 at the measured
// 6.46 TB/s.
//
// Both directions of the coupled operator run here:
//   TR = false: J e, the exact derivative of the residual rows along e with
//     the grounded fraction held fixed (residuals.cu:341-660);
//   TR = true: the reference's lambda^T dR/dx (residuals.cu:667-1163).  Its
//     viscous velocity block is the forward derivative along lambda, so it
//     shares the march; its thickness row's viscous part collapses to
//     -2 eta (d strain-rate invariant along lambda); the other blocks are
//     transposed face by face.
// With SMOOTH the block solve of the linear smoother (FactorStore) follows in
// the same pass: the residual of a cell's five rows never leaves registers, and
// the updated unknowns go to a second buffer, since neighbouring strips still
// read the old ones.
//
// Lanes at the strip's edges only feed their neighbours: the stresses reach
// two columns to the left and right, a face update one cell further to the left.
#pragma once

#include <type_traits>

#include "adjoint_kernels.cuh"

namespace glide {

constexpr int kStripWarps = 4;  // warps of a block: consecutive chunks of one strip

template <bool SMOOTH>
struct StripShape {
    static constexpr int kLeft = SMOOTH ? 3 : 2;    // feeding lanes on the left
    static constexpr int kCols = SMOOTH ? 27 : 28;  // columns a strip owns
};

// Launch arguments of the marched product (and smoother).
template <class R>
struct StripArgs {
    VjpArgs<R> a;         // o_*: residual out (null with SMOOTH: not stored)
    int mode;             // forward direction: bit 0 the reference's row conventions, bit 1 mask ignored
    int rows;             // rows of a chunk
    const R* fac;         // SMOOTH: block factors (FactorStore<R, TR>)
    size_t plane;
    Arr<R> xu, xv, xH;    // SMOOTH: updated unknowns
    R omega;
};

template <class R>
__device__ __noinline__ R pow_general(R x, R e) { return pow(x, e); }

// q^e for |e| <= 1 and a positive normal q = 2^k f, f about 1: 2^(k e) f^e as
// 2^n exp(r), with n the nearest integer to k e and r = (k e - n) ln 2 + e ln f
// carried as a sum of two numbers, so that only the logarithm's and the
// exponential's own last places are lost.  Measured against a 64-bit mantissa on
// 4 million q in 1e-12 .. 1e14 for each of m = 0, 0.2, 1/3, 0.5, 0.75, 2 and 2.9:
// rms error 5.0e-17 to 6.8e-17, largest 1.5e-16 to 2.4e-16; pow() 6.5e-17 to
// 6.8e-17 and 2.2e-16.
__device__ __forceinline__ double pow_small(double q, double e) {
    const int hi = __double2hiint(q);
    const int k = (hi - 0x3fe6a09e) >> 20;  // f in [sqrt(1/2), sqrt(2))
    const double f = __hiloint2double(hi - (k << 20), __double2loint(q));
    constexpr double ln2 = 0.693147180559945286, ln2_low = 2.319046813846299558e-17;
    const double ke = double(k) * e, ke_low = fma(double(k), e, -ke);
    const double n = rint(ke), t = ke - n, lf = log(f);
    const double a = t * ln2, b = e * lf;
    const double low = fma(t, ln2, -a) + fma(e, lf, -b) + fma(t, ln2_low, ke_low * ln2);
    const double r = a + b, bb = r - a;
    const double r_low = (a - (r - bb)) + (b - bb) + low;
    const double x = exp(r);
    return fma(x, r_low, x) * __hiloint2double((int(n) + 1023) << 20, 0);
}

// Two powers of one exponent, in line so that their chains overlap: pow() is some
// 150 dependent operations behind a call of its own.
struct PowPair { double a, b; };
__device__ __forceinline__ PowPair pow_pair(double x, double y, double e) {
    constexpr double lo = 1e-280, up = 1e280;  // 2^n stays a normal number
    if (fabs(e) <= 1.0 && x > lo && x < up && y > lo && y < up) return {pow_small(x, e), pow_small(y, e)};
    return {pow_general(x, e), pow_general(y, e)};
}

// d q^e / dq from the power itself.  At q = 0 the quotient says nothing (0 / 0
// where the derivative is finite).
__device__ __forceinline__ double pow_slope(double q, double pw, double e) {
    return q > 0.0 ? e * pw / q : e * pow_general(q, e - 1.0);
}

// The neighbouring lanes' values.  All 32 lanes must call: never inside a
// conditional expression or a branch that is not uniform over the warp.
template <class R>
__device__ __forceinline__ R lane_left(R x) { return __shfl_up_sync(0xffffffffu, x, 1); }
template <class R>
__device__ __forceinline__ R lane_right(R x) { return __shfl_down_sync(0xffffffffu, x, 1); }

// Lax-Friedrichs face coefficients between cells 0 and 1 (flux.cu:40-64);
// zero on the domain edge.
template <class R>
__device__ __forceinline__ void face_coeffs(R w, R H0, R H1, bool on, R& d_w, R& d_0, R& d_1) {
    const R q2 = w * w + R(10);
    const R ra = rsqrt_r(q2);
    const R hw = on ? R(0.5) * w : R(0), ha = on ? R(0.5) * (q2 * ra) : R(0);
    d_0 = hw + ha;
    d_1 = hw - ha;
    d_w = on ? R(0.5) * ((H0 + H1) - (w * ra) * (H1 - H0)) : R(0);
}

// The values of one row a lane loads: face rows t + 1, cell row t.
template <class R>
struct StripRow {
    R u, v, eu, ev, H, phi, bed, beta, B, eH, mask;
};

// What is compiled for the sliding law.  Binary64 has a kernel for linear sliding
// and one for the rest: the power's code in one kernel for both cost the product 90
// bytes of spills at its 168 registers (J e with m = 1: 219 us at 2048^2, 135 on
// its own; 53 and 35 at 1000 x 760).  In binary32 the power is cheap and one
// kernel decides as it runs.
enum SlideCode { kSlideLinear, kSlidePower, kSlideEither };

template <class R, bool TR, bool SMOOTH, int SLIDE, class BLK>
__device__ __forceinline__ void linear_strip(const StripArgs<R>& q, BLK blk) {
    constexpr int HL = StripShape<SMOOTH>::kLeft, W = StripShape<SMOOTH>::kCols;
    const VjpArgs<R>& a = q.a;
    const PhysR<R>& p = a.p;
    const int ny = a.ny, nx = a.nx;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int j = int(blk.x()) * W - HL + lane;
    const int ra = (int(blk.y()) * kStripWarps + wp) * q.rows, rb = min(ra + q.rows, ny);
    const bool ref_rows = (q.mode & 1) != 0, use_mask = TR || SMOOTH || (q.mode & 2) == 0;
    const bool linear = SLIDE == kSlideEither ? p.m == R(1) : SLIDE == kSlideLinear;
    const bool calving = p.calving_rate != R(0), f = a.use_forcing != 0;
    const R dxi = p.dxi, hdx = R(0.5) * p.dxi;
    const unsigned ju = unsigned(clampi(j, 0, nx)), jc = unsigned(clampi(j, 0, nx - 1));
    const unsigned pu = unsigned(a.u.pitch), pc = unsigned(a.H.pitch);  // v and cell arrays share a pitch
    const bool in_c = j >= 0 && j < nx;   // a cell column
    const bool face_u = j > 0 && j < nx;  // an interior u face
    const bool own = lane >= HL && lane < HL + W && j <= nx, own_c = own && j < nx;
    double ssu = 0, ssv = 0, ssh = 0;

    auto load = [&](int t) {  // face rows t + 1, cell row t, clamped into the arrays
        StripRow<R> r;
        const unsigned ou = unsigned(clampi(t + 1, 0, ny - 1)) * pu + ju;
        const unsigned ov = unsigned(clampi(t + 1, 0, ny)) * pc + jc;
        const unsigned oc = unsigned(clampi(t, 0, ny - 1)) * pc + jc;
        r.u = __ldg(a.u.p + ou); r.eu = __ldg(a.lu.p + ou);
        r.v = __ldg(a.v.p + ov); r.ev = __ldg(a.lv.p + ov);
        r.H = __ldg(a.H.p + oc); r.eH = __ldg(a.lH.p + oc);
        r.phi = __ldg(a.phi.p + oc); r.bed = __ldg(a.bed.p + oc);
        r.beta = __ldg(a.beta.p + oc); r.B = __ldg(a.B.p + oc);
        r.mask = use_mask ? __ldg(a.mask.p + oc) : R(0);
        return r;
    };

    if (ra < ny) {  // uniform over the warp
        const int t0 = ra - (SMOOTH ? 2 : 1);
        const int first = SMOOTH ? ra - 1 : ra;  // first row whose residual is formed
        // values of row t (suffix 0) and t - 1 (m: faces, p: cells)
        R um = __ldg(a.u.p + unsigned(clampi(t0 - 1, 0, ny - 1)) * pu + ju);
        R eum = __ldg(a.lu.p + unsigned(clampi(t0 - 1, 0, ny - 1)) * pu + ju);
        R u0 = __ldg(a.u.p + unsigned(clampi(t0, 0, ny - 1)) * pu + ju);
        R eu0 = __ldg(a.lu.p + unsigned(clampi(t0, 0, ny - 1)) * pu + ju);
        R v0 = __ldg(a.v.p + unsigned(clampi(t0, 0, ny)) * pc + jc);
        R ev0 = __ldg(a.lv.p + unsigned(clampi(t0, 0, ny)) * pc + jc);
        R v0l = lane_left(v0), ev0l = lane_left(ev0), umr = lane_right(um), eumr = lane_right(eum);
        const R vm0 = (t0 > 0 && t0 < ny && face_u) ? hdx : R(0);
        R vs0 = vm0 * ((um - u0) + (v0 - v0l)), dvs0 = vm0 * ((eum - eu0) + (ev0 - ev0l));
        R vs0r = lane_right(vs0), dvs0r = lane_right(dvs0);
        R evm = 0, hsp = 0, dhsp = 0, nyyp = 0, accU = 0, accH = 0, rvp = 0, gup = 0, ddb = 0;
        R Hp = 0, Sp = 0, kapp = 0, xp = 0, pp = 0, flp = 0, maskp = 0, eHp = 0;
        StripRow<R> nxt = load(t0);
        for (int t = t0; t <= rb; ++t) {
            const StripRow<R> c = nxt;
            if (t < rb) nxt = load(t + 1);
            const int r = t - 1;  // the row this step finishes
            // what finishing it needs, loaded before the arithmetic
            R fu = 0, fv = 0, fH = 0, M[25];
            if (f && t >= first) fv = __ldg(a.f_v.p + unsigned(max(t, 0)) * pc + jc);
            if (r >= first) {
                const unsigned rr = unsigned(max(r, 0));
                if (f) {
                    fu = __ldg(a.f_u.p + rr * pu + ju);
                    fH = __ldg(a.f_H.p + rr * pc + jc);
                }
                if constexpr (SMOOTH) FactorStore<R, TR>::get(q.fac, q.plane, size_t(rr) * pc + jc, M);
            }
            // ---- strain rates: vertex row t + 1, cell row t
            const R v1l = lane_left(c.v), ev1l = lane_left(c.ev);
            const R vm = (t + 1 > 0 && t + 1 < ny && face_u) ? hdx : R(0);
            const R vs1 = vm * ((u0 - c.u) + (c.v - v1l)), dvs1 = vm * ((eu0 - c.eu) + (c.ev - ev1l));
            const R vs1r = lane_right(vs1), dvs1r = lane_right(dvs1);
            const R u0r = lane_right(u0), eu0r = lane_right(eu0);
            const R ux = (u0r - u0) * dxi, vy = (v0 - c.v) * dxi;
            const R dux = (eu0r - eu0) * dxi, dvy = (ev0 - c.ev) * dxi;
            const R eII = ux * ux + vy * vy + ux * vy +
                          R(0.25) * (vs0 * vs0 + vs0r * vs0r + vs1 * vs1 + vs1r * vs1r) + p.eps_reg;
            const R deII = R(2) * ux * dux + R(2) * vy * dvy + (ux * dvy + dux * vy) +
                           R(0.5) * (vs0 * dvs0 + vs0r * dvs0r + vs1 * dvs1 + vs1r * dvs1r);
            // viscosity and its derivative along e: eta = B/2 eII^g, eta' = eta g eII'/eII
            R eta, etad;
            if (p.glen3) {
                const R rc = rcbrt_r(eII);
                eta = R(0.5) * c.B * rc;
                etad = eta * p.gexp * deII * (rc * rc * rc);
            } else {
                eta = R(0.5) * c.B * pow_general(eII, p.gexp);
                etad = eta * p.gexp * deII / eII;
            }
            const R etaH = eta * c.H, detaH = TR ? etad * c.H : etad * c.H + eta * c.eH;
            // ---- normal stresses of cell row t, shear on vertex row t
            const R ex = R(2) * ux + vy, ey = ux + R(2) * vy;
            const R nxx = in_c ? R(2) * (etaH * (R(2) * dux + dvy) + ex * detaH) : R(0);
            const R nyy = (t >= 0 && t < ny) ? R(2) * (etaH * (dux + R(2) * dvy) + ey * detaH) : R(0);
            const R hs = etaH + lane_left(etaH), dhs = detaH + lane_left(detaH);
            const R sxy = R(0.5) * ((hsp + hs) * dvs0 + vs0 * (dhsp + dhs));
            R ru = dxi * ((nxx - lane_left(nxx)) + sxy), rv = dxi * ((nyyp - nyy) + (lane_right(sxy) - sxy));
            // ---- the faces of row t
            const bool face_v = t > 0 && t < ny;
            const R pb = c.beta * c.phi, fl = R(1) - c.phi, cf = fl * R(kFlot);
            const R S = (c.phi * c.bed - cf * c.H) + c.H, kap = R(1) - cf;
            const R Hl = lane_left(c.H), Sl = lane_left(S);
            const R dSu = face_u ? S - Sl : R(0), dSv = face_v ? Sp - S : R(0);
            const R Hmu = face_u ? R(0.5) * (Hl + c.H) : R(0), Hmv = face_v ? R(0.5) * (c.H + Hp) : R(0);
            const R beu = R(0.5) * (lane_left(pb) + pb), bev = R(0.5) * (pp + pb);
            R uw, u_0, u_1, vw, v_0, v_1;
            face_coeffs(u0, Hl, c.H, face_u, uw, u_0, u_1);
            face_coeffs(v0, c.H, Hp, face_v, vw, v_0, v_1);
            R cross = 0;  // TR, nonlinear sliding: what face row t adds to u faces t - 1 and t, per unit of u
            if (linear) {
                ru -= (beu + p.water_drag) * eu0;
                rv -= (bev + p.water_drag) * ev0;
            } else {
                const R e = (p.m - R(1)) / R(2);
                const R qu = u0 * u0 + R(0.25) * (v0l * v0l + v0 * v0 + v1l * v1l + c.v * c.v) + p.u_reg;
                const R qv = v0 * v0 + R(0.25) * (um * um + umr * umr + u0 * u0 + u0r * u0r) + p.u_reg;
                R hu, hv;
                if constexpr (sizeof(R) == 8) {
                    // one power a face (its derivative divides), and only in steps
                    // whose faces enter a finished row: v face t rows t - 1 and t, u
                    // face t row t and, with TR, the v faces t and t + 1.  Four calls
                    // of pow() in every step, two powers and two derivatives, had made
                    // J e with m = 1/3 slower than the 16 x 16 tiles: 51 us at 512^2,
                    // now 31 (tiles 31); 474, now 322, at 2048^2 (353); 16.4, now 10.6,
                    // at 64^2 (12.3).  J^T lambda 49 -> 32 at 512^2 (60), 449 -> 298 at
                    // 2048^2 (825).
                    hu = hv = 0;
                    if (TR || (t >= first && (SMOOTH || t < rb))) {
                        const PowPair pw = pow_pair(qu, qv, e);
                        const R dpu = pow_slope(qu, pw.a, e), dpv = pow_slope(qv, pw.b, e);
                        ru -= (beu * (R(2) * dpu * u0 * u0 + pw.a) + p.water_drag) * eu0;
                        rv -= (bev * (R(2) * dpv * v0 * v0 + pw.b) + p.water_drag) * ev0;
                        hu = -beu * (R(0.5) * dpu * u0);
                        hv = -bev * (R(0.5) * dpv * v0);
                    }
                } else {
                    const R dpu = e * pow_general(qu, e - R(1)), dpv = e * pow_general(qv, e - R(1));
                    ru -= (beu * (R(2) * dpu * u0 * u0 + pow_general(qu, e)) + p.water_drag) * eu0;
                    rv -= (bev * (R(2) * dpv * v0 * v0 + pow_general(qv, e)) + p.water_drag) * ev0;
                    hu = -beu * (R(0.5) * dpu * u0), hv = -bev * (R(0.5) * dpv * v0);
                }
                if (TR) {
                    const R gu = hu * eu0, gv = hv * ev0, gs = gu + lane_right(gu);
                    rv += v0 * (gup + gs);
                    gup = gs;
                    cross = gv + lane_left(gv);
                    ru += u0 * cross;
                } else {
                    ru += hu * (v0l * ev0l + v0 * ev0 + v1l * ev1l + c.v * c.ev);
                    rv += hv * (um * eum + umr * eumr + u0 * eu0 + u0r * eu0r);
                }
            }
            // mass row of cell t, and what face row t adds to that of cell t - 1
            const R x = TR ? c.eH * (R(1) - c.mask) : c.eH;
            R rH, low;
            if (TR) {
                const R glu = lane_left(x) - x, glv = x - xp, Hmur = lane_right(Hmu), dSur = lane_right(dSu);
                const R av = ev0 * Hmv, bv = ev0 * dSv;
                ru += dxi * (glu * uw);
                rv += dxi * (glv * vw);
                rH = x * p.dti - R(2) * eta * deII + dxi * (glu * u_1 + lane_right(glu * u_0) + glv * v_0) -
                     kap * dxi * ((eu0 * Hmu - eu0r * Hmur) - av) - hdx * (eu0 * dSu + eu0r * dSur + bv);
                low = dxi * (glv * v_1) - hdx * bv - kapp * dxi * av;
            } else {
                const R xl = lane_left(x), kx = kap * x;
                const R Fu = uw * eu0 + u_0 * xl + u_1 * x, Fv = vw * ev0 + v_0 * x + v_1 * xp;
                ru -= hdx * dSu * (xl + x) + Hmu * dxi * (kx - lane_left(kx));
                rv -= hdx * dSv * (x + xp) + Hmv * dxi * (kapp * xp - kx);
                rH = x * p.dti + dxi * ((lane_right(Fu) - Fu) + Fv);
                low = -dxi * Fv;
            }
            if (calving) {  // towards the left, right and upper neighbour; of cell t - 1 towards this one
                const R k = p.calving_rate * dxi;
                rH += k * fl * (lane_left(fl) + lane_right(fl) + flp) * x;
                low += k * flp * fl * xp;
            }
            // ---- the finished row: u and H of row t - 1, v of face row t
            const R fin_u = accU - dxi * sxy + um * cross, fin_H = accH + low;
            R b0, b3, b4;
            if (TR) {
                b0 = face_u ? fin_u - fu : R(0);
                b3 = face_v ? rv - fv : R(0);
                b4 = maskp > R(0) ? R(0) : fin_H - fH;
            } else {
                b0 = (face_u ? fin_u : (ref_rows ? R(0) : eum)) - fu;
                b3 = (face_v ? rv : (ref_rows ? R(0) : ev0)) - fv;
                b4 = (ref_rows ? (R(1) - maskp) * fin_H : (maskp > R(0.5) ? eHp : fin_H)) - fH;
            }
            if constexpr (SMOOTH) {
                const R b1 = lane_right(b0);
                if (r >= first) {
                    const R b[5] = {b0, b1, rvp, b3, (TR && maskp > R(0.5)) ? R(0) : b4};
                    R d[5];
                    block_solve<R>(M, b, d);
                    const bool cell = in_c && r >= 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) d[k] = cell ? R(0.5) * d[k] : R(0);
                    const R dl = lane_left(d[1]);
                    if (r >= ra) {
                        const unsigned iu = unsigned(r) * pu + unsigned(j), ic = unsigned(r) * pc + unsigned(j);
                        if (own) q.xu.p[iu] = eum - q.omega * (dl + d[0]);
                        if (own_c) {
                            q.xv.p[ic] = evm - q.omega * (ddb + d[2]);
                            q.xH.p[ic] = eHp - q.omega * d[4];
                            if (r == ny - 1) q.xv.p[ic + pc] = ev0 - q.omega * d[3];
                        }
                        if (a.o_u.p) {
                            if (own) a.o_u.p[iu] = b0;
                            if (own_c) {
                                a.o_v.p[ic] = rvp;
                                a.o_H.p[ic] = b4;
                                if (r == ny - 1) a.o_v.p[ic + pc] = b3;
                            }
                        }
                    }
                    ddb = d[3];
                }
            } else if (r >= ra) {
                const unsigned iu = unsigned(r) * pu + unsigned(j), ic = unsigned(r) * pc + unsigned(j);
                const bool sub = a.s_u.p != nullptr;
                if (own) {
                    const R o = sub ? b0 - a.s_u.p[iu] : b0;
                    a.o_u.p[iu] = o;
                    ssu += double(o) * double(o);
                }
                if (own_c) {
                    const R ov = sub ? rvp - a.s_v.p[ic] : rvp, oh = sub ? b4 - a.s_H.p[ic] : b4;
                    a.o_v.p[ic] = ov;
                    a.o_H.p[ic] = oh;
                    ssv += double(ov) * double(ov);
                    ssh += double(oh) * double(oh);
                    if (r == ny - 1) {
                        const R o = sub ? b3 - a.s_v.p[ic + pc] : b3;
                        a.o_v.p[ic + pc] = o;
                        ssv += double(o) * double(o);
                    }
                }
            }
            // ---- next row
            accU = ru; accH = rH; rvp = b3;
            um = u0; eum = eu0; umr = u0r; eumr = eu0r; evm = ev0;
            u0 = c.u; eu0 = c.eu; v0 = c.v; ev0 = c.ev; v0l = v1l; ev0l = ev1l;
            vs0 = vs1; dvs0 = dvs1; vs0r = vs1r; dvs0r = dvs1r;
            hsp = hs; dhsp = dhs; nyyp = nyy;
            Hp = c.H; Sp = S; kapp = kap; xp = x; pp = pb; flp = fl; maskp = c.mask; eHp = c.eH;
        }
    }
    if (!SMOOTH && a.partial) {  // fixed-order sums of squares: lanes, then the block's warps
        __shared__ double red[3][kStripWarps];
        for (int o = 16; o > 0; o >>= 1) {
            ssu += __shfl_down_sync(0xffffffffu, ssu, o);
            ssv += __shfl_down_sync(0xffffffffu, ssv, o);
            ssh += __shfl_down_sync(0xffffffffu, ssh, o);
        }
        if (lane == 0) { red[0][wp] = ssu; red[1][wp] = ssv; red[2][wp] = ssh; }
        __syncthreads();
        if (threadIdx.x < 3) {
            double acc = 0;
            for (int k = 0; k < kStripWarps; ++k) acc += red[threadIdx.x][k];
            a.partial[size_t(blk.y() * blk.gx() + blk.x()) * 3 + threadIdx.x] = acc;
        }
    }
}

// f(the SLIDE to launch, as an integral constant)
template <class R, class F>
void with_slide_code(bool linear, F&& f) {
    if constexpr (sizeof(R) == 4) f(std::integral_constant<int, kSlideEither>{});
    else if (linear) f(std::integral_constant<int, kSlideLinear>{});
    else f(std::integral_constant<int, kSlidePower>{});
}

template <class R, bool SMOOTH>
struct StripBlocks {
    // resident blocks per SM the registers are fitted to
    static constexpr int n = sizeof(R) == 8 ? (SMOOTH ? 2 : 3) : (SMOOTH ? 4 : 5);
};

template <class R, bool TR, bool SMOOTH, int SLIDE>
__global__ void __launch_bounds__(32 * kStripWarps, StripBlocks<R, SMOOTH>::n) k_linear_strip(StripArgs<R> q) {
    linear_strip<R, TR, SMOOTH, SLIDE>(q, SoloBlock{});
}

}  // namespace glide
