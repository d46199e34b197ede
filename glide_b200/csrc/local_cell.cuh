// local_cell.cuh -- the local 5x5 Newton iteration of one Vanka cell.
//
// The unknowns of cell (i, j) are x = (u_l, u_r, v_t, v_b, H) with every
// neighbour and the viscosity frozen (vanka.cu:91-475).  With linear sliding
// (m = 1) the momentum rows are polynomials in x: bilinear in the velocities
// and H (stresses), quadratic in H (driving stress); only the mass row's
// Lax-Friedrichs fluxes need a square root per face.  So everything that does
// not change over the iterations is gathered once per sweep into a few
// coefficients per row, the iteration works on the increments d = x - x_start
// in registers, and no iteration touches memory.
//
// The Newton matrix is a diagonal plus two rank-one terms (the own cell's
// normal stresses) bordered by the thickness column and the mass row, so it
// is solved by elimination into a 2x2 and a scalar: 4 diagonal reciprocals,
// one determinant and one Schur complement instead of five pivots in sequence.  The diagonal entries are at most
// -(ssa_damping + water_drag), which is why the caller takes this path only
// where that sum is positive; the determinant is at least 1.
//
// The sweep is bound by arithmetic and its latency, not by memory: about 340
// operations an iteration here against about 900 in the general form
// (local_system + lu5_solve).  Measured in binary32, 600 x 424, 2 V-cycles:
// 19.2 -> 9.0 ms.  Binary32 only: see Solver::launch_sweep.
#pragma once

#include "stencil.cuh"

namespace glide {

struct LocalCell {
    using R = float;
    R x[5];        // unknowns at the start of the sweep
    R r0[4];       // momentum residuals of the frozen part at the start
    R dd[4];       // minus the neighbours' normal stress and drag on each row's own face
    R P[4], Q[4];  // corner shear coefficients (tl, tr, bl, br): E = P + Q H, zero off the interior vertices
    R sg[4];       // corner shear strains at the start
    R Hn[4];       // neighbour thicknesses (l, r, t, b)
    R dS[4];       // surface differences of the four faces at the start, oriented as the rows use them
    R g, kap;      // own normal-stress coefficient 2 eta dxi^2; d(surface)/dH
    R m0, mh;      // mass row: H dti - f_H (+ calving) at the start; its slope in H
    bool pin[4];   // Dirichlet faces

    template <class S>
    __device__ __forceinline__ void load(const S& s, const PhysR<R>& p, int i, int j, R fu0, R fu1, R fv0, R fv1,
                                         R fH) {
        const int ny = s.ny, nx = s.nx;
        const R d2 = p.dxi * p.dxi;
        x[0] = s.U(i, j); x[1] = s.U(i, j + 1); x[2] = s.V(i, j); x[3] = s.V(i + 1, j); x[4] = s.Hc(i, j);
        pin[0] = j == 0; pin[1] = j == nx - 1; pin[2] = i == 0; pin[3] = i == ny - 1;
        Hn[0] = s.Hc(i, j - 1); Hn[1] = s.Hc(i, j + 1); Hn[2] = s.Hc(i - 1, j); Hn[3] = s.Hc(i + 1, j);
        const R ec = s.ETA(i, j);
        const R phc = s.PHI(i, j), bec = s.BETA(i, j), bdc = s.BED(i, j);
        g = R(2) * ec * d2;
        // surface S = phi bed + (1 - (1 - phi) 0.917) H, as base + H
        const R cf = (R(1) - phc) * R(kFlot);
        kap = R(1) - cf;
        const R Sc = (phc * bdc - cf * x[4]) + x[4];
        const R ph[4] = {s.PHI(i, j - 1), s.PHI(i, j + 1), s.PHI(i - 1, j), s.PHI(i + 1, j)};
        const R be[4] = {s.BETA(i, j - 1), s.BETA(i, j + 1), s.BETA(i - 1, j), s.BETA(i + 1, j)};
        const R bd[4] = {s.BED(i, j - 1), s.BED(i, j + 1), s.BED(i - 1, j), s.BED(i + 1, j)};
        R cal = R(0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const R Sn = (ph[q] * bd[q] - (R(1) - ph[q]) * R(kFlot) * Hn[q]) + Hn[q];
            dS[q] = (q == 0 || q == 3) ? Sc - Sn : Sn - Sc;
            cal += (R(1) - phc) * (R(1) - ph[q]);
        }
        cal *= p.calving_rate * p.dxi;
        // neighbours' normal stresses: k (2 w + frozen), k = 2 eta H dxi^2
        const R el = s.ETA(i, j - 1) * Hn[0], er = s.ETA(i, j + 1) * Hn[1];
        const R et = s.ETA(i - 1, j) * Hn[2], eb = s.ETA(i + 1, j) * Hn[3];
        const R kl = j > 0 ? R(2) * el * d2 : R(0), kr = j < nx - 1 ? R(2) * er * d2 : R(0);
        const R kt = i > 0 ? R(2) * et * d2 : R(0), kb = i < ny - 1 ? R(2) * eb * d2 : R(0);
        const R nl = R(2) * (x[0] - s.U(i, j - 1)) + (s.V(i, j - 1) - s.V(i + 1, j - 1));
        const R nr = R(2) * (s.U(i, j + 2) - x[1]) + (s.V(i, j + 1) - s.V(i + 1, j + 1));
        const R nt = (s.U(i - 1, j + 1) - s.U(i - 1, j)) + R(2) * (s.V(i - 1, j) - x[2]);
        const R nb = (s.U(i + 1, j + 1) - s.U(i + 1, j)) + R(2) * (x[3] - s.V(i + 2, j));
        const R wd = p.water_drag;
        R drag[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) drag[q] = R(0.5) * (be[q] * ph[q] + bec * phc) + wd;
        dd[0] = -(R(2) * kl + drag[0]); dd[1] = -(R(2) * kr + drag[1]);
        dd[2] = -(R(2) * kt + drag[2]); dd[3] = -(R(2) * kb + drag[3]);
        r0[0] = -fu0 - kl * nl - drag[0] * x[0];
        r0[1] = -fu1 + kr * nr - drag[1] * x[1];
        r0[2] = -fv0 + kt * nt - drag[2] * x[2];
        r0[3] = -fv1 - kb * nb - drag[3] * x[3];
        // corner shears (tl, tr, bl, br)
        const R q4 = R(0.25) * d2;
        const bool top = i > 0, bot = i < ny - 1, lft = j > 0, rgt = j < nx - 1;
        const R etl = s.ETA(i - 1, j - 1) * s.Hc(i - 1, j - 1), etr = s.ETA(i - 1, j + 1) * s.Hc(i - 1, j + 1);
        const R ebl = s.ETA(i + 1, j - 1) * s.Hc(i + 1, j - 1), ebr = s.ETA(i + 1, j + 1) * s.Hc(i + 1, j + 1);
        const R Qc = q4 * ec;
        Q[0] = top && lft ? Qc : R(0); Q[1] = top && rgt ? Qc : R(0);
        Q[2] = bot && lft ? Qc : R(0); Q[3] = bot && rgt ? Qc : R(0);
        P[0] = top && lft ? q4 * (etl + et + el) : R(0); P[1] = top && rgt ? q4 * (et + etr + er) : R(0);
        P[2] = bot && lft ? q4 * (el + ebl + eb) : R(0); P[3] = bot && rgt ? q4 * (er + eb + ebr) : R(0);
        sg[0] = (s.U(i - 1, j) - x[0]) + (x[2] - s.V(i, j - 1));
        sg[1] = (s.U(i - 1, j + 1) - x[1]) + (s.V(i, j + 1) - x[2]);
        sg[2] = (x[0] - s.U(i + 1, j)) + (x[3] - s.V(i + 1, j - 1));
        sg[3] = (x[1] - s.U(i + 1, j + 1)) + (s.V(i + 1, j + 1) - x[3]);
        mh = p.dti + cal;
        m0 = x[4] * p.dti - fH + cal * x[4];
    }

    // Lax-Friedrichs share of one face in the mass row: with sw the face
    // velocity signed outwards and hd = dxi / 2 (0 on boundary faces),
    // q = hd (sw (H + Hn) + a (H - Hn)), a = sqrt(w^2 + 10).
    static __device__ __forceinline__ void face(R sw, R h, R Hn, R hd, R& r, R& jw, R& jh) {
        const R q2 = sw * sw + R(10);
        const R ra = rsqrtf(q2);
        const R a = q2 * ra;
        const R sum = h + Hn, dif = h - Hn;
        r += hd * (sw * sum + a * dif);
        jw = hd * (sum + (sw * ra) * dif);
        jh += hd * (sw + a);
    }

    // Newton steps until the squared residual is at most tol or `steps` are
    // done; d accumulates x - x_start.  Returns the steps taken; `masked` is
    // the last step's active-set decision.
    __device__ __forceinline__ int solve(const PhysR<R>& p, R ssa_damping, R mc_damping, R relax, R thk, int steps,
                                         R (&d)[5], R& masked) const {
        const R tol = R(kNewtonTol), hd = R(0.5) * p.dxi;
        R rnorm = R(1);
        int k = 0;
        while (k < steps && rnorm > tol) {
            const R h = x[4] + d[4];
            R r[5], c[4], D[4];
            // mass row
            R a0, a1, a2, a3, a4 = mh;
            r[4] = m0 + mh * d[4];
            face(-(x[0] + d[0]), h, Hn[0], pin[0] ? R(0) : hd, r[4], a0, a4);
            face(x[1] + d[1], h, Hn[1], pin[1] ? R(0) : hd, r[4], a1, a4);
            face(x[2] + d[2], h, Hn[2], pin[2] ? R(0) : hd, r[4], a2, a4);
            face(-(x[3] + d[3]), h, Hn[3], pin[3] ? R(0) : hd, r[4], a3, a4);
            a0 = -a0;
            a3 = -a3;
            a4 += mc_damping;
            // own normal stresses
            const R G = g * h;
            R A, B;
            {
                const R s1 = (x[1] - x[0]) + (d[1] - d[0]), s2 = (x[2] - x[3]) + (d[2] - d[3]);
                A = g * (R(2) * s1 + s2);
                B = g * (s1 + R(2) * s2);
            }
            r[0] = r0[0] + dd[0] * d[0] + A * h;
            r[1] = r0[1] + dd[1] * d[1] - A * h;
            r[2] = r0[2] + dd[2] * d[2] - B * h;
            r[3] = r0[3] + dd[3] * d[3] + B * h;
            c[0] = A; c[1] = -A; c[2] = -B; c[3] = B;
#pragma unroll
            for (int q = 0; q < 4; ++q) D[q] = dd[q] - ssa_damping;
            {
                const R e = P[0] + Q[0] * h, s = sg[0] + (d[2] - d[0]), es = e * s, qs = Q[0] * s;
                r[0] += es; r[2] -= es; c[0] += qs; c[2] -= qs; D[0] -= e; D[2] -= e;
            }
            {
                const R e = P[1] + Q[1] * h, s = sg[1] - (d[1] + d[2]), es = e * s, qs = Q[1] * s;
                r[1] += es; r[2] += es; c[1] += qs; c[2] += qs; D[1] -= e; D[2] -= e;
            }
            {
                const R e = P[2] + Q[2] * h, s = sg[2] + (d[0] + d[3]), es = e * s, qs = Q[2] * s;
                r[0] -= es; r[3] -= es; c[0] -= qs; c[3] -= qs; D[0] -= e; D[3] -= e;
            }
            {
                const R e = P[3] + Q[3] * h, s = sg[3] + (d[1] - d[3]), es = e * s, qs = Q[3] * s;
                r[1] -= es; r[3] += es; c[1] -= qs; c[3] += qs; D[1] -= e; D[3] -= e;
            }
            // driving stress hd (H + Hn) dS
            {
                const R ds = kap * d[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const bool own1 = q == 0 || q == 3;  // the cell is the face's second cell
                    const R t = own1 ? dS[q] + ds : dS[q] - ds;
                    const R w = hd * (h + Hn[q]);
                    r[q] -= w * t;
                    c[q] -= own1 ? hd * t + w * kap : hd * t - w * kap;
                }
            }
            // pinned rows
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (pin[q]) r[q] = x[q] + d[q];
            const bool act = (h - p.dt * r[4]) <= thk;
            masked = act ? R(1) : R(0);
            if (act) r[4] = h - thk;
            rnorm = r[0] * r[0] + r[1] * r[1] + r[2] * r[2] + r[3] * r[3] + r[4] * r[4];
            // D y + (alpha, -alpha, -beta, beta) + c eta = r for the velocities,
            // alpha = G (2 s + t), beta = G (s + 2 t), s = y1 - y0, t = y2 - y3;
            // a . y + a4 eta = r4.  Pinned unknowns leave the other rows.
            const R i0 = pin[0] ? R(0) : R(1) / D[0], i1 = pin[1] ? R(0) : R(1) / D[1];
            const R i2 = pin[2] ? R(0) : R(1) / D[2], i3 = pin[3] ? R(0) : R(1) / D[3];
            const R gp = G * (i0 + i1), gq = G * (i2 + i3);
            const R m11 = R(1) - R(2) * gp, m22 = R(1) - R(2) * gq;
            const R idet = R(1) / (m11 * m22 - gp * gq);
            R y[4], z[4];  // y = y_r - eta z
            {
                y[0] = i0 * r[0]; y[1] = i1 * r[1]; y[2] = i2 * r[2]; y[3] = i3 * r[3];
                const R s = y[1] - y[0], t = y[2] - y[3];
                const R ra = G * (R(2) * s + t), rb = G * (s + R(2) * t);
                const R al = (m22 * ra + gq * rb) * idet, bt = (gp * ra + m11 * rb) * idet;
                y[0] -= i0 * al; y[1] += i1 * al; y[2] += i2 * bt; y[3] -= i3 * bt;
            }
            {
                z[0] = i0 * c[0]; z[1] = i1 * c[1]; z[2] = i2 * c[2]; z[3] = i3 * c[3];
                const R s = z[1] - z[0], t = z[2] - z[3];
                const R ra = G * (R(2) * s + t), rb = G * (s + R(2) * t);
                const R al = (m22 * ra + gq * rb) * idet, bt = (gp * ra + m11 * rb) * idet;
                z[0] -= i0 * al; z[1] += i1 * al; z[2] += i2 * bt; z[3] -= i3 * bt;
            }
            const R num = r[4] - (a0 * y[0] + a1 * y[1] + a2 * y[2] + a3 * y[3]);
            const R den = a4 - (a0 * z[0] + a1 * z[1] + a2 * z[2] + a3 * z[3]);
            const R eta = act ? R(0) : num / den;
#pragma unroll
            for (int q = 0; q < 4; ++q) d[q] -= relax * (pin[q] ? r[q] : y[q] - eta * z[q]);
            d[4] = fmax(d[4] - relax * (act ? r[4] : eta), thk - x[4]);
            ++k;
        }
        return k;
    }
};

}  // namespace glide
