// adjoint_tile.cuh -- the transposed product of one 16 x 16 tile, in the order
// of the reference's rows.
//
// strip.cuh runs the linear operator everywhere but in one place: a mixed
// handle's solves with both tolerances zero, adjoint (here, on the binary32 and
// the binary64 half) and forward (tangent_tile.cuh, on the binary32 half, which
// solves the tangent systems).  Such a solve returns the iterate of its last
// cycle, whose low-order digits are the binary32 rounding of these sums.  The
// march adds the same terms in another order, no less exact, but the iterates
// move: a gradient by 2e-7 to 4e-6 of its norm with the binary32 half marched,
// by up to 3e-8 with the binary64 half alone, a velocity by up to 8e-6 after two
// forward steps (1 to 3 cycles, 64^2 to 560^2).  A caller that fixes the cycles
// asks for that iterate, so it keeps the one it had, at this kernel's price (264
// against 93 us for the binary32 product of 2048^2); a solve to a tolerance
// takes the march.
//
// The reference forms lambda^T dR/dx by scattering every residual row's partials
// with atomics (residuals.cu:667-1163).  Here each output entry gathers the same
// partials from the rows that touch it, in a fixed order, with the reference's
// use of the forward derivative of eta and its target filters: no contribution
// to the u faces on x = 0, nx, the v faces on y = 0, ny, or masked cells.
#pragma once

#include "adjoint_kernels.cuh"
#include "tma.cuh"

namespace glide {

// Forward derivative of the cell viscosity along (du, dv) (viscosity.cu:63-116).
template <class R, class S>
__device__ __forceinline__ R eta_dot_at(const S& s, R Bc, const PhysR<R>& p, int i, int j) {
    const R dxi = p.dxi;
    const int ny = s.ny, nx = s.nx;
    R ul = s.U(i, j), ur = s.U(i, j + 1), vt = s.V(i, j), vb = s.V(i + 1, j);
    R dul = s.LU(i, j), dur = s.LU(i, j + 1), dvt = s.LV(i, j), dvb = s.LV(i + 1, j);
    R ux = (ur - ul) * dxi, vy = (vt - vb) * dxi;
    R dux = (dur - dul) * dxi, dvy = (dvt - dvb) * dxi;
    R m_tl = (i > 0 && j > 0), m_tr = (i > 0 && j < nx - 1);
    R m_bl = (i < ny - 1 && j > 0), m_br = (i < ny - 1 && j < nx - 1);
    R e1 = R(0.5) * ((s.U(i - 1, j) - ul) * dxi + (vt - s.V(i, j - 1)) * dxi) * m_tl;
    R d1 = R(0.5) * ((s.LU(i - 1, j) - dul) * dxi + (dvt - s.LV(i, j - 1)) * dxi) * m_tl;
    R e2 = R(0.5) * ((s.U(i - 1, j + 1) - ur) * dxi + (s.V(i, j + 1) - vt) * dxi) * m_tr;
    R d2 = R(0.5) * ((s.LU(i - 1, j + 1) - dur) * dxi + (s.LV(i, j + 1) - dvt) * dxi) * m_tr;
    R e3 = R(0.5) * ((ul - s.U(i + 1, j)) * dxi + (vb - s.V(i + 1, j - 1)) * dxi) * m_bl;
    R d3 = R(0.5) * ((dul - s.LU(i + 1, j)) * dxi + (dvb - s.LV(i + 1, j - 1)) * dxi) * m_bl;
    R e4 = R(0.5) * ((ur - s.U(i + 1, j + 1)) * dxi + (s.V(i + 1, j + 1) - vb) * dxi) * m_br;
    R d4 = R(0.5) * ((dur - s.LU(i + 1, j + 1)) * dxi + (s.LV(i + 1, j + 1) - dvb) * dxi) * m_br;
    R shear = R(0.25) * (e1 * e1 + e2 * e2 + e3 * e3 + e4 * e4);
    R dshear = R(0.25) * (R(2) * e1 * d1 + R(2) * e2 * d2 + R(2) * e3 * d3 + R(2) * e4 * d4);
    R eII = ux * ux + vy * vy + ux * vy + shear + p.eps_reg;
    R deII = R(2) * ux * dux + R(2) * vy * dvy + (ux * dvy + dux * vy) + dshear;
    return R(0.5) * Bc * p.gexp * glen_pow_m1(eII, p) * deII;
}

// Staged tile for the transpose: forward state, lambda and B in box layout
// (TMA on large levels) with a two-cell halo -- u faces need rows
// [i0-3, i0+19), so the box starts at row i0 - 3 and is 24 rows high in
// binary32, 22 in binary64 (both multiples of 128 bytes) -- and eta, eta-dot
// on cells [i0-2, i0+18).
constexpr int kAdjBoxY = 3;
template <class R>
struct AdjTile {
    static constexpr int BH = sizeof(R) == 4 ? 24 : 22, NB = 9, NC = kTile + 4, P = sizeof(R) == 4 ? 24 : NC;
    BoxT<R, BH> u, v, H, phi, bed, beta, B, lu, lv;  // staging order of the box maps
    R eta[NC][P], etad[NC][P];
};

template <class R>
struct AdjView {
    const AdjTile<R>& a;
    const Arr<R>* lH;
    const Arr<R>* mask;
    int i0, j0, ny, nx;
    static constexpr int A = 2;
    __device__ int r(int i) const { return i - (i0 - kAdjBoxY); }
    __device__ int c(int j) const { return j - (j0 - kBoxX); }
    __device__ R U(int i, int j) const { return a.u[r(i)][c(j)]; }
    __device__ R V(int i, int j) const { return a.v[r(i)][c(j)]; }
    __device__ R LU(int i, int j) const { return a.lu[r(i)][c(j)]; }
    __device__ R LV(int i, int j) const { return a.lv[r(i)][c(j)]; }
    __device__ R Hc(int i, int j) const { return a.H[r(i)][c(j)]; }
    __device__ R PHI(int i, int j) const { return a.phi[r(i)][c(j)]; }
    __device__ R BED(int i, int j) const { return a.bed[r(i)][c(j)]; }
    __device__ R BETA(int i, int j) const { return a.beta[r(i)][c(j)]; }
    __device__ R BC(int i, int j) const { return a.B[r(i)][c(j)]; }
    __device__ R ETA(int i, int j) const { return a.eta[i - (i0 - A)][j - (j0 - A)]; }
    __device__ R ETAD(int i, int j) const { return a.etad[i - (i0 - A)][j - (j0 - A)]; }
    // masked cell multiplier of a source cell inside the domain
    __device__ R LHm(int i, int j) const { return lH->at(i, j) * (R(1) - mask->at(i, j)); }
};

// Contributions of the mass row of cell (i,j) (residuals.cu:717-786).
template <class R>
struct CellSrc { R H0, Hl, Hr, Ht, Hb, Ul, Ur, Vt, Vb; };

template <class R, class S>
__device__ __forceinline__ CellSrc<R> cell_src(const S& s, const PhysR<R>& p, int i, int j, R fH) {
    const int ny = s.ny, nx = s.nx;
    const R dxi = p.dxi;
    CellSrc<R> o;
    R Hc = s.Hc(i, j), phc = s.PHI(i, j), dc;
    R lam = s.LHm(i, j);
    R h = lam * p.dti;
    FluxT<R> f = lflux(s.U(i, j), s.Hc(i, j - 1), Hc, j, nx);
    h += -lam * f.d_H1 * dxi; o.Hl = -lam * f.d_H0 * dxi; o.Ul = -lam * f.d_w * dxi;
    calve(Hc, phc, s.PHI(i, j - 1), p.calving_rate, dc); h += lam * dc * dxi;
    f = lflux(s.U(i, j + 1), Hc, s.Hc(i, j + 1), j + 1, nx);
    h += lam * f.d_H0 * dxi; o.Hr = lam * f.d_H1 * dxi; o.Ur = lam * f.d_w * dxi;
    calve(Hc, phc, s.PHI(i, j + 1), p.calving_rate, dc); h += lam * dc * dxi;
    f = lflux(s.V(i, j), Hc, s.Hc(i - 1, j), i, ny);
    h += lam * f.d_H0 * dxi; o.Ht = lam * f.d_H1 * dxi; o.Vt = lam * f.d_w * dxi;
    calve(Hc, phc, s.PHI(i - 1, j), p.calving_rate, dc); h += lam * dc * dxi;
    f = lflux(s.V(i + 1, j), s.Hc(i + 1, j), Hc, i + 1, ny);
    h += -lam * f.d_H1 * dxi; o.Hb = -lam * f.d_H0 * dxi; o.Vb = -lam * f.d_w * dxi;
    calve(Hc, phc, s.PHI(i + 1, j), p.calving_rate, dc); h += lam * dc * dxi;
    h += -fH;
    o.H0 = h;
    return o;
}

// Contributions of the x-momentum row on u face (i,j) (residuals.cu:791-936).
template <class R>
struct USrc { R U, H0, Hl, Htl, Ht, Hbl, Hb, Vtl, Vtr, Vbl, Vbr; };

template <class R, class S>
__device__ __forceinline__ USrc<R> u_src(const S& s, const PhysR<R>& p, int i, int j, R fu) {
    const int ny = s.ny, nx = s.nx;
    const R dxi = p.dxi;
    USrc<R> o;
    R Hc = s.Hc(i, j), Hl = s.Hc(i, j - 1), ul = s.U(i, j), lul = s.LU(i, j);
    R accU = 0, h0 = 0, hl = 0;
    {
        NormalT<R> a = sxx(ul, s.U(i, j + 1), s.V(i, j), s.V(i + 1, j), s.ETA(i, j) * Hc, dxi, j, nx);
        R t = a.d_ul * lul + a.d_ur * s.LU(i, j + 1) + a.d_vt * s.LV(i, j) + a.d_vb * s.LV(i + 1, j) +
              a.d_eH * (Hc * s.ETAD(i, j));
        accU += t * dxi;
        h0 += lul * a.d_eH * s.ETA(i, j) * dxi;
    }
    {
        NormalT<R> a = sxx(s.U(i, j - 1), ul, s.V(i, j - 1), s.V(i + 1, j - 1), s.ETA(i, j - 1) * Hl, dxi, j - 1, nx);
        R t = a.d_ul * s.LU(i, j - 1) + a.d_ur * lul + a.d_vt * s.LV(i, j - 1) + a.d_vb * s.LV(i + 1, j - 1) +
              a.d_eH * (Hl * s.ETAD(i, j - 1));
        accU += -t * dxi;
        hl += -lul * a.d_eH * s.ETA(i, j - 1) * dxi;
    }
    {
        R Htl = s.Hc(i - 1, j - 1), Ht = s.Hc(i - 1, j);
        R eH = vertex_eH(s.ETA(i - 1, j - 1), s.ETA(i - 1, j), s.ETA(i, j - 1), s.ETA(i, j), Htl, Ht, Hl, Hc);
        R deH = R(0.25) * Htl * s.ETAD(i - 1, j - 1) + R(0.25) * Ht * s.ETAD(i - 1, j) +
                R(0.25) * Hl * s.ETAD(i, j - 1) + R(0.25) * Hc * s.ETAD(i, j);
        ShearT<R> a = sxy(s.U(i - 1, j), ul, s.V(i, j - 1), s.V(i, j), eH, dxi, i, j, ny, nx);
        R t = a.d_ut * s.LU(i - 1, j) + a.d_ub * lul + a.d_vl * s.LV(i, j - 1) + a.d_vr * s.LV(i, j) + a.d_eH * deH;
        accU += t * dxi;
        R g = lul * a.d_eH;
        o.Htl = g * R(0.25) * s.ETA(i - 1, j - 1) * dxi;
        o.Ht = g * R(0.25) * s.ETA(i - 1, j) * dxi;
        hl += g * R(0.25) * s.ETA(i, j - 1) * dxi;
        h0 += g * R(0.25) * s.ETA(i, j) * dxi;
    }
    {
        R Hbl = s.Hc(i + 1, j - 1), Hb = s.Hc(i + 1, j);
        R eH = vertex_eH(s.ETA(i, j - 1), s.ETA(i, j), s.ETA(i + 1, j - 1), s.ETA(i + 1, j), Hl, Hc, Hbl, Hb);
        R deH = R(0.25) * Hl * s.ETAD(i, j - 1) + R(0.25) * Hc * s.ETAD(i, j) +
                R(0.25) * Hbl * s.ETAD(i + 1, j - 1) + R(0.25) * Hb * s.ETAD(i + 1, j);
        ShearT<R> a = sxy(ul, s.U(i + 1, j), s.V(i + 1, j - 1), s.V(i + 1, j), eH, dxi, i + 1, j, ny, nx);
        R t = a.d_ut * lul + a.d_ub * s.LU(i + 1, j) + a.d_vl * s.LV(i + 1, j - 1) + a.d_vr * s.LV(i + 1, j) +
              a.d_eH * deH;
        accU += -t * dxi;
        R g = lul * a.d_eH;
        hl += -g * R(0.25) * s.ETA(i, j - 1) * dxi;
        h0 += -g * R(0.25) * s.ETA(i, j) * dxi;
        o.Hbl = -g * R(0.25) * s.ETA(i + 1, j - 1) * dxi;
        o.Hb = -g * R(0.25) * s.ETA(i + 1, j) * dxi;
    }
    {
        BasalT<R> b = basal(ul, s.V(i, j - 1), s.V(i, j), s.V(i + 1, j - 1), s.V(i + 1, j), s.PHI(i, j - 1),
                            s.PHI(i, j), s.BETA(i, j - 1), s.BETA(i, j), p);
        accU += lul * b.d_w;
        o.Vtl = lul * b.d_a; o.Vtr = lul * b.d_b; o.Vbl = lul * b.d_c; o.Vbr = lul * b.d_d;
    }
    {
        DriveT<R> d = driving(Hl, Hc, s.BED(i, j - 1), s.BED(i, j), s.PHI(i, j - 1), s.PHI(i, j), dxi, j, nx);
        hl += -lul * d.d_H0;
        h0 += -lul * d.d_H1;
    }
    accU += -fu;
    o.U = accU; o.H0 = h0; o.Hl = hl;
    return o;
}

// Contributions of the y-momentum row on v face (i,j) (residuals.cu:938-1103).
template <class R>
struct VSrc { R V, Ht, H0, Htl, Hl, Htr, Hr, Utl, Utr, Ubl, Ubr; };

template <class R, class S>
__device__ __forceinline__ VSrc<R> v_src(const S& s, const PhysR<R>& p, int i, int j, R fv) {
    const int ny = s.ny, nx = s.nx;
    const R dxi = p.dxi;
    VSrc<R> o;
    R Hc = s.Hc(i, j), Ht = s.Hc(i - 1, j), vt = s.V(i, j), lvt = s.LV(i, j);
    R accV = 0, ht = 0, h0 = 0;
    {
        NormalT<R> a = syy(s.U(i - 1, j), s.U(i - 1, j + 1), s.V(i - 1, j), vt, s.ETA(i - 1, j) * Ht, dxi, i - 1, ny);
        R t = a.d_ul * s.LU(i - 1, j) + a.d_ur * s.LU(i - 1, j + 1) + a.d_vt * s.LV(i - 1, j) + a.d_vb * lvt +
              a.d_eH * (Ht * s.ETAD(i - 1, j));
        accV += t * dxi;
        ht += lvt * a.d_eH * s.ETA(i - 1, j) * dxi;
    }
    {
        NormalT<R> a = syy(s.U(i, j), s.U(i, j + 1), vt, s.V(i + 1, j), s.ETA(i, j) * Hc, dxi, i, ny);
        R t = a.d_ul * s.LU(i, j) + a.d_ur * s.LU(i, j + 1) + a.d_vt * lvt + a.d_vb * s.LV(i + 1, j) +
              a.d_eH * (Hc * s.ETAD(i, j));
        accV += -t * dxi;
        h0 += -lvt * a.d_eH * s.ETA(i, j) * dxi;
    }
    {
        R Htl = s.Hc(i - 1, j - 1), Hl = s.Hc(i, j - 1);
        R eH = vertex_eH(s.ETA(i - 1, j - 1), s.ETA(i - 1, j), s.ETA(i, j - 1), s.ETA(i, j), Htl, Ht, Hl, Hc);
        R deH = R(0.25) * Htl * s.ETAD(i - 1, j - 1) + R(0.25) * Ht * s.ETAD(i - 1, j) +
                R(0.25) * Hl * s.ETAD(i, j - 1) + R(0.25) * Hc * s.ETAD(i, j);
        ShearT<R> a = sxy(s.U(i - 1, j), s.U(i, j), s.V(i, j - 1), vt, eH, dxi, i, j, ny, nx);
        R t = a.d_ut * s.LU(i - 1, j) + a.d_ub * s.LU(i, j) + a.d_vl * s.LV(i, j - 1) + a.d_vr * lvt + a.d_eH * deH;
        accV += -t * dxi;
        R g = lvt * a.d_eH;
        o.Htl = -g * R(0.25) * s.ETA(i - 1, j - 1) * dxi;
        ht += -g * R(0.25) * s.ETA(i - 1, j) * dxi;
        o.Hl = -g * R(0.25) * s.ETA(i, j - 1) * dxi;
        h0 += -g * R(0.25) * s.ETA(i, j) * dxi;
    }
    {
        R Htr = s.Hc(i - 1, j + 1), Hr = s.Hc(i, j + 1);
        R eH = vertex_eH(s.ETA(i - 1, j), s.ETA(i - 1, j + 1), s.ETA(i, j), s.ETA(i, j + 1), Ht, Htr, Hc, Hr);
        R deH = R(0.25) * Ht * s.ETAD(i - 1, j) + R(0.25) * Htr * s.ETAD(i - 1, j + 1) +
                R(0.25) * Hc * s.ETAD(i, j) + R(0.25) * Hr * s.ETAD(i, j + 1);
        ShearT<R> a = sxy(s.U(i - 1, j + 1), s.U(i, j + 1), vt, s.V(i, j + 1), eH, dxi, i, j + 1, ny, nx);
        R t = a.d_ut * s.LU(i - 1, j + 1) + a.d_ub * s.LU(i, j + 1) + a.d_vl * lvt + a.d_vr * s.LV(i, j + 1) +
              a.d_eH * deH;
        accV += t * dxi;
        R g = lvt * a.d_eH;
        ht += g * R(0.25) * s.ETA(i - 1, j) * dxi;
        o.Htr = g * R(0.25) * s.ETA(i - 1, j + 1) * dxi;
        h0 += g * R(0.25) * s.ETA(i, j) * dxi;
        o.Hr = g * R(0.25) * s.ETA(i, j + 1) * dxi;
    }
    {
        BasalT<R> b = basal(vt, s.U(i - 1, j), s.U(i - 1, j + 1), s.U(i, j), s.U(i, j + 1), s.PHI(i - 1, j),
                            s.PHI(i, j), s.BETA(i - 1, j), s.BETA(i, j), p);
        accV += lvt * b.d_w;
        o.Utl = lvt * b.d_a; o.Utr = lvt * b.d_b; o.Ubl = lvt * b.d_c; o.Ubr = lvt * b.d_d;
    }
    {
        DriveT<R> d = driving(Hc, Ht, s.BED(i, j), s.BED(i - 1, j), s.PHI(i, j), s.PHI(i - 1, j), dxi, i, ny);
        ht += -lvt * d.d_H1;
        h0 += -lvt * d.d_H0;
    }
    accV += -fv;
    o.V = accV; o.Ht = ht; o.H0 = h0;
    return o;
}

// Box maps in AdjTile staging order: u, v, H, phi, bed, beta, B, lambda_u,
// lambda_v.  Each warp computes a 4 x 8 patch of the 16 x 16 tile.
template <class R, class BLK>
__device__ __forceinline__ void vjp_tile(const VjpArgs<R>& a, const BoxMaps<9>& maps, BLK blk) {
    using TT = AdjTile<R>;
    constexpr int NC = TT::NC;
    __shared__ __align__(128) TT T;
    __shared__ double red[3][kTile * kTile / 32];
    __shared__ unsigned long long bar;
    const int i0 = blk.y() * kTile, j0 = blk.x() * kTile;
    const int ny = a.ny, nx = a.nx;
    {
        BoxT<R, TT::BH>* const dst[TT::NB] = {&T.u, &T.v, &T.H, &T.phi, &T.bed, &T.beta, &T.B, &T.lu, &T.lv};
        const Arr<R> src[TT::NB] = {a.u, a.v, a.H, a.phi, a.bed, a.beta, a.B, a.lu, a.lv};
        if (!stage_boxes<R, TT::NB, TT::BH, kAdjBoxY>(dst, src, maps, i0, j0, &bar, a.err)) return;
    }
    AdjView<R> s{T, &a.lH, &a.mask, i0, j0, ny, nx};
    for (int k = threadIdx.x; k < NC * NC; k += blockDim.x) {
        int r = k / NC, c = k % NC;
        int gi = i0 - 2 + r, gj = j0 - 2 + c;
        const R Bc = s.BC(gi, gj);
        T.eta[r][c] = eta_at<R>(s, Bc, a.p, gi, gj);
        T.etad[r][c] = eta_dot_at<R>(s, Bc, a.p, gi, gj);
    }
    __syncthreads();
    const int wp = threadIdx.x >> 5, ln = threadIdx.x & 31;
    const int I = i0 + 4 * (wp >> 1) + (ln >> 3), J = j0 + 8 * (wp & 1) + (ln & 7);
    double ssu = 0, ssv = 0, ssh = 0;
    const bool f = a.use_forcing != 0;
    const PhysR<R>& p = a.p;
    auto fu = [&](int i, int j) { return f ? a.f_u.at(i, j) : R(0); };
    auto fv = [&](int i, int j) { return f ? a.f_v.at(i, j) : R(0); };
    auto fh = [&](int i, int j) { return f ? a.f_H.at(i, j) : R(0); };
    if (I < ny && J < nx) {
        // Every residual row touching a target of this thread is evaluated
        // once; the target sums take fixed slots of those rows.
        const bool has_l = J > 0, has_r = J + 1 < nx, has_t = I > 0, has_b = I + 1 < ny;
        const CellSrc<R> c0 = cell_src(s, p, I, J, fh(I, J));
        const CellSrc<R> cl = has_l ? cell_src(s, p, I, J - 1, fh(I, J - 1)) : CellSrc<R>{};
        const CellSrc<R> ct = has_t ? cell_src(s, p, I - 1, J, fh(I - 1, J)) : CellSrc<R>{};
        const CellSrc<R> cr = has_r ? cell_src(s, p, I, J + 1, fh(I, J + 1)) : CellSrc<R>{};
        const CellSrc<R> cb = has_b ? cell_src(s, p, I + 1, J, fh(I + 1, J)) : CellSrc<R>{};
        const USrc<R> u0 = u_src(s, p, I, J, fu(I, J));
        const USrc<R> ur = u_src(s, p, I, J + 1, fu(I, J + 1));
        const USrc<R> utr = has_t ? u_src(s, p, I - 1, J + 1, fu(I - 1, J + 1)) : USrc<R>{};
        const USrc<R> ut = has_t ? u_src(s, p, I - 1, J, fu(I - 1, J)) : USrc<R>{};
        const USrc<R> ubr = has_b ? u_src(s, p, I + 1, J + 1, fu(I + 1, J + 1)) : USrc<R>{};
        const USrc<R> ub = has_b ? u_src(s, p, I + 1, J, fu(I + 1, J)) : USrc<R>{};
        const VSrc<R> v0 = v_src(s, p, I, J, fv(I, J));
        const VSrc<R> vb = v_src(s, p, I + 1, J, fv(I + 1, J));
        const VSrc<R> vbl = has_l ? v_src(s, p, I + 1, J - 1, fv(I + 1, J - 1)) : VSrc<R>{};
        const VSrc<R> vl = has_l ? v_src(s, p, I, J - 1, fv(I, J - 1)) : VSrc<R>{};
        const VSrc<R> vbr = has_r ? v_src(s, p, I + 1, J + 1, fv(I + 1, J + 1)) : VSrc<R>{};
        const VSrc<R> vr = has_r ? v_src(s, p, I, J + 1, fv(I, J + 1)) : VSrc<R>{};

        // u face (I, J): interior faces only
        R ou = 0;
        if (has_l) ou = c0.Ul + cl.Ur + u0.U + vb.Utl + vbl.Utr + v0.Ubl + vl.Ubr;
        if (a.s_u.p) ou = ou - a.s_u.at(I, J);
        a.o_u.at(I, J) = ou;
        ssu += double(ou) * double(ou);
        if (J == nx - 1) {
            R e = a.s_u.p ? R(0) - a.s_u.at(I, nx) : R(0);
            a.o_u.at(I, nx) = e;
            ssu += double(e) * double(e);
        }
        // v face (I, J): interior faces only
        R ov = 0;
        if (has_t) ov = c0.Vt + ct.Vb + v0.V + ur.Vtl + u0.Vtr + utr.Vbl + ut.Vbr;
        if (a.s_v.p) ov = ov - a.s_v.at(I, J);
        a.o_v.at(I, J) = ov;
        ssv += double(ov) * double(ov);
        if (I == ny - 1) {
            R e = a.s_v.p ? R(0) - a.s_v.at(ny, J) : R(0);
            a.o_v.at(ny, J) = e;
            ssv += double(e) * double(e);
        }
        // cell (I, J); masked cells receive nothing
        R oh = 0;
        if (!(a.mask.at(I, J) > R(0))) {
            oh = c0.H0;
            if (has_r) oh += cr.Hl;
            if (has_l) oh += cl.Hr;
            if (has_b) oh += cb.Ht;
            if (has_t) oh += ct.Hb;
            oh += u0.H0;
            oh += ur.Hl;
            if (has_b) oh += ubr.Htl + ub.Ht;
            if (has_t) oh += utr.Hbl + ut.Hb;
            oh += vb.Ht;
            oh += v0.H0;
            if (has_r) oh += vbr.Htl + vr.Hl;
            if (has_l) oh += vbl.Htr + vl.Hr;
        }
        if (a.s_H.p) oh = oh - a.s_H.at(I, J);
        a.o_H.at(I, J) = oh;
        ssh += double(oh) * double(oh);
    }
    if (a.partial) {
        for (int o = 16; o > 0; o >>= 1) {
            ssu += __shfl_down_sync(0xffffffffu, ssu, o);
            ssv += __shfl_down_sync(0xffffffffu, ssv, o);
            ssh += __shfl_down_sync(0xffffffffu, ssh, o);
        }
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        if (l == 0) { red[0][w] = ssu; red[1][w] = ssv; red[2][w] = ssh; }
        __syncthreads();
        if (threadIdx.x < 3) {
            double acc = 0;
            for (int q = 0; q < kTile * kTile / 32; ++q) acc += red[threadIdx.x][q];
            a.partial[size_t(blk.y() * blk.gx() + blk.x()) * 3 + threadIdx.x] = acc;
        }
    }
}

template <class R>
__global__ void __launch_bounds__(kTile * kTile) k_vjp(VjpArgs<R> a,
                                                         const __grid_constant__ BoxMaps<9> maps) {
    vjp_tile<R>(a, maps, SoloBlock{});
}

}  // namespace glide
