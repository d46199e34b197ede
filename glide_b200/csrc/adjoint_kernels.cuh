// adjoint_kernels.cuh -- block factors and sweep of the linear smoothers, the
// arguments of the linear operator's march (strip.cuh) and the parameter
// gradients.
#pragma once

#include <cuda_bf16.h>

#include "forward_kernels.cuh"
#include "tma.cuh"

namespace glide {

// Fields of one application of the linear operator, J e or J^T lambda: lu, lv,
// lH carry e or lambda.
template <class R>
struct VjpArgs {
    Arr<R> u, v, H, phi, mask, bed, B, beta;
    Arr<R> lu, lv, lH;
    Arr<R> f_u, f_v, f_H;   // forcing (use_forcing)
    Arr<R> o_u, o_v, o_H;   // outputs
    Arr<R> s_u, s_v, s_H;   // optional subtrahends
    double* partial;
    int* err;  // set when a bounded wait gives up
    PhysR<R> p;
    int ny, nx, use_forcing;
};

// -------------------------------------------------------------------------
// Block factors of the linear smoothers.  During a linear solve the state is
// fixed, so each cell's 5x5 block (local Newton matrix + damping, pinned
// rows, transposed for the adjoint) is factored once per V-cycle and stored:
// 25 values per cell, structure-of-arrays (value k of cell (i,j) at
// f[k * plane + i * pitch + j]), L below the diagonal, U above it and the
// pivot reciprocals on it.  The smoother then costs one triangular solve.
//
// The binary32 tangent smoother (the forward direction) stores its factors
// in bfloat16 pairs (8 significant bits, the binary32 exponent range) and
// solves with them in binary32: the stored factors are 25 of the 34 values a
// sweep moves per cell, and the smoother needs only an approximate inverse,
// since the Newton residual it serves covers every row.  The adjoint keeps
// binary32 factors: its sweep zeroes the pinned rows' right-hand side, so
// the values next to them are the smoother's own and would carry the
// factors' rounding into the converged adjoint.  Binary64 smoothers keep
// binary64 factors.  The buffer is sized for R either way.
// -------------------------------------------------------------------------
// Storage of one cell's 25 factors: kPlanes planes of `type`, at
// f[q * plane + i * pitch + j].
template <class R, bool TR>
struct FactorStore {
    using type = R;
    static constexpr int kPlanes = 25;
    static __device__ __forceinline__ void put(R* base, size_t plane, size_t at, const R (&M)[25]) {
        R* f = base + at;
#pragma unroll
        for (int k = 0; k < 25; ++k) f[k * plane] = M[k];
    }
    static __device__ __forceinline__ void get(const R* base, size_t plane, size_t at, R (&M)[25]) {
        const R* f = base + at;
#pragma unroll
        for (int k = 0; k < 25; ++k) M[k] = __ldg(f + k * plane);
    }
};
// bfloat16 pairs: factors 2q and 2q + 1 in plane q (factor 24 alone in plane
// 12), one 4-byte load per pair.
template <>
struct FactorStore<float, false> {
    using type = __nv_bfloat162;
    static constexpr int kPlanes = 13;
    static __device__ __forceinline__ void put(float* base, size_t plane, size_t at, const float (&M)[25]) {
        __nv_bfloat162* f = reinterpret_cast<__nv_bfloat162*>(base) + at;
#pragma unroll
        for (int q = 0; q < 13; ++q) f[q * plane] = __floats2bfloat162_rn(M[2 * q], q < 12 ? M[2 * q + 1] : 0.0f);
    }
    static __device__ __forceinline__ void get(const float* base, size_t plane, size_t at, float (&M)[25]) {
        const unsigned* f = reinterpret_cast<const unsigned*>(base) + at;
#pragma unroll
        for (int q = 0; q < 13; ++q) {
            const unsigned w = __ldg(f + q * plane);
            __nv_bfloat162 h;
            static_assert(sizeof(h) == sizeof(w), "a bfloat16 pair is one word");
            memcpy(&h, &w, sizeof(w));
            const float2 v = __bfloat1622float2(h);
            M[2 * q] = v.x;
            if (q < 12) M[2 * q + 1] = v.y;
        }
    }
};

// x = (L U)^-1 b with the stored factors (pivot reciprocals on the diagonal)
template <class R>
__device__ __forceinline__ void block_solve(const R (&M)[25], const R (&b)[5], R (&x)[5]) {
    const R y0 = b[0];
    const R y1 = b[1] - M[5] * y0;
    const R y2 = b[2] - M[10] * y0 - M[11] * y1;
    const R y3 = b[3] - M[15] * y0 - M[16] * y1 - M[17] * y2;
    const R y4 = b[4] - M[20] * y0 - M[21] * y1 - M[22] * y2 - M[23] * y3;
    x[4] = y4 * M[24];
    x[3] = (y3 - M[19] * x[4]) * M[18];
    x[2] = (y2 - M[13] * x[3] - M[14] * x[4]) * M[12];
    x[1] = (y1 - M[7] * x[2] - M[8] * x[3] - M[9] * x[4]) * M[6];
    x[0] = (y0 - M[1] * x[1] - M[2] * x[2] - M[3] * x[3] - M[4] * x[4]) * M[0];
}

template <class R>
struct BlockArgs {
    Arr<R> u, v, H, phi, mask, bed, B, beta;
    Arr<R> ru, rv, rH;  // residual of the linear system (sweep)
    Arr<R> xu, xv, xH;  // unknowns, updated in place (sweep)
    R* f;               // factors (FactorStore<R, TR> layout; the buffer holds 25 planes of R)
    size_t plane;
    int pitch;
    int* err;           // set when a bounded wait gives up
    PhysR<R> p;
    R omega, ssa_damping, mc_damping;
    int ny, nx;
};

template <class R, bool TR, class BLK>
__device__ __forceinline__ void block_factor_tile(const BlockArgs<R>& a, const BoxMaps<7>& maps, BLK blk) {
    using TileT = StateBoxTile<R>;
    constexpr int NC = TileT::NE;
    __shared__ __align__(128) TileT t;
    __shared__ unsigned long long bar;
    const int i0 = blk.y() * kTile, j0 = blk.x() * kTile;
    const int ny = a.ny, nx = a.nx;
    if (!stage_state_boxes<R>(t, maps, a.u, a.v, a.H, a.phi, a.bed, a.beta, a.B, i0, j0, &bar, a.err)) return;
    StateBoxView<R> s{t, i0, j0, ny, nx};
    for (int k = threadIdx.x; k < NC * NC; k += blockDim.x) {
        int r = k / NC, c = k % NC;
        int gi = i0 - 1 + r, gj = j0 - 1 + c;
        t.eta[r][c] = eta_at<R>(s, s.BC(gi, gj), a.p, gi, gj);
    }
    __syncthreads();
    const int i = i0 + threadIdx.x / kTile, j = j0 + threadIdx.x % kTile;
    if (i >= ny || j >= nx) return;
    R x[5] = {s.U(i, j), s.U(i, j + 1), s.V(i, j), s.V(i + 1, j), s.Hc(i, j)};
    R J[25], rr[5];
    local_system<R>(s, a.p, i, j, x, J, rr);
    J[0] -= a.ssa_damping; J[6] -= a.ssa_damping; J[12] -= a.ssa_damping; J[18] -= a.ssa_damping;
    J[24] += a.mc_damping;
    if (j == 0) pin(J, 0);
    if (j == nx - 1) pin(J, 1);
    if (i == 0) pin(J, 2);
    if (i == ny - 1) pin(J, 3);
    if (a.mask.at(i, j) > R(0.5)) pin(J, 4);
    R M[25];
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int c = 0; c < 5; ++c) M[r * 5 + c] = TR ? J[c * 5 + r] : J[r * 5 + c];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const R inv = R(1) / M[k * 5 + k];
#pragma unroll
        for (int r = k + 1; r < 5; ++r) {
            M[r * 5 + k] *= inv;
#pragma unroll
            for (int c = k + 1; c < 5; ++c) M[r * 5 + c] -= M[r * 5 + k] * M[k * 5 + c];
        }
        M[k * 5 + k] = inv;
    }
    FactorStore<R, TR>::put(a.f, a.plane, size_t(i) * a.pitch + j, M);
}

template <class R, bool TR>
__global__ void __launch_bounds__(kTile * kTile)
    k_block_factor(BlockArgs<R> a, const __grid_constant__ BoxMaps<7> maps) {
    block_factor_tile<R, TR>(a, maps, SoloBlock{});
}

// One linear block-smoother sweep with stored factors: x += omega * delta
// with delta = B^-1 (f - Op x) per cell, face corrections averaged between
// the two cells of a face (adjoint: lambda -= omega * B^-T r, r = J^T lambda - f).
constexpr int kSweepThreads = kTile * kTile + 2 * kTile;

template <class R, bool TR, class BLK>
__device__ __forceinline__ void block_sweep_tile(const BlockArgs<R>& a, BLK blk) {
    constexpr int ND = kTile + 1;
    __shared__ R dl[ND][ND][4];
    const int i0 = blk.y() * kTile, j0 = blk.x() * kTile;
    const int ny = a.ny, nx = a.nx;
    int i, j;
    const int tid = threadIdx.x;
    if (tid < kTile * kTile) { i = i0 + tid / kTile; j = j0 + tid % kTile; }
    else if (tid < kTile * kTile + kTile) { i = i0 + (tid - kTile * kTile); j = j0 - 1; }
    else { i = i0 - 1; j = j0 + (tid - kTile * kTile - kTile); }
    const bool live = i >= 0 && i < ny && j >= 0 && j < nx;
    // the owned cells' unknowns, loaded with the factors rather than after the
    // barrier (only this thread writes them)
    const bool own = tid < kTile * kTile && live;
    R xu0 = R(0), xv0 = R(0), xh0 = R(0);
    if (own) {
        xu0 = a.xu.at(i, j);
        xv0 = a.xv.at(i, j);
        xh0 = a.xH.at(i, j);
    }
    R d4 = 0;
    R dd[4] = {0, 0, 0, 0};
    if (live) {
        R b[5] = {a.ru.at(i, j), a.ru.at(i, j + 1), a.rv.at(i, j), a.rv.at(i + 1, j), a.rH.at(i, j)};
        if (TR) {  // the adjoint zeroes the pinned rows' right-hand side
            if (j == 0) b[0] = R(0);
            if (j == nx - 1) b[1] = R(0);
            if (i == 0) b[2] = R(0);
            if (i == ny - 1) b[3] = R(0);
            if (a.mask.at(i, j) > R(0.5)) b[4] = R(0);
        }
        R M[25];
        FactorStore<R, TR>::get(a.f, a.plane, size_t(i) * a.pitch + j, M);
        R x[5];
        block_solve<R>(M, b, x);
        for (int q = 0; q < 4; ++q) dd[q] = R(0.5) * x[q];
        d4 = x[4];
    }
    {
        const int di = i - (i0 - 1), dj = j - (j0 - 1);
#pragma unroll
        for (int q = 0; q < 4; ++q) dl[di][dj][q] = dd[q];
    }
    __syncthreads();
    if (own) {
        const int di = i - (i0 - 1), dj = j - (j0 - 1);
        const R w = a.omega;
        R du = (j > 0 ? dl[di][dj - 1][1] : R(0)) + dl[di][dj][0];
        a.xu.at(i, j) = xu0 - w * du;
        if (j == nx - 1) a.xu.at(i, nx) = a.xu.at(i, nx) - w * dl[di][dj][1];
        R dv = (i > 0 ? dl[di - 1][dj][3] : R(0)) + dl[di][dj][2];
        a.xv.at(i, j) = xv0 - w * dv;
        if (i == ny - 1) a.xv.at(ny, j) = a.xv.at(ny, j) - w * dl[di][dj][3];
        a.xH.at(i, j) = xh0 - w * d4;
    }
}

template <class R, bool TR>
__global__ void __launch_bounds__(kSweepThreads) k_block_sweep(BlockArgs<R> a) {
    block_sweep_tile<R, TR>(a, SoloBlock{});
}

// -------------------------------------------------------------------------
// Gradients (grad.cu:2-169, glide/operators.py:589-593), gathered per cell
// with the reference's index guards.
// -------------------------------------------------------------------------
template <class R>
struct GradArgs {
    Arr<R> u, v, H, phi, bed, beta;
    Arr<R> lu, lv, lH;
    Arr<R> g_beta, g_bed, g_Hp, g_smb;
    PhysR<R> p;
    R dt;
    int ny, nx;
};

template <class R>
struct GView {
    const GradArgs<R>& a;
    int ny, nx;
    __device__ R U(int i, int j) const { return a.u.at(clampi(i, 0, ny - 1), clampi(j, 0, nx)); }
    __device__ R V(int i, int j) const { return a.v.at(clampi(i, 0, ny), clampi(j, 0, nx - 1)); }
    __device__ R C(const Arr<R>& f, int i, int j) const { return f.at(clampi(i, 0, ny - 1), clampi(j, 0, nx - 1)); }
};

template <class R>
__device__ __forceinline__ void gradients_at(const GradArgs<R>& a, int I, int J) {
    const int ny = a.ny, nx = a.nx;
    if (J >= nx) return;
    GView<R> g{a, ny, nx};
    const R dxi = a.p.dxi;
    // basal drag / driving stress of u face (i, j)
    auto ub = [&](int i, int j) {
        return basal(g.U(i, j), g.V(i, j - 1), g.V(i, j), g.V(i + 1, j - 1), g.V(i + 1, j), g.C(a.phi, i, j - 1),
                     g.C(a.phi, i, j), g.C(a.beta, i, j - 1), g.C(a.beta, i, j), a.p);
    };
    auto ud = [&](int i, int j) {
        return driving(g.C(a.H, i, j - 1), g.C(a.H, i, j), g.C(a.bed, i, j - 1), g.C(a.bed, i, j),
                       g.C(a.phi, i, j - 1), g.C(a.phi, i, j), dxi, j, nx);
    };
    auto vb = [&](int i, int j) {
        return basal(g.V(i, j), g.U(i - 1, j), g.U(i - 1, j + 1), g.U(i, j), g.U(i, j + 1), g.C(a.phi, i - 1, j),
                     g.C(a.phi, i, j), g.C(a.beta, i - 1, j), g.C(a.beta, i, j), a.p);
    };
    auto vd = [&](int i, int j) {
        return driving(g.C(a.H, i, j), g.C(a.H, i - 1, j), g.C(a.bed, i, j), g.C(a.bed, i - 1, j),
                       g.C(a.phi, i, j), g.C(a.phi, i - 1, j), dxi, i, ny);
    };
    if (a.g_beta.p) {
        R s = a.lu.at(I, J + 1) * ub(I, J + 1).d_b0;
        if (J < nx - 1) s += a.lu.at(I, J) * ub(I, J).d_b1;
        s += a.lv.at(I + 1, J) * vb(I + 1, J).d_b0;
        if (I < ny - 1) s += a.lv.at(I, J) * vb(I, J).d_b1;
        a.g_beta.at(I, J) = s;
    }
    if (a.g_bed.p) {
        R s = -a.lu.at(I, J + 1) * ud(I, J + 1).d_b0;
        if (J < nx - 1) s += -a.lu.at(I, J) * ud(I, J).d_b1;
        s += -a.lv.at(I + 1, J) * vd(I + 1, J).d_b1;
        if (I < ny - 1) s += -a.lv.at(I, J) * vd(I, J).d_b0;
        a.g_bed.at(I, J) = s;
    }
    if (a.g_Hp.p) a.g_Hp.at(I, J) = -a.lH.at(I, J) / a.dt;
    if (a.g_smb.p) a.g_smb.at(I, J) = -a.lH.at(I, J);
}

template <class R>
__global__ void k_gradients(GradArgs<R> a) {
    gradients_at(a, blockIdx.y, blockIdx.x * blockDim.x + threadIdx.x);
}

}  // namespace glide
