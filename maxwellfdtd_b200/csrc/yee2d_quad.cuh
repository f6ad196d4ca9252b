// yee2d_quad.cuh -- single-precision 2-D updates (Hy, Dx, Dz, Ex, Ez), four cells of a row per
// thread (sm_100a).
//
// One cell per thread (h2d_kernel / e2d_kernel) spends about 130 instructions and 8 four-byte
// loads on a cell, and what bounded it was the latency of those loads at full occupancy: a third
// of DRAM throughput.  Rows are padded to 32 elements, so four cells x0 .. x0 + 3 (x0 a multiple
// of 4) are one aligned 16-byte load per array: a quarter of the requests and of the address and
// boundary work per cell, four times the bytes in flight per thread.  The E update also takes the
// material response of its cells (up to three poles, Kerr; no plasma) right after their D update,
// so that D and E are not read again by a launch of their own.  The last, partial group of a row
// computes four cells too (the padding is allocated) and stores only the row's own.  The
// arithmetic is h2d_cell's, e2d_cell's and material_cell_n's, expression for expression, so results
// are bit-identical.
//
// Measured per step: 1801 x 1203 cells with Drude and Lorentz media, tolerance mode 57.6 us with
// one cell per thread and the material kernel, 37.1 now (41.6 with the psi loads after the first
// stores; the batched kernels, which hold their parameters in shared memory, spill with them ahead:
// 262 -> 287 us, so they keep them behind); 32 batched
// models of 128-1024 cells a side, exact mode 277 us, 250 now (latency: 45 % of the warps active).
#pragma once

#include "yee.cuh"

namespace mfd {

__device__ __forceinline__ void q_load(const float* p, float (&v)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
// nv: how many of the four cells lie in the row (the padding behind it stays zero).
__device__ __forceinline__ void q_store(float* p, const float (&v)[4], int nv) {
    if (nv == 4) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (j < nv) p[j] = v[j];
    }
}

// q[j] = x[j] / d as cdiv<FAST> gives it, one band test for the four.
template <int FAST>
__device__ __forceinline__ void q_div(const DivC<float>& D, const float (&x)[4], float (&q)[4]) {
    if constexpr (FAST == DIV_EXACT) {
        unsigned mn = 0xffffffffu, mx = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            q[j] = qcorr(x[j], D.d, D.r);
            const unsigned ax = __float_as_uint(x[j]) & 0x7fffffffu;
            mn = min(mn, ax - 1u);   // zero wraps to the maximum
            mx = max(mx, ax);
        }
        const unsigned lob1 = D.lob - 1u, hib = D.lob + D.span;
        if (mn >= lob1 && mx <= hib) return;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned ax = __float_as_uint(x[j]) & 0x7fffffffu;
            if (ax != 0u && (ax - 1u < lob1 || ax > hib)) q[j] = qscaled(x[j], D.d, D.r, lob1, hib);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = cdiv<FAST>(x[j], D);
    }
}

// One CPML face of four cells: psi row P of the face, derivative d; u = psi for the field, d over
// kappa.  An x face holds some of the cells (psi and profile by cell), a z face the whole row.
template <int P, int FAST, typename F>
__device__ __forceinline__ void q_face_x(const LayerDev<float>& l, bool right, bool k1, int x0, int nv, int iz, float (&d)[4], F&& field) {
    if (!l.nb || (right ? x0 + 3 < l.ib - 1 : x0 >= l.ib)) return;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int ix = x0 + j;
        if (j >= nv || (right ? ix < l.ib - 1 : ix >= l.ib)) continue;
        const int q = right ? ix - (l.ib - 1) : ix, k = q + l.nb * iz;
        const float ps = l.B[q] * l.psi[P][k] + l.A[q] * d[j];
        l.psi[P][k] = ps;
        field(j, ps);
        if (!k1) d[j] = cdiv<FAST>(d[j], l.K[q]);
    }
}
template <int P, int FAST, typename F>
__device__ __forceinline__ void q_face_z(const LayerDev<float>& l, bool right, bool k1, int px, int x0, int nv, int iz, float (&d)[4], F&& field) {
    if (!l.nb || (right ? iz < l.ib - 1 : iz >= l.ib)) return;
    const int q = right ? iz - (l.ib - 1) : iz;
    float* at = l.psi[P] + (x0 + px * q);
    float ps[4];
    q_load(at, ps);
    const float B = l.B[q], A = l.A[q];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        ps[j] = B * ps[j] + A * d[j];
        field(j, ps[j]);
        if (!k1) d[j] = cdiv<FAST>(d[j], l.K[q]);
    }
    q_store(at, ps, nv);
}

// The same with the psi loads apart (a kernel with registers to spare):
// One CPML face of four cells, x (Z false: it may hold some of the cells only, in: bits) or z: psi
// row P of derivative d.  load() issues the psi loads with the group's field loads, before any
// store; step() computes, stores and passes cell j's psi to field(j, psi).
template <bool Z, int P>
struct QFace {
    unsigned in = 0;
    int q, k;
    float ps[4];

    __device__ __forceinline__ void load(const LayerDev<float>& l, bool right, int px, int x0, int nv, int iz) {
        in = 0;
        if (!l.nb) return;
        if constexpr (Z) {
            if (right ? iz < l.ib - 1 : iz >= l.ib) return;
            q = right ? iz - (l.ib - 1) : iz;
            k = x0 + px * q;
            in = 15u;
            q_load(l.psi[P] + k, ps);
        } else {
            if (right ? x0 + nv <= l.ib - 1 : x0 >= l.ib) return;
            q = right ? x0 - (l.ib - 1) : x0;   // of cell 0; may lie before the layer
            k = q + l.nb * iz;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                ps[j] = 0.0f;
                if (j < nv && (right ? q + j >= 0 : x0 + j < l.ib)) {
                    in |= 1u << j;
                    ps[j] = l.psi[P][k + j];
                }
            }
        }
    }

    template <int FAST, typename F>
    __device__ __forceinline__ void step(const LayerDev<float>& l, bool k1, int nv, float (&d)[4], F&& field) {
        if (!in) return;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!Z && !(in >> j & 1u)) continue;
            const int qj = Z ? q : q + j;
            ps[j] = l.B[qj] * ps[j] + l.A[qj] * d[j];
            if (!Z) l.psi[P][k + j] = ps[j];
            field(j, ps[j]);
            if (!k1) d[j] = cdiv<FAST>(d[j], l.K[qj]);
        }
        if (Z) q_store(l.psi[P] + k, ps, nv);
    }
};

// Both faces of an axis.  A group in both of them (it spans the gap of two x layers, or the layers
// overlap) loads the right one's psi after the left one's step.
template <bool Z, int P>
struct QAxis {
    QFace<Z, P> f;
    bool right;
    __device__ __forceinline__ void load(const LayerDev<float>& l, const LayerDev<float>& r, int px, int x0, int nv, int iz) {
        right = false;
        f.load(l, false, px, x0, nv, iz);
        if (!f.in) {
            right = true;
            f.load(r, true, px, x0, nv, iz);
        }
    }
    template <int FAST, typename F>
    __device__ __forceinline__ void step(const LayerDev<float>& l, const LayerDev<float>& r, int px, bool k1, int x0, int nv, int iz,
                                         float (&d)[4], F&& field) {
        f.template step<FAST>(right ? r : l, k1, nv, d, field);
        if (!right && f.in && r.nb) {
            f.load(r, true, px, x0, nv, iz);
            f.template step<FAST>(r, k1, nv, d, field);
        }
    }
};

// Cells x0 .. x0 + 3 of row iz (x0 a multiple of 4 below nx).  k1: every kappa is 1.
template <bool MATH, int FAST, bool PRE = false>
__device__ __forceinline__ void h2d_quad(const HParams<float>& p, bool k1, int accum, long long prev_step, int x0, int iz) {
    const int nx = p.L.nx, nz = p.L.nz, sz = p.L.sz;
    const int nv = min(4, nx - x0);
    const int c = x0 + sz * iz;
    float ex[4], ez[5], up[4], hy[4], sa[4] = {0.0f, 0.0f, 0.0f, 0.0f}, e2[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    q_load(p.Ex + c, ex);
    {
        float t[4];
        q_load(p.Ez + c, t);
#pragma unroll
        for (int j = 0; j < 4; ++j) ez[j] = t[j];
    }
    // the z+1 row and the x+1 column of the last cell; across a grid face the boundary's value
    const bool xr = x0 + 4 >= nx, zr = iz == nz - 1;
    const int bx = p.bc[MFD_XR], bz = p.bc[MFD_ZR];
    ez[4] = p.Ez[c + (!xr ? 4 : bx == MFD_BC_PERIODIC ? -x0 : nv - 1)];
    q_load(p.Ex + (c + (!zr ? sz : bz == MFD_BC_PERIODIC ? -(nz - 1) * sz : 0)), up);
    q_load(p.Hy + c, hy);
    QAxis<false, 1> X;
    QAxis<true, 1> Z;
    if (PRE) {
        X.load(p.lay[MFD_XL], p.lay[MFD_XR], p.L.px, x0, nv, iz);
        Z.load(p.lay[MFD_ZL], p.lay[MFD_ZR], p.L.px, x0, nv, iz);
    }
    if (accum) {
        q_load(p.Sa + c, sa);
        if (p.sum_e2) q_load(p.E2 + c, e2);
    }
    uchar4 g = make_uchar4(0, 0, 0, 0);
    if (MATH) g = *reinterpret_cast<const uchar4*>(p.geom + c);
    if (xr) {
        if (bx == MFD_BC_DIRICHLET) ez[4] = 0.0f;
#pragma unroll
        for (int j = 1; j < 4; ++j)
            if (j == nv) ez[j] = ez[4];
    }
    if (zr && bz == MFD_BC_DIRICHLET) {
#pragma unroll
        for (int j = 0; j < 4; ++j) up[j] = 0.0f;
    }
    if (accum) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float a = -ez[j] * hy[j], b = ex[j] * hy[j];
            sa[j] = sa[j] + sqrt0(a * a + b * b) * p.dt;
            e2[j] = e2[j] + (ex[j] * ex[j] + ez[j] * ez[j]) * p.dt;
            if (j < nv && !(fabsf(ex[j]) <= FLT_MAX)) guard_at(p.flags, prev_step, ex[j]);
        }
        q_store(p.Sa + c, sa, nv);
        if (p.sum_e2) q_store(p.E2 + c, e2, nv);
    }
    float Mh[4] = {p.Mh0, p.Mh0, p.Mh0, p.Mh0};
    if (MATH && (g.x | g.y | g.z | g.w)) {
        if (g.x) Mh[0] = p.matMh[g.x - 1];
        if (g.y) Mh[1] = p.matMh[g.y - 1];
        if (g.z) Mh[2] = p.matMh[g.z - 1];
        if (g.w) Mh[3] = p.matMh[g.w - 1];
    }
    float n[4], dz[4], dx[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) n[j] = up[j] - ex[j];
    q_div<FAST>(p.ddz, n, dz);
#pragma unroll
    for (int j = 0; j < 4; ++j) n[j] = ez[j + 1] - ez[j];
    q_div<FAST>(p.ddx, n, dx);
    auto plus = [&](int j, float ps) { hy[j] = mad<FAST>(Mh[j], ps, hy[j]); };
    auto minus = [&](int j, float ps) { hy[j] = mad<FAST>(-Mh[j], ps, hy[j]); };
    if constexpr (PRE) {
        X.template step<FAST>(p.lay[MFD_XL], p.lay[MFD_XR], p.L.px, k1, x0, nv, iz, dx, plus);
        Z.template step<FAST>(p.lay[MFD_ZL], p.lay[MFD_ZR], p.L.px, k1, x0, nv, iz, dz, minus);
    } else {
        q_face_x<1, FAST>(p.lay[MFD_XL], false, k1, x0, nv, iz, dx, plus);
        q_face_x<1, FAST>(p.lay[MFD_XR], true, k1, x0, nv, iz, dx, plus);
        q_face_z<1, FAST>(p.lay[MFD_ZL], false, k1, p.L.px, x0, nv, iz, dz, minus);
        q_face_z<1, FAST>(p.lay[MFD_ZR], true, k1, p.L.px, x0, nv, iz, dz, minus);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) hy[j] = mad<FAST>(-Mh[j], dz[j] - dx[j], hy[j]);
    q_store(p.Hy + c, hy, nv);
}

// Material response of the 128 cells of a warp's groups (x0w: the first), one cell per lane and
// turn: E of the dispersive and Kerr cells from the D that the warp just stored.  Per cell in the
// groups' own threads it took 4 unrolled copies of the code per pole count (stalls on instruction
// fetches) or spilled; here a lane takes a cell of the row, loads are coalesced, one copy runs.
template <typename R>
__device__ __forceinline__ void q_response(const EParams<float, R>& p, int x0w, int iz, int cur) {
    float* Ep[2] = {p.Ex, p.Ez};
#pragma unroll 1
    for (int ix = x0w + (int)(threadIdx.x & 31); ix < min(x0w + 128, p.L.nx); ix += 32) {
        const int c = ix + p.L.sz * iz, g = p.geom[c];
        if (!g) continue;
        const MatDev<float, R>* m = p.mats + (g - 1);
        if (m->simple) continue;
        const float Dv[2] = {p.Dx[c], p.Dz[c]};
        const long long bi = (long long)(ix - m->bx0) + (long long)m->bnx * (iz - m->bz0);
        switch (m->nq) {
            case 0: material_cell_n<float, R, 2, 0, false>(m, bi, Ep, c, Dv, cur, p.dt); break;
            case 1: material_cell_n<float, R, 2, 1, false>(m, bi, Ep, c, Dv, cur, p.dt); break;
            case 2: material_cell_n<float, R, 2, 2, false>(m, bi, Ep, c, Dv, cur, p.dt); break;
            default: material_cell_n<float, R, 2, 3, false>(m, bi, Ep, c, Dv, cur, p.dt); break;
        }
    }
}

// Returns whether some cell's E is left to the material response.
template <typename R, bool MAT, int FAST, bool PRE>
__device__ __forceinline__ bool e2d_quad(const EParams<float, R>& p, bool k1, int x0, int iz) {
    const int nx = p.L.nx, nz = p.L.nz, sz = p.L.sz;
    const int c = x0 + sz * iz;
    const int nv = min(4, nx - x0);
    float hy[4], dn[4], D0[4], D2[4];
    q_load(p.Hy + c, hy);
    const bool xl = x0 == 0, zl = iz == 0;
    const int bx = p.bc[MFD_XL], bz = p.bc[MFD_ZL];
    float left = p.Hy[c + (!xl ? -1 : bx == MFD_BC_PERIODIC ? nx - 1 : 0)];
    q_load(p.Hy + (c + (!zl ? -sz : bz == MFD_BC_PERIODIC ? (nz - 1) * sz : 0)), dn);
    q_load(p.Dx + c, D0);
    q_load(p.Dz + c, D2);
    QAxis<false, 0> X;
    QAxis<true, 0> Z;
    if (PRE) {
        X.load(p.lay[MFD_XL], p.lay[MFD_XR], p.L.px, x0, nv, iz);
        Z.load(p.lay[MFD_ZL], p.lay[MFD_ZR], p.L.px, x0, nv, iz);
    }
    uchar4 g4 = make_uchar4(0, 0, 0, 0);
    if (MAT) g4 = *reinterpret_cast<const uchar4*>(p.geom + c);
    if (xl && bx == MFD_BC_DIRICHLET) left = 0.0f;
    if (zl && bz == MFD_BC_DIRICHLET) {
#pragma unroll
        for (int j = 0; j < 4; ++j) dn[j] = 0.0f;
    }
    float Md1[4], Md2[4], Me[4];
    unsigned resp = 0;   // cells whose E comes from the response
#pragma unroll
    for (int j = 0; j < 4; ++j) { Md1[j] = p.Md10; Md2[j] = p.Md20; Me[j] = p.Me0; }
    const unsigned char g[4] = {g4.x, g4.y, g4.z, g4.w};
    if (MAT && (g4.x | g4.y | g4.z | g4.w)) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (g[j]) {
                const MatDev<float, R>& m = p.mats[g[j] - 1];
                Md1[j] = m.Md1; Md2[j] = m.Md2; Me[j] = m.Me;
                if (!m.simple) resp |= 1u << j;
            }
    }
    float n[4], dx[4], dz[4];
    n[0] = hy[0] - left;
#pragma unroll
    for (int j = 1; j < 4; ++j) n[j] = hy[j] - hy[j - 1];
    q_div<FAST>(p.ddx, n, dx);
#pragma unroll
    for (int j = 0; j < 4; ++j) n[j] = hy[j] - dn[j];
    q_div<FAST>(p.ddz, n, dz);
    auto plus = [&](int j, float ps) { D2[j] = mad<FAST>(Md2[j], ps, D2[j]); };
    auto minus = [&](int j, float ps) { D0[j] = mad<FAST>(-Md2[j], ps, D0[j]); };
    if constexpr (PRE) {
        X.template step<FAST>(p.lay[MFD_XL], p.lay[MFD_XR], p.L.px, k1, x0, nv, iz, dx, plus);
        Z.template step<FAST>(p.lay[MFD_ZL], p.lay[MFD_ZR], p.L.px, k1, x0, nv, iz, dz, minus);
    } else {
        q_face_x<0, FAST>(p.lay[MFD_XL], false, k1, x0, nv, iz, dx, plus);
        q_face_x<0, FAST>(p.lay[MFD_XR], true, k1, x0, nv, iz, dx, plus);
        q_face_z<0, FAST>(p.lay[MFD_ZL], false, k1, p.L.px, x0, nv, iz, dz, minus);
        q_face_z<0, FAST>(p.lay[MFD_ZR], true, k1, p.L.px, x0, nv, iz, dz, minus);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        D0[j] = Md1[j] * D0[j] + Md2[j] * (0.0f - dz[j]);
        D2[j] = Md1[j] * D2[j] + Md2[j] * (dx[j] - 0.0f);
    }
    if (MAT && resp) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j < nv && !(resp >> j & 1u)) {
                p.Ex[c + j] = D0[j] * Me[j];
                p.Ez[c + j] = D2[j] * Me[j];
            }
    } else {
        float e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = D0[j] * Me[j];
        q_store(p.Ex + c, e, nv);
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = D2[j] * Me[j];
        q_store(p.Ez + c, e, nv);
    }
    q_store(p.Dx + c, D0, nv);
    q_store(p.Dz + c, D2, nv);
    return resp != 0;
}

// The E update of a warp's groups (every lane of the warp calls it; act: the lane's group lies in
// the grid).  RESP: with the material response (else a material kernel follows).
template <typename R, bool MAT, int FAST, bool RESP, bool PRE = false>
__device__ __forceinline__ void e2d_warp(const EParams<float, R>& p, bool k1, int cur, bool act, int x0, int iz) {
    const bool resp = act && e2d_quad<R, MAT, FAST, PRE>(p, k1, x0, iz);
    if constexpr (MAT && RESP) {
        if (__any_sync(0xffffffffu, resp)) {
            __syncwarp();
            q_response(p, x0 - 4 * (int)(threadIdx.x & 31), iz, cur);
        }
    }
}

// A block of 32 x Q_TY threads: 128 cells by Q_TY rows.
constexpr int Q_TY = 8;

template <bool MATH, int FAST>
__global__ void __launch_bounds__(32 * Q_TY, 4) h2d_quad_kernel(const __grid_constant__ HParams<float> p, const bool k1) {
    const int x0 = 4 * (blockIdx.x * 32 + threadIdx.x), iz = blockIdx.y * Q_TY + threadIdx.y;
    if (x0 < p.L.nx && iz < p.L.nz) h2d_quad<MATH, FAST, true>(p, k1, p.accum, p.prev_step, x0, iz);
}

template <typename R, bool MAT, int FAST, bool RESP>
__global__ void __launch_bounds__(32 * Q_TY, 4) e2d_quad_kernel(const __grid_constant__ EParams<float, R> p, const bool k1, const int cur) {
    const int x0 = 4 * (blockIdx.x * 32 + threadIdx.x), iz = blockIdx.y * Q_TY + threadIdx.y;
    e2d_warp<R, MAT, FAST, RESP, true>(p, k1, cur, x0 < p.L.nx && iz < p.L.nz, x0, iz);
}

}  // namespace mfd
