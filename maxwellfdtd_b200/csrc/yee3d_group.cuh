// yee3d_group.cuh -- single-precision 3-D cell updates, W cells of a row per thread (sm_100a).
//
// The cell code of h3d_cell / e3d_cell costs a batched 3-D half-step some 470 instructions per
// cell, most of them addresses, boundary conditions, layer tests and four-byte loads and stores,
// and the batch was short of issue slots (55 % active) with every warp slot in use.  A group of W
// cells x0 .. x0 + W - 1 (x0 a multiple of W) shares them: one aligned access of 4 W bytes per
// array, one set of neighbour offsets, one test per layer face.  A row's last, partial group
// computes W cells (the padding is allocated) and stores the row's own.  The arithmetic is
// h3d_cell's and e3d_cell's, expression for expression: results are bit-identical.  What bounds a
// batch now is the latency of its loads at half of the warp slots.
#pragma once

#include "yee3d_split.cuh"

namespace mfd {

template <int W>
__device__ __forceinline__ void g_load(const float* p, float (&v)[W]) {
    static_assert(W == 2, "the accesses are of two cells");
    const float2 a = *reinterpret_cast<const float2*>(p);
    v[0] = a.x; v[1] = a.y;
}
// nv: how many of the cells lie in the row (the padding behind it stays zero).
template <int W>
__device__ __forceinline__ void g_store(float* p, const float (&v)[W], int nv) {
    static_assert(W == 2, "the accesses are of two cells");
    if (nv == W) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else p[0] = v[0];
}
// The material indices of a group, packed (byte j: cell j).
template <int W>
__device__ __forceinline__ unsigned g_geom(const uint8_t* p) {
    static_assert(W == 2, "the accesses are of two cells");
    return *reinterpret_cast<const unsigned short*>(p);
}

// One CPML face of axis AX (0 x, 1 y, 2 z) of a group: the psi pair P, P + 1 of derivatives da, db
// (cpml_h and cpml_e in yee.cuh).  Every load of the face comes before its first store; the psi
// terms of cell j go to field(j, pa, pb).  An x face may hold some of the cells only.
template <int AX, int P, int FAST, int W, typename F>
__device__ __forceinline__ void g_face(const LayerDev<float>& l, bool right, bool k1, const Layout& L, int x0, int nv, int iy, int iz,
                                       float (&da)[W], float (&db)[W], F&& field) {
    if (!l.nb) return;
    float pa[W], pb[W];
    if constexpr (AX == 0) {
        if (right ? x0 + nv <= l.ib - 1 : x0 >= l.ib) return;
        const int q = right ? x0 - (l.ib - 1) : x0;   // of cell 0; may lie before the layer
        const int k = q + l.nb * (iy + L.ny * iz);
        unsigned in = 0;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            pa[j] = pb[j] = 0.0f;
            if (j < nv && (right ? q + j >= 0 : x0 + j < l.ib)) {
                in |= 1u << j;
                pa[j] = l.psi[P][k + j];
                pb[j] = l.psi[P + 1][k + j];
            }
        }
#pragma unroll
        for (int j = 0; j < W; ++j) {
            if (!(in >> j & 1u)) continue;
            const float B = l.B[q + j], A = l.A[q + j];
            pa[j] = mad<FAST>(B, pa[j], A * da[j]);
            pb[j] = mad<FAST>(B, pb[j], A * db[j]);
            l.psi[P][k + j] = pa[j];
            l.psi[P + 1][k + j] = pb[j];
            field(j, pa[j], pb[j]);
            if (!k1) {
                da[j] = cdiv<FAST>(da[j], l.K[q + j]);
                db[j] = cdiv<FAST>(db[j], l.K[q + j]);
            }
        }
    } else {
        const int i = AX == 1 ? iy : iz;
        if (right ? i < l.ib - 1 : i >= l.ib) return;
        const int q = right ? i - (l.ib - 1) : i;
        const int k = x0 + L.px * (AX == 1 ? q + l.nb * iz : iy + L.ny * q);
        g_load<W>(l.psi[P] + k, pa);
        g_load<W>(l.psi[P + 1] + k, pb);
        const float B = l.B[q], A = l.A[q];
#pragma unroll
        for (int j = 0; j < W; ++j) {
            pa[j] = mad<FAST>(B, pa[j], A * da[j]);
            pb[j] = mad<FAST>(B, pb[j], A * db[j]);
            field(j, pa[j], pb[j]);
            if (!k1) {
                da[j] = cdiv<FAST>(da[j], l.K[q]);
                db[j] = cdiv<FAST>(db[j], l.K[q]);
            }
        }
        g_store<W>(l.psi[P] + k, pa, nv);
        g_store<W>(l.psi[P + 1] + k, pb, nv);
    }
}

// Cells x0 .. x0 + W - 1 (x0 a multiple of W below nx) of row (iy, iz).  acc: the running sums of
// the previous step; k1: every kappa is 1.
template <bool MATH, int FAST, int W>
__device__ __forceinline__ void h3d_group(const HParams<float>& p, const Div3& D3, bool k1, bool acc, long long prev_step, int x0, int iy,
                                          int iz) {
    const int nx = p.L.nx, ny = p.L.ny, nz = p.L.nz, sy = p.L.px, sz = p.L.sz;
    const int nv = min(W, nx - x0), c = x0 + sy * iy + sz * iz;
    const bool xr = x0 + W >= nx, yr = iy == ny - 1, zr = iz == nz - 1;
    const int bx = p.bc[MFD_XR], by = p.bc[MFD_YR], bz = p.bc[MFD_ZR];
    const int ox = !xr ? W : bx == MFD_BC_PERIODIC ? -x0 : nv - 1;
    const int oy = !yr ? sy : by == MFD_BC_PERIODIC ? -(ny - 1) * sy : 0;
    const int oz = !zr ? sz : bz == MFD_BC_PERIODIC ? -(nz - 1) * sz : 0;
    float ex[W], ey[W], ez[W], hx[W], hy[W], hz[W], exy[W], ezy[W], exz[W], eyz[W];
    g_load<W>(p.Ex + c, ex);
    g_load<W>(p.Ey + c, ey);
    g_load<W>(p.Ez + c, ez);
    float eyx = p.Ey[c + ox], ezx = p.Ez[c + ox];   // x + 1 of the last cell
    g_load<W>(p.Ex + (c + oy), exy);
    g_load<W>(p.Ez + (c + oy), ezy);
    g_load<W>(p.Ex + (c + oz), exz);
    g_load<W>(p.Ey + (c + oz), eyz);
    g_load<W>(p.Hx + c, hx);
    g_load<W>(p.Hy + c, hy);
    g_load<W>(p.Hz + c, hz);
    const unsigned g = MATH ? g_geom<W>(p.geom + c) : 0u;
    if (acc) {
        float sa[W], e2[W];
        g_load<W>(p.Sa + c, sa);
#pragma unroll
        for (int j = 0; j < W; ++j) e2[j] = 0.0f;
        if (p.sum_e2) g_load<W>(p.E2 + c, e2);
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const float a = mad<FAST>(ey[j], hz[j], -(ez[j] * hy[j])), b = mad<FAST>(ez[j], hx[j], -(ex[j] * hz[j])),
                        d = mad<FAST>(ex[j], hy[j], -(ey[j] * hx[j]));
            sa[j] = mad<FAST>(sqrtm<FAST>(sum3sq<FAST>(a, b, d)), p.dt, sa[j]);
            e2[j] = mad<FAST>(sum3sq<FAST>(ex[j], ey[j], ez[j]), p.dt, e2[j]);
            if (j < nv && maybe_nonfinite(ex[j])) guard_at(p.flags, prev_step, ex[j]);
        }
        g_store<W>(p.Sa + c, sa, nv);
        if (p.sum_e2) g_store<W>(p.E2 + c, e2, nv);
    }
    if (xr && bx == MFD_BC_DIRICHLET) eyx = ezx = 0.0f;
    if (yr && by == MFD_BC_DIRICHLET) {
#pragma unroll
        for (int j = 0; j < W; ++j) exy[j] = ezy[j] = 0.0f;
    }
    if (zr && bz == MFD_BC_DIRICHLET) {
#pragma unroll
        for (int j = 0; j < W; ++j) exz[j] = eyz[j] = 0.0f;
    }
    float Mh[W];
#pragma unroll
    for (int j = 0; j < W; ++j) {
        Mh[j] = p.Mh0;
        if (MATH && (g >> 8 * j & 255u)) Mh[j] = p.matMh[(g >> 8 * j & 255u) - 1];
    }
    float dExy[W], dExz[W], dEyx[W], dEyz[W], dEzx[W], dEzy[W];
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const bool last = j == W - 1 || j == nv - 1;
        const float ey1 = last ? eyx : ey[j < W - 1 ? j + 1 : j], ez1 = last ? ezx : ez[j < W - 1 ? j + 1 : j];
        const float num[6] = {exy[j] - ex[j], exz[j] - ex[j], ey1 - ey[j], eyz[j] - ey[j], ez1 - ez[j], ezy[j] - ez[j]};
        float q[6];
        div6<FAST>(D3, num, q);
        dExy[j] = q[0]; dExz[j] = q[1]; dEyx[j] = q[2]; dEyz[j] = q[3]; dEzx[j] = q[4]; dEzy[j] = q[5];
    }
    auto fx = [&](int j, float pa, float pb) { hy[j] = mad<FAST>(Mh[j], pb, hy[j]); hz[j] = mad<FAST>(-Mh[j], pa, hz[j]); };
    auto fy = [&](int j, float pa, float pb) { hx[j] = mad<FAST>(-Mh[j], pb, hx[j]); hz[j] = mad<FAST>(Mh[j], pa, hz[j]); };
    auto fz = [&](int j, float pa, float pb) { hx[j] = mad<FAST>(Mh[j], pb, hx[j]); hy[j] = mad<FAST>(-Mh[j], pa, hy[j]); };
    g_face<0, 2, FAST, W>(p.lay[MFD_XL], false, k1, p.L, x0, nv, iy, iz, dEyx, dEzx, fx);
    g_face<0, 2, FAST, W>(p.lay[MFD_XR], true, k1, p.L, x0, nv, iy, iz, dEyx, dEzx, fx);
    g_face<1, 2, FAST, W>(p.lay[MFD_YL], false, k1, p.L, x0, nv, iy, iz, dExy, dEzy, fy);
    g_face<1, 2, FAST, W>(p.lay[MFD_YR], true, k1, p.L, x0, nv, iy, iz, dExy, dEzy, fy);
    g_face<2, 2, FAST, W>(p.lay[MFD_ZL], false, k1, p.L, x0, nv, iy, iz, dExz, dEyz, fz);
    g_face<2, 2, FAST, W>(p.lay[MFD_ZR], true, k1, p.L, x0, nv, iy, iz, dExz, dEyz, fz);
#pragma unroll
    for (int j = 0; j < W; ++j) {
        hx[j] = mad<FAST>(-Mh[j], dEzy[j] - dEyz[j], hx[j]);
        hy[j] = mad<FAST>(-Mh[j], dExz[j] - dEzx[j], hy[j]);
        hz[j] = mad<FAST>(-Mh[j], dEyx[j] - dExy[j], hz[j]);
    }
    g_store<W>(p.Hx + c, hx, nv);
    g_store<W>(p.Hy + c, hy, nv);
    g_store<W>(p.Hz + c, hz, nv);
}

template <typename R, bool MAT, int FAST, int W>
__device__ __forceinline__ void e3d_group(const EParams<float, R>& p, const Div3& D3, bool k1, int x0, int iy, int iz) {
    const int nx = p.L.nx, ny = p.L.ny, nz = p.L.nz, sy = p.L.px, sz = p.L.sz;
    const int nv = min(W, nx - x0), c = x0 + sy * iy + sz * iz;
    const bool xl = x0 == 0, yl = iy == 0, zl = iz == 0;
    const int bx = p.bc[MFD_XL], by = p.bc[MFD_YL], bz = p.bc[MFD_ZL];
    const int ox = !xl ? -1 : bx == MFD_BC_PERIODIC ? nx - 1 : 0;
    const int oy = !yl ? -sy : by == MFD_BC_PERIODIC ? (ny - 1) * sy : 0;
    const int oz = !zl ? -sz : bz == MFD_BC_PERIODIC ? (nz - 1) * sz : 0;
    float hx[W], hy[W], hz[W], hxy[W], hzy[W], hxz[W], hyz[W], D0[W], D1[W], D2[W];
    g_load<W>(p.Hx + c, hx);
    g_load<W>(p.Hy + c, hy);
    g_load<W>(p.Hz + c, hz);
    float hyl = p.Hy[c + ox], hzl = p.Hz[c + ox];   // x - 1 of the first cell
    g_load<W>(p.Hx + (c + oy), hxy);
    g_load<W>(p.Hz + (c + oy), hzy);
    g_load<W>(p.Hx + (c + oz), hxz);
    g_load<W>(p.Hy + (c + oz), hyz);
    g_load<W>(p.Dx + c, D0);
    g_load<W>(p.Dy + c, D1);
    g_load<W>(p.Dz + c, D2);
    const unsigned g = MAT ? g_geom<W>(p.geom + c) : 0u;
    if (xl && bx == MFD_BC_DIRICHLET) hyl = hzl = 0.0f;
    if (yl && by == MFD_BC_DIRICHLET) {
#pragma unroll
        for (int j = 0; j < W; ++j) hxy[j] = hzy[j] = 0.0f;
    }
    if (zl && bz == MFD_BC_DIRICHLET) {
#pragma unroll
        for (int j = 0; j < W; ++j) hxz[j] = hyz[j] = 0.0f;
    }
    float Md1[W], Md2[W], Me[W];
    unsigned resp = 0;   // cells whose E comes from the material kernel
#pragma unroll
    for (int j = 0; j < W; ++j) {
        Md1[j] = p.Md10; Md2[j] = p.Md20; Me[j] = p.Me0;
        const unsigned gj = g >> 8 * j & 255u;
        if (MAT && gj) {
            const MatDev<float, R>& m = p.mats[gj - 1];
            Md1[j] = m.Md1; Md2[j] = m.Md2; Me[j] = m.Me;
            if (!m.simple) resp |= 1u << j;
        }
    }
    float dHxy[W], dHxz[W], dHyx[W], dHyz[W], dHzx[W], dHzy[W];
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const float num[6] = {hx[j] - hxy[j], hx[j] - hxz[j], hy[j] - (j ? hy[j - (j > 0)] : hyl), hy[j] - hyz[j],
                              hz[j] - (j ? hz[j - (j > 0)] : hzl), hz[j] - hzy[j]};
        float q[6];
        div6<FAST>(D3, num, q);
        dHxy[j] = q[0]; dHxz[j] = q[1]; dHyx[j] = q[2]; dHyz[j] = q[3]; dHzx[j] = q[4]; dHzy[j] = q[5];
    }
    auto fx = [&](int j, float pa, float pb) { D1[j] = mad<FAST>(-Md2[j], pb, D1[j]); D2[j] = mad<FAST>(Md2[j], pa, D2[j]); };
    auto fy = [&](int j, float pa, float pb) { D0[j] = mad<FAST>(Md2[j], pb, D0[j]); D2[j] = mad<FAST>(-Md2[j], pa, D2[j]); };
    auto fz = [&](int j, float pa, float pb) { D0[j] = mad<FAST>(-Md2[j], pb, D0[j]); D1[j] = mad<FAST>(Md2[j], pa, D1[j]); };
    g_face<0, 0, FAST, W>(p.lay[MFD_XL], false, k1, p.L, x0, nv, iy, iz, dHyx, dHzx, fx);
    g_face<0, 0, FAST, W>(p.lay[MFD_XR], true, k1, p.L, x0, nv, iy, iz, dHyx, dHzx, fx);
    g_face<1, 0, FAST, W>(p.lay[MFD_YL], false, k1, p.L, x0, nv, iy, iz, dHxy, dHzy, fy);
    g_face<1, 0, FAST, W>(p.lay[MFD_YR], true, k1, p.L, x0, nv, iy, iz, dHxy, dHzy, fy);
    g_face<2, 0, FAST, W>(p.lay[MFD_ZL], false, k1, p.L, x0, nv, iy, iz, dHxz, dHyz, fz);
    g_face<2, 0, FAST, W>(p.lay[MFD_ZR], true, k1, p.L, x0, nv, iy, iz, dHxz, dHyz, fz);
#pragma unroll
    for (int j = 0; j < W; ++j) {
        D0[j] = mad<FAST>(Md1[j], D0[j], Md2[j] * (dHzy[j] - dHyz[j]));
        D1[j] = mad<FAST>(Md1[j], D1[j], Md2[j] * (dHxz[j] - dHzx[j]));
        D2[j] = mad<FAST>(Md1[j], D2[j], Md2[j] * (dHyx[j] - dHxy[j]));
    }
    g_store<W>(p.Dx + c, D0, nv);
    g_store<W>(p.Dy + c, D1, nv);
    g_store<W>(p.Dz + c, D2, nv);
    if (MAT && resp) {
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (j < nv && !(resp >> j & 1u)) {
                p.Ex[c + j] = D0[j] * Me[j];
                p.Ey[c + j] = D1[j] * Me[j];
                p.Ez[c + j] = D2[j] * Me[j];
            }
    } else {
#pragma unroll
        for (int j = 0; j < W; ++j) { D0[j] *= Me[j]; D1[j] *= Me[j]; D2[j] *= Me[j]; }
        g_store<W>(p.Ex + c, D0, nv);
        g_store<W>(p.Ey + c, D1, nv);
        g_store<W>(p.Ez + c, D2, nv);
    }
}

}  // namespace mfd
