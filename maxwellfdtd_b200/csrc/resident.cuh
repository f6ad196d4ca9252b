// resident.cuh -- many time steps of one small model in one cooperative launch (sm_100a).
//
// A small grid's step is a handful of launches of a few microseconds each, whose cost is the
// launches: 21 us per step for 2001 cells in 1-D, 43 us for 61 x 48 x 55 cells, 100 times what
// the cells' bytes take.  Here every block stays on its SM for the whole run of steps.  A block
// owns a contiguous run of cells (x-fastest order) and one thread always updates the same cell,
// so per step the blocks meet only twice, at a grid barrier after the H update and at one after
// the E update:
//   H update (+ running sums and guard of the step before)              | barrier
//   E update, material response, source points on E and D, monitor points | barrier
//   source points on H (and the monitor points of a block that has such)
// A block applies the source points, TFSF points and monitor points that lie in its own cells
// (lists made on the host per block), in the order of the model's sources.  Points on E and D follow
// the block's own E update: between the two barriers no other block reads its E or D.  Points on H
// have to wait for the second barrier: until then other blocks may still read that H for their E
// update.  After it, up to the next barrier, H is read by its own block only, so they go before the
// block's next H update, and the block's monitor points, which read H, go after them.  Order between
// sources matters within one component only, which the split keeps.
//
// The arithmetic is the single-launch kernels' (h1d_kernel ... e3d_cell, material_cell_n, the
// point-source expression, tfsf_point), operation for operation, so results are bit-identical.
// Values that another SM wrote before the last barrier (E in the H update, H in the E update)
// are read past L1 with ld.relaxed.gpu (MemShared below); everything else a thread reads was
// written by its own SM.
//
// What bounds it: an empty barrier of 148 blocks takes 1.1 us, then comes the chain L2 load ->
// arithmetic -> store of about 1 us per half-step for one cell per thread; from about 500 cells
// per SM on the instructions of the cells.  Up to one cell per thread of eight blocks the grid is
// one thread-block cluster with the hardware's barrier (2 001 cells: 4.5 us per step with the grid
// barrier, 3.7 so).  Measured per step, separate launches / resident: 2 001 cells 1-D double
// 20.5 / 3.7 us, 201 x 149 float 15.3 / 5.5, 61 x 48 x 55 float 42.7 / 11.8, 701 x 513 double 25.2 /
// 15.7; the smallest ones vary by 4 % either way with where the pool places their arrays.  The engine's
// resident_limit says up to which size it is used.
#pragma once

#include "aux.cuh"
#include "yee.cuh"
#include "yee3d_split.cuh"

namespace mfd {

// most threads of a block: 640 leave 102 registers a thread, which the single-precision cells
// need (61 x 48 x 55 cells: 13.4 us per step; 512 threads 15.1, 768 13.9); 512 leave 128
template <typename T>
constexpr int RES_THREADS = sizeof(T) == 4 ? 640 : 512;
constexpr int RES_MINCELLS = 128;        // cells per block below which no further block is added
constexpr int RES_CLUSTER = 8;           // blocks of a model that steps as one thread-block cluster
constexpr int RES_MAXOPS = 32;           // sources (and the TFSF replay, one) of a resident model
constexpr unsigned RES_POLLS = 1u << 24; // polls of a barrier before it gives up (seconds)
constexpr int RES_PRE = 3;               // sources whose next waveform value a thread fetches ahead

// One source of the model (the TFSF replay twice: its statements on E and D and those on H), those
// on E and D first, then those on H, each group in the model's tuple order: the points of block b are
// entries list[off[b]] .. list[off[b + 1] - 1] (a point index, or for TFSF the pair (statement, local)).
template <typename T>
struct ResOp {
    int tfsf, kind;
    T coeff;
    T* F;
    const long long* cells;
    const double* wave;
    const double* amp;
    const double* gt;
    long long npts;
    const int* off;
    const int* list;
};

// A block's point of a source or monitor, kept in shared memory.
struct ResPoint {
    int c;        // padded cell
    int m, j;     // monitor (TFSF: statement) and point index
    int pad;
    double amp;   // separable waveform: its amplitude
};

template <typename T>
struct ResidentParams {
    int ncell, per;              // cells of the grid, cells per block
    int nops, nmon;
    const ResOp<T>* ops;
    const RectParams<T>* rp;     // TFSF statements
    const int* moff;             // monitor points of block b: pairs (monitor, point)
    const int* mlist;
    MonParams<T> mp;
    unsigned* bar;               // arrivals at the grid barrier, zero at launch
    int* fault;                  // set when a barrier's wait ran out
    T dt;
    int nmat;
    bool cluster;                // the grid is one thread-block cluster
    bool k1;                     // every CPML kappa is 1 (the default): no division by it
    // byte offsets of the tables a block copies to dynamic shared memory (-1: left in global
    // memory, too large)
    int o_geom, geom_bytes;      // the material map of the block's cells
    int o_mats, o_math;          // material coefficients
    int o_lay[6];                // CPML profiles of a face: K, A, B
    int o_rect;                  // TFSF statements
    int o_mon;                   // monitor descriptors
    int o_ops;                   // the sources
    int o_pts, npts_cap;         // the block's source and monitor points (ResPoint)
    int nops_e;                  // sources on E and D: the first of the nops
};

// Arrive at and wait for the barrier number k (from 1).  Returns false, in every thread of the
// block, when the wait ran out.  A grid of one cluster takes the hardware's cluster barrier (about
// 0.3 us instead of 1.1 through L2), which every thread reaches: there is no wait to run out.
__device__ __forceinline__ bool res_barrier(unsigned* bar, unsigned k, int* fault, int* s_ok, bool cluster) {
    if (cluster) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
    __syncthreads();
    if (gridDim.x == 1) return true;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        const unsigned target = k * gridDim.x;
        unsigned v = 0, polls = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
        } while (v < target && ++polls < RES_POLLS);
        if (v < target) {
            *fault = 1;
            *s_ok = 0;
        }
    }
    __syncthreads();
    return *s_ok != 0;
}

__device__ __forceinline__ void res_copy(void* dst, const void* src, int bytes) {
    for (int i = threadIdx.x; i < bytes; i += blockDim.x) ((char*)dst)[i] = ((const char*)src)[i];
}

// A value that another SM may have written before the last grid barrier: read past L1.
struct MemShared {
    static __device__ __forceinline__ float ld(const float* p) {
        float v;
        asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
        return v;
    }
    static __device__ __forceinline__ double ld(const double* p) {
        double v;
        asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
        return v;
    }
};

// ------------------------------------------------------------------------------------------
// The cell updates in two parts: load() issues every load of the cell, finish() computes and
// stores.  A barrier leaves L1 empty, so a load is a trip to L2; with the stores of one psi pair
// before the loads of the next (the order of h3d_cell) those trips follow one another, here they
// overlap.  The arithmetic is that of h1d_kernel .. e3d_cell, expression for expression.  A cell
// is in at most one CPML face per axis (the engine's rule).
// ------------------------------------------------------------------------------------------
// The CPML face of axis A (0 x, 1 y, 2 z) at index i; rest: the index of its psi row.
template <typename T, int NPSI>
struct ResFace {
    bool in;
    bool right;
    int q, k;
    T v[NPSI];
    template <int A, int P0, int FS, typename P>
    __device__ __forceinline__ void load(const P& p, int ix, int iy, int iz) {
        const LayerDev<T>&l = p.lay[2 * A], &r = p.lay[2 * A + 1];
        const int i = A == 0 ? ix : A == 1 ? iy : iz;
        const bool left = l.nb && i < l.ib;
        right = r.nb && i >= r.ib - 1;
        in = left || right;
        q = right ? i - (r.ib - 1) : i;
        const int nb = right ? r.nb : l.nb;
        const int ny = p.L.ny, px = p.L.px;
        if constexpr (A == 0) k = q + nb * (FS == 3 ? iy + ny * iz : iz);
        else if constexpr (A == 1) k = ix + px * (q + nb * iz);
        else k = FS == 1 ? q : ix + px * (FS == 3 ? iy + ny * q : q);
#pragma unroll
        for (int j = 0; j < NPSI; ++j) v[j] = T(0);
        if (in) {
#pragma unroll
            for (int j = 0; j < NPSI; ++j) v[j] = (right ? r.psi[P0 + j] : l.psi[P0 + j])[k];
        }
    }
    // psi j of derivative d: B psi + A d, stored and returned
    template <int A, int P0, bool FUSE, int FAST, typename P>
    __device__ __forceinline__ T step(const P& p, int j, T d) {
        const LayerDev<T>&l = p.lay[2 * A], &r = p.lay[2 * A + 1];
        const T Bq = (right ? r.B : l.B)[q], Aq = (right ? r.A : l.A)[q];
        T ps;
        if constexpr (FUSE) ps = mad<FAST>(Bq, v[j], Aq * d);
        else ps = Bq * v[j] + Aq * d;
        (right ? r.psi[P0 + j] : l.psi[P0 + j])[k] = ps;
        return ps;
    }
    template <int A, int FAST, typename P>
    __device__ __forceinline__ T over_k(const P& p, bool k1, T d) {
        if (k1) return d;
        const LayerDev<T>&l = p.lay[2 * A], &r = p.lay[2 * A + 1];
        return cdiv<FAST>(d, (right ? r.K : l.K)[q]);
    }
};

// Offset to the neighbour across a face: `at` the cell is on the face, `in` the inner offset,
// `wrap` the periodic one; a Neumann face reads the cell itself, a Dirichlet face zero (zero()).
__device__ __forceinline__ int res_off(bool at, int bc, int in, int wrap) {
    return !at ? in : bc == MFD_BC_PERIODIC ? wrap : 0;
}

template <typename T, int FS, bool MAT, int FAST>
struct ResH {
    static constexpr int NE = FS == 3 ? 9 : FS == 2 ? 4 : FS == 1 ? 2 : 3;   // E values read
    static constexpr int NH = FS == 3 ? 3 : FS == FSET_EY2 ? 2 : 1;
    static constexpr int NP = FS == 3 ? 2 : 1, P0 = FS == 3 ? 2 : 1;          // psi values per face, the first
    T e[NE], h[NH], sa, e2;
    ResFace<T, NP> X, Y, Z;
    int c, g;

    __device__ __forceinline__ void load(const HParams<T>& p, bool acc, int ix, int iy, int iz) {
        const int nx = p.L.nx, ny = p.L.ny, nz = p.L.nz, sy = p.L.px, sz = p.L.sz;
        c = ix + sy * iy + sz * iz;
        const bool xr = ix == nx - 1, yr = iy == ny - 1, zr = iz == nz - 1;
        const int bx = p.bc[MFD_XR], by = p.bc[MFD_YR], bz = p.bc[MFD_ZR];
        const int ox = res_off(xr, bx, 1, -(nx - 1)), oy = res_off(yr, by, sy, -(ny - 1) * sy),
                  oz = res_off(zr, bz, sz, -(nz - 1) * sz);
        if constexpr (FS == 3) {
            e[0] = MemShared::ld(p.Ex + c); e[1] = MemShared::ld(p.Ey + c); e[2] = MemShared::ld(p.Ez + c);
            e[3] = MemShared::ld(p.Ey + (c + ox)); e[4] = MemShared::ld(p.Ez + (c + ox));
            e[5] = MemShared::ld(p.Ex + (c + oy)); e[6] = MemShared::ld(p.Ez + (c + oy));
            e[7] = MemShared::ld(p.Ex + (c + oz)); e[8] = MemShared::ld(p.Ey + (c + oz));
            h[0] = p.Hx[c]; h[1] = p.Hy[c]; h[2] = p.Hz[c];
        } else if constexpr (FS == 2) {
            e[0] = MemShared::ld(p.Ex + c); e[1] = MemShared::ld(p.Ez + c);
            e[2] = MemShared::ld(p.Ez + (c + ox)); e[3] = MemShared::ld(p.Ex + (c + oz));
            h[0] = p.Hy[c];
        } else if constexpr (FS == FSET_EY2) {
            e[0] = MemShared::ld(p.Ey + c);
            e[1] = MemShared::ld(p.Ey + (c + ox)); e[2] = MemShared::ld(p.Ey + (c + oz));
            h[0] = p.Hx[c]; h[1] = p.Hz[c];
        } else {
            e[0] = MemShared::ld(p.Ex + c); e[1] = MemShared::ld(p.Ex + (c + oz));
            h[0] = p.Hy[c];
        }
        sa = acc ? p.Sa[c] : T(0);
        e2 = MAT && acc ? p.E2[c] : T(0);
        if constexpr (FS != 1) X.template load<0, P0, FS>(p, ix, iy, iz);
        if constexpr (FS == 3) Y.template load<1, P0, FS>(p, ix, iy, iz);
        Z.template load<2, P0, FS>(p, ix, iy, iz);
        g = MAT ? (int)p.geom[c] : 0;
        // values across a Dirichlet face are zero
        const bool zx = xr && bx == MFD_BC_DIRICHLET, zy = yr && by == MFD_BC_DIRICHLET, zz = zr && bz == MFD_BC_DIRICHLET;
        if constexpr (FS == 3) {
            if (zx) e[3] = e[4] = T(0);
            if (zy) e[5] = e[6] = T(0);
            if (zz) e[7] = e[8] = T(0);
        } else if constexpr (FS == 2) {
            if (zx) e[2] = T(0);
            if (zz) e[3] = T(0);
        } else if constexpr (FS == FSET_EY2) {
            if (zx) e[1] = T(0);
            if (zz) e[2] = T(0);
        } else {
            if (zz) e[1] = T(0);
        }
    }

    __device__ __forceinline__ void finish(const HParams<T>& p, const Div3& D3, bool k1, bool acc, long long prev_step) {
        T Mh = p.Mh0;
        if (MAT && g) Mh = p.matMh[g - 1];
        if constexpr (FS == 3) {
            const T ex = e[0], ey = e[1], ez = e[2];
            T hx = h[0], hy = h[1], hz = h[2];
            if (acc) {
                const T a = mad<FAST>(ey, hz, -(ez * hy)), b = mad<FAST>(ez, hx, -(ex * hz)), d = mad<FAST>(ex, hy, -(ey * hx));
                p.Sa[c] = mad<FAST>(sqrtm<FAST>(sum3sq<FAST>(a, b, d)), p.dt, sa);
                if (MAT) p.E2[c] = mad<FAST>(sum3sq<FAST>(ex, ey, ez), p.dt, e2);
                if (maybe_nonfinite(ex)) guard_at(p.flags, prev_step, ex);
            }
            const T num[6] = {e[5] - ex, e[7] - ex, e[3] - ey, e[8] - ey, e[4] - ez, e[6] - ez};
            T q[6];
            curl_div<T, FAST>(D3, p.ddx, p.ddy, p.ddz, num, q);
            T dExy = q[0], dExz = q[1], dEyx = q[2], dEyz = q[3], dEzx = q[4], dEzy = q[5];
            if (X.in) {
                const T pa = X.template step<0, 2, true, FAST>(p, 0, dEyx), pb = X.template step<0, 2, true, FAST>(p, 1, dEzx);
                hy = mad<FAST>(Mh, pb, hy);
                hz = mad<FAST>(-Mh, pa, hz);
                dEyx = X.template over_k<0, FAST>(p, k1, dEyx);
                dEzx = X.template over_k<0, FAST>(p, k1, dEzx);
            }
            if (Y.in) {
                const T pa = Y.template step<1, 2, true, FAST>(p, 0, dExy), pb = Y.template step<1, 2, true, FAST>(p, 1, dEzy);
                hx = mad<FAST>(-Mh, pb, hx);
                hz = mad<FAST>(Mh, pa, hz);
                dExy = Y.template over_k<1, FAST>(p, k1, dExy);
                dEzy = Y.template over_k<1, FAST>(p, k1, dEzy);
            }
            if (Z.in) {
                const T pa = Z.template step<2, 2, true, FAST>(p, 0, dExz), pb = Z.template step<2, 2, true, FAST>(p, 1, dEyz);
                hx = mad<FAST>(Mh, pb, hx);
                hy = mad<FAST>(-Mh, pa, hy);
                dExz = Z.template over_k<2, FAST>(p, k1, dExz);
                dEyz = Z.template over_k<2, FAST>(p, k1, dEyz);
            }
            p.Hx[c] = mad<FAST>(-Mh, dEzy - dEyz, hx);
            p.Hy[c] = mad<FAST>(-Mh, dExz - dEzx, hy);
            p.Hz[c] = mad<FAST>(-Mh, dEyx - dExy, hz);
        } else if constexpr (FS == 2) {
            const T ex = e[0], ez = e[1];
            T hy = h[0];
            if (acc) {
                const T a = -ez * hy, b = ex * hy;
                p.Sa[c] = sa + sqrt0(a * a + b * b) * p.dt;
                if (MAT) p.E2[c] = e2 + (ex * ex + ez * ez) * p.dt;
                guard_at(p.flags, prev_step, ex);
            }
            T dExz = cdiv<FAST>(e[3] - ex, p.ddz);
            T dEzx = cdiv<FAST>(e[2] - ez, p.ddx);
            if (X.in) {
                hy = mad<FAST>(Mh, X.template step<0, 1, false, FAST>(p, 0, dEzx), hy);
                dEzx = X.template over_k<0, FAST>(p, k1, dEzx);
            }
            if (Z.in) {
                hy = mad<FAST>(-Mh, Z.template step<2, 1, false, FAST>(p, 0, dExz), hy);
                dExz = Z.template over_k<2, FAST>(p, k1, dExz);
            }
            p.Hy[c] = mad<FAST>(-Mh, dExz - dEzx, hy);
        } else if constexpr (FS == FSET_EY2) {
            const T ey = e[0];
            T hx = h[0], hz = h[1];
            if (acc) {
                const T a = ey * hz, d = T(0) - ey * hx;
                p.Sa[c] = sa + sqrt0(a * a + d * d) * p.dt;
                if (MAT) p.E2[c] = e2 + ey * ey * p.dt;
                guard_at(p.flags, prev_step, ey);
            }
            T dEyx = cdiv<FAST>(e[1] - ey, p.ddx);
            T dEyz = cdiv<FAST>(e[2] - ey, p.ddz);
            if (X.in) {
                hz = mad<FAST>(-Mh, X.template step<0, 1, false, FAST>(p, 0, dEyx), hz);
                dEyx = X.template over_k<0, FAST>(p, k1, dEyx);
            }
            if (Z.in) {
                hx = mad<FAST>(Mh, Z.template step<2, 1, false, FAST>(p, 0, dEyz), hx);
                dEyz = Z.template over_k<2, FAST>(p, k1, dEyz);
            }
            p.Hx[c] = mad<FAST>(-Mh, T(0) - dEyz, hx);
            p.Hz[c] = mad<FAST>(-Mh, dEyx - T(0), hz);
        } else {
            const T ex = e[0];
            T hy = h[0];
            if (acc) {
                const T a = ex * hy;
                p.Sa[c] = sa + sqrt_sq(a) * p.dt;
                if (MAT) p.E2[c] = e2 + ex * ex * p.dt;
                guard_at(p.flags, prev_step, ex);
            }
            T dExz = cdiv<FAST>(e[1] - ex, p.ddz);
            if (Z.in) {
                hy = mad<FAST>(-Mh, Z.template step<2, 1, false, FAST>(p, 0, dExz), hy);
                dExz = Z.template over_k<2, FAST>(p, k1, dExz);
            }
            hy -= Mh * (T(0) + dExz);
            p.Hy[c] = hy;
        }
    }
};

template <typename T, typename R, int FS, bool MAT, int FAST>
struct ResE {
    static constexpr int NH = FS == 3 ? 9 : FS == 2 ? 3 : FS == 1 ? 2 : 4;   // H values read
    static constexpr int NC = FS == 3 ? 3 : FS == 2 ? 2 : 1;                 // E and D components
    static constexpr int NP = FS == 3 ? 2 : 1;
    T h[NH], d[NC];
    ResFace<T, NP> X, Y, Z;
    int c, g;

    __device__ __forceinline__ void load(const EParams<T, R>& p, int ix, int iy, int iz) {
        const int nx = p.L.nx, ny = p.L.ny, nz = p.L.nz, sy = p.L.px, sz = p.L.sz;
        c = ix + sy * iy + sz * iz;
        const bool xl = ix == 0, yl = iy == 0, zl = iz == 0;
        const int bx = p.bc[MFD_XL], by = p.bc[MFD_YL], bz = p.bc[MFD_ZL];
        const int ox = res_off(xl, bx, -1, nx - 1), oy = res_off(yl, by, -sy, (ny - 1) * sy),
                  oz = res_off(zl, bz, -sz, (nz - 1) * sz);
        if constexpr (FS == 3) {
            h[0] = MemShared::ld(p.Hx + c); h[1] = MemShared::ld(p.Hy + c); h[2] = MemShared::ld(p.Hz + c);
            h[3] = MemShared::ld(p.Hy + (c + ox)); h[4] = MemShared::ld(p.Hz + (c + ox));
            h[5] = MemShared::ld(p.Hx + (c + oy)); h[6] = MemShared::ld(p.Hz + (c + oy));
            h[7] = MemShared::ld(p.Hx + (c + oz)); h[8] = MemShared::ld(p.Hy + (c + oz));
            d[0] = p.Dx[c]; d[1] = p.Dy[c]; d[2] = p.Dz[c];
        } else if constexpr (FS == 2) {
            h[0] = MemShared::ld(p.Hy + c); h[1] = MemShared::ld(p.Hy + (c + ox)); h[2] = MemShared::ld(p.Hy + (c + oz));
            d[0] = p.Dx[c]; d[1] = p.Dz[c];
        } else if constexpr (FS == FSET_EY2) {
            h[0] = MemShared::ld(p.Hx + c); h[1] = MemShared::ld(p.Hz + c);
            h[2] = MemShared::ld(p.Hz + (c + ox)); h[3] = MemShared::ld(p.Hx + (c + oz));
            d[0] = p.Dy[c];
        } else {
            h[0] = MemShared::ld(p.Hy + c); h[1] = MemShared::ld(p.Hy + (c + oz));
            d[0] = p.Dx[c];
        }
        if constexpr (FS != 1) X.template load<0, 0, FS>(p, ix, iy, iz);
        if constexpr (FS == 3) Y.template load<1, 0, FS>(p, ix, iy, iz);
        Z.template load<2, 0, FS>(p, ix, iy, iz);
        g = MAT ? (int)p.geom[c] : 0;
        const bool zx = xl && bx == MFD_BC_DIRICHLET, zy = yl && by == MFD_BC_DIRICHLET, zz = zl && bz == MFD_BC_DIRICHLET;
        if constexpr (FS == 3) {
            if (zx) h[3] = h[4] = T(0);
            if (zy) h[5] = h[6] = T(0);
            if (zz) h[7] = h[8] = T(0);
        } else if constexpr (FS == 2) {
            if (zx) h[1] = T(0);
            if (zz) h[2] = T(0);
        } else if constexpr (FS == FSET_EY2) {
            if (zx) h[2] = T(0);
            if (zz) h[3] = T(0);
        } else {
            if (zz) h[1] = T(0);
        }
    }

    __device__ __forceinline__ void finish(const EParams<T, R>& p, const Div3& D3, bool k1, int ix, int iy, int iz, int cur, T dt) {
        T Md1 = p.Md10, Md2 = p.Md20, Me = p.Me0;
        const MatDev<T, R>* m = nullptr;
        bool simple = true;
        if (MAT && g) {
            m = p.mats + (g - 1);
            Md1 = m->Md1; Md2 = m->Md2; Me = m->Me; simple = m->simple != 0;
        }
        T Dv[NC];
        if constexpr (FS == 3) {
            const T hx = h[0], hy = h[1], hz = h[2];
            const T num[6] = {hx - h[5], hx - h[7], hy - h[3], hy - h[8], hz - h[4], hz - h[6]};
            T q[6];
            curl_div<T, FAST>(D3, p.ddx, p.ddy, p.ddz, num, q);
            T dHxy = q[0], dHxz = q[1], dHyx = q[2], dHyz = q[3], dHzx = q[4], dHzy = q[5];
            T D0 = d[0], D1 = d[1], D2 = d[2];
            if (X.in) {
                const T pa = X.template step<0, 0, true, FAST>(p, 0, dHyx), pb = X.template step<0, 0, true, FAST>(p, 1, dHzx);
                D1 = mad<FAST>(-Md2, pb, D1);
                D2 = mad<FAST>(Md2, pa, D2);
                dHyx = X.template over_k<0, FAST>(p, k1, dHyx);
                dHzx = X.template over_k<0, FAST>(p, k1, dHzx);
            }
            if (Y.in) {
                const T pa = Y.template step<1, 0, true, FAST>(p, 0, dHxy), pb = Y.template step<1, 0, true, FAST>(p, 1, dHzy);
                D0 = mad<FAST>(Md2, pb, D0);
                D2 = mad<FAST>(-Md2, pa, D2);
                dHxy = Y.template over_k<1, FAST>(p, k1, dHxy);
                dHzy = Y.template over_k<1, FAST>(p, k1, dHzy);
            }
            if (Z.in) {
                const T pa = Z.template step<2, 0, true, FAST>(p, 0, dHxz), pb = Z.template step<2, 0, true, FAST>(p, 1, dHyz);
                D0 = mad<FAST>(-Md2, pb, D0);
                D1 = mad<FAST>(Md2, pa, D1);
                dHxz = Z.template over_k<2, FAST>(p, k1, dHxz);
                dHyz = Z.template over_k<2, FAST>(p, k1, dHyz);
            }
            Dv[0] = mad<FAST>(Md1, D0, Md2 * (dHzy - dHyz));
            Dv[1] = mad<FAST>(Md1, D1, Md2 * (dHxz - dHzx));
            Dv[2] = mad<FAST>(Md1, D2, Md2 * (dHyx - dHxy));
        } else if constexpr (FS == 2) {
            const T hy = h[0];
            T dHyx = cdiv<FAST>(hy - h[1], p.ddx);
            T dHyz = cdiv<FAST>(hy - h[2], p.ddz);
            T D0 = d[0], D2 = d[1];
            if (X.in) {
                D2 = mad<FAST>(Md2, X.template step<0, 0, false, FAST>(p, 0, dHyx), D2);
                dHyx = X.template over_k<0, FAST>(p, k1, dHyx);
            }
            if (Z.in) {
                D0 = mad<FAST>(-Md2, Z.template step<2, 0, false, FAST>(p, 0, dHyz), D0);
                dHyz = Z.template over_k<2, FAST>(p, k1, dHyz);
            }
            Dv[0] = Md1 * D0 + Md2 * (T(0) - dHyz);
            Dv[1] = Md1 * D2 + Md2 * (dHyx - T(0));
        } else if constexpr (FS == FSET_EY2) {
            T dHxz = cdiv<FAST>(h[0] - h[3], p.ddz);
            T dHzx = cdiv<FAST>(h[1] - h[2], p.ddx);
            T D1 = d[0];
            if (X.in) {
                D1 = mad<FAST>(-Md2, X.template step<0, 0, false, FAST>(p, 0, dHzx), D1);
                dHzx = X.template over_k<0, FAST>(p, k1, dHzx);
            }
            if (Z.in) {
                D1 = mad<FAST>(Md2, Z.template step<2, 0, false, FAST>(p, 0, dHxz), D1);
                dHxz = Z.template over_k<2, FAST>(p, k1, dHxz);
            }
            Dv[0] = Md1 * D1 + Md2 * (dHxz - dHzx);
        } else {
            T dHyz = cdiv<FAST>(h[0] - h[1], p.ddz);
            T D0 = d[0];
            if (Z.in) {
                D0 = mad<FAST>(-Md2, Z.template step<2, 0, false, FAST>(p, 0, dHyz), D0);
                dHyz = Z.template over_k<2, FAST>(p, k1, dHyz);
            }
            Dv[0] = Md1 * D0 + Md2 * (T(0) - dHyz);
        }
        T* Dp[NC];
        T* Ep[NC];
        if constexpr (FS == 3) {
            Dp[0] = p.Dx; Dp[1] = p.Dy; Dp[2] = p.Dz;
            Ep[0] = p.Ex; Ep[1] = p.Ey; Ep[2] = p.Ez;
        } else if constexpr (FS == 2) {
            Dp[0] = p.Dx; Dp[1] = p.Dz;
            Ep[0] = p.Ex; Ep[1] = p.Ez;
        } else {
            Dp[0] = FS == 1 ? p.Dx : p.Dy;
            Ep[0] = FS == 1 ? p.Ex : p.Ey;
        }
        if (MAT && !simple) {   // dispersive and Kerr cells: E from the cell's new D (material_flat_kernel)
            const long long bi = (long long)(ix - m->bx0) +
                                 (long long)m->bnx * ((long long)(iy - m->by0) + (long long)m->bny * (iz - m->bz0));
            switch (m->nq) {    // no plasma, at most three poles (the engine's rule)
                case 0: material_cell_n<T, R, NC, 0, false>(m, bi, Ep, c, Dv, cur, dt); break;
                case 1: material_cell_n<T, R, NC, 1, false>(m, bi, Ep, c, Dv, cur, dt); break;
                case 2: material_cell_n<T, R, NC, 2, false>(m, bi, Ep, c, Dv, cur, dt); break;
                default: material_cell_n<T, R, NC, 3, false>(m, bi, Ep, c, Dv, cur, dt); break;
            }
        } else {
#pragma unroll
            for (int k = 0; k < NC; ++k) Ep[k][c] = Dv[k] * Me;
        }
#pragma unroll
        for (int k = 0; k < NC; ++k) Dp[k][c] = Dv[k];
    }
};

// A source's points a .. b - 1 of this block at step it0 (0-based), as the kernel below applies them;
// pts: those points in shared memory, or null.  pre: w0 is the waveform value of the thread's first.
template <typename T>
__device__ __forceinline__ void res_source(const ResOp<T>& op, const RectParams<T>& rp, const ResPoint* pts, int a, int b, long long it0,
                                           bool pre, double w0) {
    for (int i = a + (int)threadIdx.x; i < b; i += blockDim.x) {
        if (op.tfsf) {
            if (pts) tfsf_point(rp, pts[i - a].m, pts[i - a].j, it0);
            else tfsf_point(rp, op.list[2 * i], op.list[2 * i + 1], it0);
            continue;
        }
        const int j = pts ? pts[i - a].j : op.list[i];
        const long long c = pts ? pts[i - a].c : op.cells[j];
        double w = pre && pts && i == a + (int)threadIdx.x ? w0 : op.wave ? op.wave[it0 * op.npts + j] : op.gt[it0];
        if (!op.wave) w = (pts ? pts[i - a].amp : op.amp[j]) * w;
        if (op.kind == MFD_SRC_SOFT) op.F[c] = (T)((double)op.F[c] + (double)op.coeff * w);
        else op.F[c] = (T)w;
    }
}

// The block's monitor points a .. b - 1; pts as above.
template <typename T>
__device__ __forceinline__ void res_monitors(const MonParams<T>& mp, const int* list, const ResPoint* pts, int a, int b, long long it0, int slot) {
    for (int i = a + (int)threadIdx.x; i < b; i += blockDim.x) {
        if (pts) monitor_store(mp, mp.mons[pts[i - a].m], pts[i - a].j, pts[i - a].c, it0, slot);
        else monitor_point(mp, list[2 * i], list[2 * i + 1], it0, slot);
    }
}

// FS: 1, 2, 3 (the model's dimension) or FSET_EY2.  MAT: the model has a material map.
// HPTS: some source writes H.  Models without such take the step's plain order, in code of its own:
// sharing the two-part form with them cost 0.8 % of a step of 2001 cells (double, 3.68 -> 3.71 us) and
// 3.6 % of one of 701 x 513 (double, second field set, 15.7 -> 16.3 us), whatever the loop's form.
template <typename T, typename R, int FS, bool MAT, int FAST, bool HPTS>
__global__ void __launch_bounds__(RES_THREADS<T>, 1)
    resident_kernel(const __grid_constant__ HParams<T> hp0, const __grid_constant__ EParams<T, R> ep0, const Div3 D3,
                    const __grid_constant__ ResidentParams<T> r, const long long it_first, const int nsteps, const int accum,
                    const int slot0) {
    extern __shared__ __align__(16) char sm[];
    __shared__ int s_ok;
    constexpr int MON_ROW = HPTS ? RES_MAXOPS + 1 : RES_MAXOPS;
    __shared__ int s_op[MON_ROW + 1][2];   // this block's entries of each source; the last row: its monitor points
    const int tid = threadIdx.x, nth = blockDim.x;
    const int nx = hp0.L.nx, ny = hp0.L.ny, px = hp0.L.px, sz = hp0.L.sz;
    const int lo = blockIdx.x * r.per, hi = min(lo + r.per, r.ncell);
    auto decode = [&](int l, int& ix, int& iy, int& iz) {
        ix = iy = 0;
        iz = l;
        if constexpr (FS != 1) {
            iz = l / nx;
            ix = l - iz * nx;
        }
        if constexpr (FS == 3) {
            const int row = iz;
            iz = row / ny;
            iy = row - iz * ny;
        }
    };
    // ---- tables to shared memory, pointers to them -------------------------------------
    HParams<T> hp = hp0;
    EParams<T, R> ep = ep0;
    if constexpr (MAT) {
        if (r.o_geom >= 0) {
            int x, y, z;
            decode(lo, x, y, z);
            const int c0 = x + px * y + sz * z;
            decode(hi - 1, x, y, z);
            res_copy(sm + r.o_geom, hp0.geom + c0, x + px * y + sz * z - c0 + 1);
            hp.geom = ep.geom = (const uint8_t*)(sm + r.o_geom) - c0;
        }
        if (r.o_mats >= 0) {
            res_copy(sm + r.o_mats, ep0.mats, r.nmat * (int)sizeof(MatDev<T, R>));
            ep.mats = (const MatDev<T, R>*)(sm + r.o_mats);
            res_copy(sm + r.o_math, hp0.matMh, r.nmat * (int)sizeof(T));
            hp.matMh = (const T*)(sm + r.o_math);
        }
    }
#pragma unroll
    for (int f = 0; f < 6; ++f) {
        if (r.o_lay[f] < 0) continue;
        const int nb = hp0.lay[f].nb;
        DivC<T>* K = (DivC<T>*)(sm + r.o_lay[f]);
        T* A = (T*)(K + nb);
        T* B = A + nb;
        res_copy(K, hp0.lay[f].K, nb * (int)sizeof(DivC<T>));
        res_copy(A, hp0.lay[f].A, nb * (int)sizeof(T));
        res_copy(B, hp0.lay[f].B, nb * (int)sizeof(T));
        hp.lay[f].K = ep.lay[f].K = K;
        hp.lay[f].A = ep.lay[f].A = A;
        hp.lay[f].B = ep.lay[f].B = B;
    }
    const RectParams<T>* rp = r.rp;
    if (r.o_rect >= 0) {
        res_copy(sm + r.o_rect, r.rp, (int)sizeof(RectParams<T>));
        rp = (const RectParams<T>*)(sm + r.o_rect);
    }
    MonParams<T> mp = r.mp;
    if (r.o_mon >= 0) {
        res_copy(sm + r.o_mon, r.mp.mons, r.nmon * (int)sizeof(MonDev<T>));
        mp.mons = (const MonDev<T>*)(sm + r.o_mon);
    }
    const ResOp<T>* ops = r.ops;
    if (r.o_ops >= 0) {
        res_copy(sm + r.o_ops, r.ops, r.nops * (int)sizeof(ResOp<T>));
        ops = (const ResOp<T>*)(sm + r.o_ops);
    }
    if (tid == 0) {
        s_ok = 1;
        s_op[MON_ROW][0] = r.nmon ? r.moff[blockIdx.x] : 0;
        s_op[MON_ROW][1] = r.nmon ? r.moff[blockIdx.x + 1] : 0;
    }
    if (tid < r.nops) {
        s_op[tid][0] = r.ops[tid].off[blockIdx.x];
        s_op[tid][1] = r.ops[tid].off[blockIdx.x + 1];
    }
    if (HPTS && tid == 0 && r.nops > RES_MAXOPS) {   // a block has at least 32 threads
        s_op[RES_MAXOPS][0] = r.ops[RES_MAXOPS].off[blockIdx.x];
        s_op[RES_MAXOPS][1] = r.ops[RES_MAXOPS].off[blockIdx.x + 1];
    }
    __syncthreads();
    // The block's points, source by source and then the monitors', as far as they fit: point k of
    // the block is pts[k].
    ResPoint* pts = (ResPoint*)(sm + r.o_pts);
    {
        int k0 = 0;
        for (int o = 0; o <= r.nops; ++o) {
            const bool mon = o == r.nops;
            const int a = s_op[mon ? MON_ROW : o][0], b = s_op[mon ? MON_ROW : o][1];
            for (int i = a + tid; i < b && k0 + i - a < r.npts_cap; i += nth) {
                ResPoint q{0, 0, 0, 0, 0.0};
                if (mon) {
                    q.m = r.mlist[2 * i];
                    q.j = r.mlist[2 * i + 1];
                    q.c = r.mp.mons[q.m].cells[q.j];
                } else if (r.ops[o].tfsf) {
                    q.m = r.ops[o].list[2 * i];
                    q.j = r.ops[o].list[2 * i + 1];
                } else {
                    q.j = r.ops[o].list[i];
                    q.c = (int)r.ops[o].cells[q.j];
                    q.amp = r.ops[o].wave ? 0.0 : r.ops[o].amp[q.j];
                }
                pts[k0 + i - a] = q;
            }
            k0 += b - a;
        }
    }
    __syncthreads();
    const bool fit = [&] {   // every point of the block is in pts
        int n = 0;
        for (int o = 0; o < r.nops; ++o) n += s_op[o][1] - s_op[o][0];
        return n + s_op[MON_ROW][1] - s_op[MON_ROW][0] <= r.npts_cap;
    }();
    bool tail = false;   // the block has points that write H
    if constexpr (HPTS)
        for (int o = r.nops_e; o < r.nops; ++o) tail = tail || s_op[o][1] > s_op[o][0];
    int x1, y1, z1;   // the thread's first cell
    decode(min(lo + tid, hi - 1), x1, y1, z1);
    unsigned bar = 0;
    for (int s = 0; s < nsteps; ++s) {
        const long long it = it_first + s;
        const bool acc = s > 0 || accum;
        // the waveform values of this step for the thread's first point of the first sources
        double wpre[RES_PRE];
        if (fit) {
            int k0 = 0;
#pragma unroll
            for (int o = 0; o < RES_PRE; ++o) {
                wpre[o] = 0.0;
                if (o >= r.nops) continue;
                const int n = s_op[o][1] - s_op[o][0];
                if (tid < n && !ops[o].tfsf)
                    wpre[o] = ops[o].wave ? ops[o].wave[(it - 1) * ops[o].npts + pts[k0 + tid].j] : ops[o].gt[it - 1];
                k0 += n;
            }
        }
        for (int l = lo + tid; l < hi; l += nth) {
            int ix = x1, iy = y1, iz = z1;
            if (l != lo + tid) decode(l, ix, iy, iz);
            ResH<T, FS, MAT, FAST> v;
            v.load(hp, acc, ix, iy, iz);
            v.finish(hp, D3, r.k1, acc, it - 1);
        }
        if (!res_barrier(r.bar, ++bar, r.fault, &s_ok, r.cluster)) return;
        const int cur = (int)((it - 1) & 1);
        for (int l = lo + tid; l < hi; l += nth) {
            int ix = x1, iy = y1, iz = z1;
            if (l != lo + tid) decode(l, ix, iy, iz);
            ResE<T, R, FS, MAT, FAST> v;
            v.load(ep, ix, iy, iz);
            v.finish(ep, D3, r.k1, ix, iy, iz, cur, r.dt);
        }
        if constexpr (HPTS) {
            int o = 0, k0 = 0;
#pragma unroll 1
            for (bool late = false;; late = true) {   // late: after the second barrier
                for (const int end = late ? r.nops : r.nops_e; o < end; ++o) {
                    const int a = s_op[o][0], b = s_op[o][1];
                    if (a == b) continue;   // the same for the whole block
                    __syncthreads();
                    res_source(ops[o], *rp, fit ? pts + k0 : nullptr, a, b, it - 1, o < RES_PRE, o == 0 ? wpre[0] : o == 1 ? wpre[1] : wpre[2]);
                    k0 += b - a;
                }
                const int ma = s_op[MON_ROW][0], mb = s_op[MON_ROW][1];
                if (mb > ma && late == tail) {
                    __syncthreads();
                    res_monitors(mp, r.mlist, fit ? pts + k0 : nullptr, ma, mb, it - 1, slot0 + s);
                }
                if (late) {
                    __syncthreads();   // the next H update changes what these points wrote and read
                    break;
                }
                if (!res_barrier(r.bar, ++bar, r.fault, &s_ok, r.cluster)) return;
                if (!tail) break;
            }
            continue;
        }
        // the block's own source points, source by source, then its monitor points
        int k0 = 0;
        for (int o = 0; o < r.nops; ++o) {
            const int a = s_op[o][0], b = s_op[o][1];
            if (a == b) continue;   // the same for the whole block
            __syncthreads();
            const ResOp<T>& op = ops[o];
            for (int i = a + tid; i < b; i += nth) {
                if (op.tfsf) {
                    if (fit) tfsf_point(*rp, pts[k0 + i - a].m, pts[k0 + i - a].j, it - 1);
                    else tfsf_point(*rp, op.list[2 * i], op.list[2 * i + 1], it - 1);
                    continue;
                }
                double w;
                long long c;
                if (fit) {
                    const ResPoint q = pts[k0 + i - a];
                    c = q.c;
                    double v;
                    if (i == a + tid && o < RES_PRE) v = o == 0 ? wpre[0] : o == 1 ? wpre[1] : wpre[2];
                    else v = op.wave ? op.wave[(it - 1) * op.npts + q.j] : op.gt[it - 1];
                    w = op.wave ? v : q.amp * v;
                } else {
                    const int j = op.list[i];
                    w = op.wave ? op.wave[(it - 1) * op.npts + j] : op.amp[j] * op.gt[it - 1];
                    c = op.cells[j];
                }
                if (op.kind == MFD_SRC_SOFT) op.F[c] = (T)((double)op.F[c] + (double)op.coeff * w);
                else op.F[c] = (T)w;
            }
            k0 += b - a;
        }
        const int ma = s_op[MON_ROW][0], mb = s_op[MON_ROW][1];
        if (mb > ma) {
            __syncthreads();
            for (int i = ma + tid; i < mb; i += nth) {
                if (fit) {
                    const ResPoint q = pts[k0 + i - ma];
                    monitor_store(mp, mp.mons[q.m], q.j, q.c, it - 1, slot0 + s);
                }
                else monitor_point(mp, r.mlist[2 * i], r.mlist[2 * i + 1], it - 1, slot0 + s);
            }
        }
        if (!res_barrier(r.bar, ++bar, r.fault, &s_ok, r.cluster)) return;
    }
}

}  // namespace mfd
