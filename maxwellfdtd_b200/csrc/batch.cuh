// batch.cuh -- many independent 2-D and 3-D models stepped together (sm_100a).
//
// Each half-step of every member of a batch is one persistent launch: the grid is sized to
// the GPU (SMs x resident blocks) and each block walks a table of tiles (member, tile
// origin), so hundreds of small, unevenly sized models cost a handful of launches per step
// instead of a handful per model.  Every per-member quantity that changes from step to step
// (the step index, the running-sum flag, the polarisation ping-pong parity) lives in the
// member's device state and is advanced on the device, so a CUDA graph of several steps can
// be replayed unchanged.  The per-cell arithmetic is the single-model code (h2d_cell /
// e2d_cell, the 3-D h3d_cell / e3d_cell of the CPML slabs, material_cell, the point-source
// expression), so a member's results are bit-identical to running it alone.  2-D and 3-D
// members have their own tile tables and kernels (the 3-D cell code needs more registers);
// a 3-D tile is a run of groups of B3D_W cells.  A block copies its tile's
// member parameter block into shared memory whenever the member changes, so the cells read
// the layout, pointers and coefficients from there rather than through dependent global loads.
#pragma once

#include "aux.cuh"
#include "yee.cuh"
#include "yee2d_quad.cuh"
#include "yee3d_group.cuh"
#include "yee3d_split.cuh"

namespace mfd {

enum { BF_MATH = 1, BF_MAT = 2, BF_FAST = 4, BF_3D = 8, BF_RECIP = 16, BF_K1 = 32, BF_RESP = 64 };

// The half-step kernels come in two sets: DSET 0 runs the members of the exact arithmetic
// (IEEE or the verified constant division), DSET 1 those of the tolerance mode (reciprocal
// multiplies), each launched only when the batch holds such members.  One kernel for both
// measured slower: the extra cell code raised the 2-D E kernel from 32 to 40 registers.
template <int DSET>
__device__ __forceinline__ bool b_other_set(int flags) { return ((flags & BF_RECIP) != 0) != (DSET == 1); }

// Per-member state (device).  Steps are 1-based; the member runs steps first..last.
struct BMember {
    const HParams<float>* hp;              // the member's update parameters (static fields)
    const EParams<float, double>* ep;
    const MonParams<float>* mp;            // monitors (gathered every step)
    const RectParams<float>* rp;           // TFSF statements (null: none)
    long long it;                          // step being run; > last once the member is done
    long long first, last;
    long long ring_first;                  // 0-based step staged in ring slot 0
    int flags;                             // BF_*
    int pad;
    Div3 d3;                               // grid-spacing divisors of a 3-D member (div6)
};

// 2-D: cells x0 .. x0 + 4 blockDim.x - 1 (four per thread) of rows z0 .. z0 + blockDim.y - 1 of
// member m.
struct BTile {
    int m, x0, z0, w;  // 3-D linear tiles: (x0, z0, w) = (group of the row, y, z) of the tile's first group
};

struct BMatTile {   // one row segment of material g's bounding box: x0 .. x0+blockDim.x-1 at (iy, iz)
    int m, g, x0, iy, iz;
};

struct BSrc {       // one point source of a member (sources.jl:122-131, 235-244)
    float* F;
    const long long* cells;
    const double* wave;
    const double* amp;
    const double* gt;
    long long npts;
    int kind;
    float coeff;
};

struct BPoint {     // point i of source s (entries of one source pass) or of monitor s
    int m, s;
    long long i;
};

struct BRow {       // TFSF statement s of member m (grid rows of one TFSF pass)
    int m, s;
};

__device__ __forceinline__ bool b_active(const BMember& M) { return M.it <= M.last; }

// Copies the member's parameter block (8-byte words) into shared memory; every thread of the
// block takes part (call it where the whole block is).
template <typename P>
__device__ __forceinline__ void b_stage(P* dst, const P* src) {
    static_assert(sizeof(P) % 8 == 0, "parameter blocks are whole 8-byte words");
    const int tid = threadIdx.x + blockDim.x * threadIdx.y, nth = blockDim.x * blockDim.y;
    const long long* s = reinterpret_cast<const long long*>(src);
    long long* d = reinterpret_cast<long long*>(dst);
    for (int i = tid; i < (int)(sizeof(P) / 8); i += nth) d[i] = s[i];
}


// Entry of a block's k-th turn (runs of CHUNK consecutive tiles, dealt out to the blocks in turn);
// m = -1 past the end.
template <int CHUNK>
__device__ __forceinline__ BTile b_tile(const BTile* __restrict__ tiles, int k, int n) {
    const int t = ((k / CHUNK) * (int)gridDim.x + (int)blockIdx.x) * CHUNK + k % CHUNK;
    if (t < n) return tiles[t];
    return BTile{-1, 0, 0, 0};
}

#define MFD_B2D_CHUNK 4  // a block takes runs of this many consecutive tiles (fewer member changes)
#define MFD_B2D_MINB 2   // batched 2-D updates: 2 blocks of 512 threads per SM (64 registers for four cells a thread)


template <int DSET>
__global__ void __launch_bounds__(512, MFD_B2D_MINB) batch_h2d_kernel(const BMember* __restrict__ mem, const BTile* __restrict__ tiles,
                                                        const int* __restrict__ ntiles) {
    __shared__ __align__(16) HParams<float> sp;
    const int n = *ntiles;
    int cur = -1, acc = 0, flags = 0;
    bool skip = false;
    long long prev = 0;
    // Tile t of the block's k-th turn: runs of MFD_B2D_CHUNK tiles, the runs dealt out to the
    // blocks in turn, so t grows with k.  The next turn's entry is fetched while this one runs,
    // and the member's step and flags are read when the member changes.
    BTile nxt = b_tile<MFD_B2D_CHUNK>(tiles, 0, n);
    for (int k = 0; nxt.m >= 0; ++k) {
        const BTile tl = nxt;
        nxt = b_tile<MFD_B2D_CHUNK>(tiles, k + 1, n);
        if (tl.m != cur) {   // the block copies the member's parameters to shared memory (42.1 vs 40.8 Gcell/s)
            const BMember& M = mem[tl.m];
            cur = tl.m;
            flags = M.flags;
            skip = !b_active(M) || b_other_set<DSET>(flags);   // the same for the whole block
            acc = M.it > M.first ? 1 : 0;
            prev = M.it - 1;
            __syncthreads();          // the previous member's parameters are no longer read
            if (!skip) b_stage(&sp, M.hp);
            __syncthreads();
        }
        if (skip) continue;
        const HParams<float>& p = sp;
        const int x0 = tl.x0 + 4 * (int)threadIdx.x, iz = tl.z0 + threadIdx.y;
        if (x0 >= p.L.nx || iz >= p.L.nz) continue;
        const bool k1 = flags & BF_K1;
        if constexpr (DSET == 1) {
            if (flags & BF_MATH) h2d_quad<true, DIV_RECIP>(p, k1, acc, prev, x0, iz);
            else h2d_quad<false, DIV_RECIP>(p, k1, acc, prev, x0, iz);
        } else if (flags & BF_FAST) {
            if (flags & BF_MATH) h2d_quad<true, DIV_EXACT>(p, k1, acc, prev, x0, iz);
            else h2d_quad<false, DIV_EXACT>(p, k1, acc, prev, x0, iz);
        } else {   // a divisor that needs IEEE division: cell by cell
            for (int ix = x0; ix < min(x0 + 4, p.L.nx); ++ix) {
                if (flags & BF_MATH) h2d_cell<float, true, DIV_IEEE>(p, acc, prev, ix, iz);
                else h2d_cell<float, false, DIV_IEEE>(p, acc, prev, ix, iz);
            }
        }
    }
}

template <int DSET>
__global__ void __launch_bounds__(512, MFD_B2D_MINB) batch_e2d_kernel(const BMember* __restrict__ mem, const BTile* __restrict__ tiles,
                                                        const int* __restrict__ ntiles) {
    __shared__ __align__(16) EParams<float, double> sp;
    const int n = *ntiles;
    int cur = -1, flags = 0, cur_p = 0;   // cur_p: ping-pong parity of the polarisation
    bool skip = false;
    BTile nxt = b_tile<MFD_B2D_CHUNK>(tiles, 0, n);   // as in the H kernel
    for (int k = 0; nxt.m >= 0; ++k) {
        const BTile tl = nxt;
        nxt = b_tile<MFD_B2D_CHUNK>(tiles, k + 1, n);
        if (tl.m != cur) {
            const BMember& M = mem[tl.m];
            cur = tl.m;
            flags = M.flags;
            skip = !b_active(M) || b_other_set<DSET>(flags);   // the same for the whole block
            cur_p = (int)((M.it - 1) & 1);
            __syncthreads();
            if (!skip) b_stage(&sp, M.ep);
            __syncthreads();
        }
        if (skip) continue;
        const EParams<float, double>& p = sp;
        const int x0 = tl.x0 + 4 * (int)threadIdx.x, iz = tl.z0 + threadIdx.y;
        const bool act = x0 < p.L.nx && iz < p.L.nz;
        const bool k1 = flags & BF_K1;
        if constexpr (DSET == 1) {
            if (flags & BF_RESP) e2d_warp<double, true, DIV_RECIP, true>(p, k1, cur_p, act, x0, iz);
            else if (flags & BF_MAT) e2d_warp<double, true, DIV_RECIP, false>(p, k1, cur_p, act, x0, iz);
            else e2d_warp<double, false, DIV_RECIP, false>(p, k1, cur_p, act, x0, iz);
        } else if (flags & BF_FAST) {
            if (flags & BF_RESP) e2d_warp<double, true, DIV_EXACT, true>(p, k1, cur_p, act, x0, iz);
            else if (flags & BF_MAT) e2d_warp<double, true, DIV_EXACT, false>(p, k1, cur_p, act, x0, iz);
            else e2d_warp<double, false, DIV_EXACT, false>(p, k1, cur_p, act, x0, iz);
        } else if (act) {   // a divisor that needs IEEE division: cell by cell
            for (int ix = x0; ix < min(x0 + 4, p.L.nx); ++ix) {
                if (flags & BF_MAT) e2d_cell<float, double, true, DIV_IEEE>(p, ix, iz);
                else e2d_cell<float, double, false, DIV_IEEE>(p, ix, iz);
            }
        }
    }
}

// ADE / Kerr / plasma response of material g's cells (material_kernel for 2-D members).
__global__ void __launch_bounds__(128) batch_material2d_kernel(const BMember* __restrict__ mem,
                                                               const BMatTile* __restrict__ tiles,
                                                               const int* __restrict__ ntiles) {
    const int n = *ntiles;
    for (int t = blockIdx.x; t < n; t += gridDim.x) {
        const BMatTile tl = tiles[t];
        const BMember& M = mem[tl.m];
        if (!b_active(M)) continue;
        const EParams<float, double>& p = *M.ep;
        const MatDev<float, double>* m = p.mats + (tl.g - 1);
        const int ix = tl.x0 + threadIdx.x;
        if (ix >= m->bx0 + m->bnx) continue;
        const int c = ix + p.L.sz * tl.iz;
        if (p.geom[c] != tl.g) continue;
        float Dv[2] = {p.Dx[c], p.Dz[c]};
        float* Ep[2] = {p.Ex, p.Ez};
        const int cur = (int)((M.it - 1) & 1);
        const long long bi = (long long)(ix - m->bx0) + (long long)m->bnx * (tl.iz - m->bz0);
        switch (m->nq) {
            case 0: material_cell_n<float, double, 2, 0>(m, bi, Ep, c, Dv, cur, p.dt); break;
            case 1: material_cell_n<float, double, 2, 1>(m, bi, Ep, c, Dv, cur, p.dt); break;
            case 2: material_cell_n<float, double, 2, 2>(m, bi, Ep, c, Dv, cur, p.dt); break;
            case 3: material_cell_n<float, double, 2, 3>(m, bi, Ep, c, Dv, cur, p.dt); break;
            default: material_cell<float, double, 2>(m, ix, 0, tl.iz, Ep, c, Dv, cur, p.dt); break;
        }
    }
}

// Cells of a 3-D thread's group: two, which fit 64 registers.  32 models of 48-128 cells a side,
// tolerance mode: one cell 909 us per step, two 734, four (96-124 registers, a quarter of the
// warps) 856.
constexpr int B3D_W = 2;

// The group of a 3-D tile's thread.  A 3-D tile is a run of groups in x-fastest order (no idle
// lanes at rows shorter than the block): the block's threads take the blockDim.x * blockDim.y
// groups from the tile's first, (x0, z0, w) = (group of the row, y, z).
__device__ __forceinline__ bool b_group3(const Layout& L, const BTile& tl, int& x0, int& iy, int& iz) {
    // offset / row length row steps, a few at the tile shapes used: cheaper than two divisions
    const int ng = (L.nx + B3D_W - 1) / B3D_W;
    x0 = tl.x0 + (int)(threadIdx.y * blockDim.x + threadIdx.x);
    iy = tl.z0;
    iz = tl.w;
    while (x0 >= ng) {
        x0 -= ng;
        if (++iy == L.ny) {
            iy = 0;
            ++iz;
        }
    }
    x0 *= B3D_W;
    return iz < L.nz;
}

// A block takes runs of this many consecutive tiles (fewer member changes).  Runs of 2: 734 us; of 1
// 764, 4 759-777, 8 808, 16 888.
#define MFD_B3D_CHUNK 2

template <int DSET>
__global__ void __launch_bounds__(512, 2) batch_h3d_kernel(const BMember* __restrict__ mem, const BTile* __restrict__ tiles,
                                                           const int* __restrict__ ntiles) {
    __shared__ __align__(16) HParams<float> sp;
    __shared__ Div3 sd3;
    const int n = *ntiles;
    int cur = -1, flags = 0;
    bool skip = false, acc = false;
    long long prev = 0;
    BTile nxt = b_tile<MFD_B3D_CHUNK>(tiles, 0, n);   // as in the 2-D kernels
    for (int k = 0; nxt.m >= 0; ++k) {
        const BTile tl = nxt;
        nxt = b_tile<MFD_B3D_CHUNK>(tiles, k + 1, n);
        if (tl.m != cur) {   // the block copies the member's parameters to shared memory
            const BMember& M = mem[tl.m];
            cur = tl.m;
            flags = M.flags;
            skip = !b_active(M) || b_other_set<DSET>(flags);   // the same for the whole block
            acc = M.it > M.first;    // the running sums of the previous step, from a member's second step on
            prev = M.it - 1;
            __syncthreads();          // the previous member's parameters are no longer read
            if (!skip) {
                b_stage(&sp, M.hp);
                if (threadIdx.x == 0 && threadIdx.y == 0) sd3 = M.d3;
            }
            __syncthreads();
        }
        if (skip) continue;
        const HParams<float>& p = sp;
        int x0, iy, iz;
        if (!b_group3(p.L, tl, x0, iy, iz)) continue;
        const bool k1 = flags & BF_K1;
        if constexpr (DSET == 1) {
            if (flags & BF_MATH) h3d_group<true, DIV_RECIP, B3D_W>(p, sd3, k1, acc, prev, x0, iy, iz);
            else h3d_group<false, DIV_RECIP, B3D_W>(p, sd3, k1, acc, prev, x0, iy, iz);
        } else if (flags & BF_FAST) {
            if (flags & BF_MATH) h3d_group<true, DIV_EXACT, B3D_W>(p, sd3, k1, acc, prev, x0, iy, iz);
            else h3d_group<false, DIV_EXACT, B3D_W>(p, sd3, k1, acc, prev, x0, iy, iz);
        } else {   // a divisor that needs IEEE division
            if (flags & BF_MATH) h3d_group<true, DIV_IEEE, B3D_W>(p, sd3, k1, acc, prev, x0, iy, iz);
            else h3d_group<false, DIV_IEEE, B3D_W>(p, sd3, k1, acc, prev, x0, iy, iz);
        }
    }
}

template <int DSET>
__global__ void __launch_bounds__(512, 2) batch_e3d_kernel(const BMember* __restrict__ mem, const BTile* __restrict__ tiles,
                                                           const int* __restrict__ ntiles) {
    __shared__ __align__(16) EParams<float, double> sp;
    __shared__ Div3 sd3;
    const int n = *ntiles;
    int cur = -1, flags = 0;
    bool skip = false;
    BTile nxt = b_tile<MFD_B3D_CHUNK>(tiles, 0, n);   // as in the 2-D kernels
    for (int k = 0; nxt.m >= 0; ++k) {
        const BTile tl = nxt;
        nxt = b_tile<MFD_B3D_CHUNK>(tiles, k + 1, n);
        if (tl.m != cur) {   // the block copies the member's parameters to shared memory
            const BMember& M = mem[tl.m];
            cur = tl.m;
            flags = M.flags;
            skip = !b_active(M) || b_other_set<DSET>(flags);   // the same for the whole block
            __syncthreads();
            if (!skip) {
                b_stage(&sp, M.ep);
                if (threadIdx.x == 0 && threadIdx.y == 0) sd3 = M.d3;
            }
            __syncthreads();
        }
        if (skip) continue;
        const EParams<float, double>& p = sp;
        int x0, iy, iz;
        if (!b_group3(p.L, tl, x0, iy, iz)) continue;
        const bool k1 = flags & BF_K1;
        if constexpr (DSET == 1) {
            if (flags & BF_MAT) e3d_group<double, true, DIV_RECIP, B3D_W>(p, sd3, k1, x0, iy, iz);
            else e3d_group<double, false, DIV_RECIP, B3D_W>(p, sd3, k1, x0, iy, iz);
        } else if (flags & BF_FAST) {
            if (flags & BF_MAT) e3d_group<double, true, DIV_EXACT, B3D_W>(p, sd3, k1, x0, iy, iz);
            else e3d_group<double, false, DIV_EXACT, B3D_W>(p, sd3, k1, x0, iy, iz);
        } else {   // a divisor that needs IEEE division
            if (flags & BF_MAT) e3d_group<double, true, DIV_IEEE, B3D_W>(p, sd3, k1, x0, iy, iz);
            else e3d_group<double, false, DIV_IEEE, B3D_W>(p, sd3, k1, x0, iy, iz);
        }
    }
}

// ADE / Kerr / plasma response of material g's cells of 3-D members.
__global__ void __launch_bounds__(128) batch_material3d_kernel(const BMember* __restrict__ mem,
                                                               const BMatTile* __restrict__ tiles,
                                                               const int* __restrict__ ntiles) {
    const int n = *ntiles;
    for (int t = blockIdx.x; t < n; t += gridDim.x) {
        const BMatTile tl = tiles[t];
        const BMember& M = mem[tl.m];
        if (!b_active(M)) continue;
        const EParams<float, double>& p = *M.ep;
        const MatDev<float, double>* m = p.mats + (tl.g - 1);
        const int ix = tl.x0 + threadIdx.x;
        if (ix >= m->bx0 + m->bnx) continue;
        const int c = ix + p.L.px * tl.iy + p.L.sz * tl.iz;
        if (p.geom[c] != tl.g) continue;
        float Dv[3] = {p.Dx[c], p.Dy[c], p.Dz[c]};
        float* Ep[3] = {p.Ex, p.Ey, p.Ez};
        const int cur = (int)((M.it - 1) & 1);
        const long long bi = (long long)(ix - m->bx0) + (long long)m->bnx * ((tl.iy - m->by0) + (long long)m->bny * (tl.iz - m->bz0));
        switch (m->nq) {
            case 0: material_cell_n<float, double, 3, 0>(m, bi, Ep, c, Dv, cur, p.dt); break;
            case 1: material_cell_n<float, double, 3, 1>(m, bi, Ep, c, Dv, cur, p.dt); break;
            case 2: material_cell_n<float, double, 3, 2>(m, bi, Ep, c, Dv, cur, p.dt); break;
            case 3: material_cell_n<float, double, 3, 3>(m, bi, Ep, c, Dv, cur, p.dt); break;
            default: material_cell<float, double, 3>(m, ix, tl.iy, tl.iz, Ep, c, Dv, cur, p.dt); break;
        }
    }
}

// One pass of point sources: entry i is a point of the k-th source of its member, so a
// member's sources act in tuple order across passes (models.jl:128-130).
__global__ void __launch_bounds__(256) batch_source_kernel(const BMember* __restrict__ mem, const BSrc* __restrict__ srcs,
                                                           const BPoint* __restrict__ pts, const int* __restrict__ npts) {
    const int n = *npts;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const BPoint e = pts[i];
        const BMember& M = mem[e.m];
        if (!b_active(M)) continue;
        const BSrc& S = srcs[e.s];
        const long long it0 = M.it - 1;
        const double w = S.wave ? S.wave[it0 * S.npts + e.i] : S.amp[e.i] * S.gt[it0];
        const long long c = S.cells[e.i];
        if (S.kind == MFD_SRC_SOFT) S.F[c] = (float)((double)S.F[c] + (double)S.coeff * w);
        else S.F[c] = (float)w;
    }
}

// TFSF injection of the members whose TFSF acts in this source pass: grid row = (member,
// statement), as tfsf_kernel.
__global__ void __launch_bounds__(256) batch_tfsf_kernel(const BMember* __restrict__ mem, const BRow* __restrict__ rows) {
    const BRow r = rows[blockIdx.y];
    const BMember& M = mem[r.m];
    if (!b_active(M)) return;
    tfsf_point(*M.rp, r.s, blockIdx.x * blockDim.x + threadIdx.x, M.it - 1);
}

// Monitor gather (monitor_gather_kernel): field monitors without sum to their history,
// the others to the member's staging ring, slot = steps since ring_first.
__global__ void __launch_bounds__(256) batch_gather_kernel(const BMember* __restrict__ mem, const BPoint* __restrict__ pts,
                                                           const int* __restrict__ npts) {
    const int n = *npts;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const BPoint e = pts[i];
        const BMember& M = mem[e.m];
        if (!b_active(M)) continue;
        const MonParams<float>& p = *M.mp;
        const MonDev<float>& D = p.mons[e.s];
        const long long it0 = M.it - 1;
        const int cell = D.cells[e.i];
        if (D.kind == MFD_MON_FIELD && !D.sum) {
            for (int k = 0; k < p.ncomp; ++k) D.hist[((long long)k * p.nt + it0) * D.npts + e.i] = p.comp[k][cell];
        } else {
            const long long slot = it0 - M.ring_first;
            for (int k = 0; k < p.ncomp; ++k) D.ring[(slot * p.ncomp + k) * D.npts + e.i] = p.comp[k][cell];
        }
    }
}

// End of a batch step: every active member moves to its next step.
__global__ void batch_advance_kernel(BMember* __restrict__ mem, int n) {
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += gridDim.x * blockDim.x)
        if (mem[m].it <= mem[m].last) mem[m].it += 1;
}

}  // namespace mfd
