// geometry.cuh -- the material index map built on the device from analytic shapes.
//
// The reference evaluates a Julia closure geometry(x, y, z) at every grid point on the host,
// one material after another, later materials overwriting earlier ones (src/util.jl:1-31,
// src/models.jl:85-98).  For shapes given as parameters (mfd_shape, include/maxwellfdtd.h)
// each thread takes one cell, tests the shapes in order and writes the index of the last one
// that covers it; a second pass finds each material's bounding box (atomic min/max), which
// the engine reads back to size the materials' compact state.  Every test is the header's
// double-precision expression, evaluated left to right without fused multiply-adds (the
// library is built with contraction off), so it matches a host evaluation of the same
// expression bit for bit.
#pragma once

#include "mfd_device.cuh"

namespace mfd {

__host__ __device__ __forceinline__ bool shape_covers(const mfd_shape& s, double x, double y, double z) {
    const double* p = s.p;
    switch (s.kind) {
        case MFD_SHAPE_BALL: {
            const double a = x - p[0], b = y - p[1], c = z - p[2];
            return (a * a + b * b) + c * c <= p[3] * p[3];
        }
        case MFD_SHAPE_BOX:
            return p[0] <= x && x <= p[1] && p[2] <= y && y <= p[3] && p[4] <= z && z <= p[5];
        case MFD_SHAPE_ELLIPSOID: {
            const double a = (x - p[0]) / p[3], b = (y - p[1]) / p[4], c = (z - p[2]) / p[5];
            return (a * a + b * b) + c * c <= 1.0;
        }
        case MFD_SHAPE_CYLINDER: {
            const double a = x - p[0], b = y - p[1];
            return a * a + b * b <= p[2] * p[2] && p[3] <= z && z <= p[4];
        }
        case MFD_SHAPE_HALFSPACE:
            return (p[0] * x + p[1] * y) + p[2] * z >= p[3];
        case MFD_SHAPE_ALL:
            return true;
        default:
            return false;
    }
}

// The padded map (x fastest) and, in the same pass, the bounding box of each material's cells:
// box[6 (g - 1) + {0..5}] = x0, x1, y0, y1, z0, z1 (initialised to INT_MAX / -1), and their number,
// count[g - 1].  1-D and 2-D grids take the missing coordinates as 0 (2-D: y; 1-D: x and y).
//
// A warp walks rows 32 cells at a time.  The lanes of one material are found with a ballot, so
// a segment gives at most one candidate interval per material; it is merged into the block's
// boxes in shared memory (an atomic only when it widens them, which soon becomes rare), and each
// block merges its boxes into the global ones once.  What bounds it is the shapes' FP64 tests;
// the six global atomics per material cell that a pass of its own took before were serialised
// on six addresses per material (mfd_create of a 96 x 96 x 512 whole-domain glass: 19.6 ms
// then, 1.1 now; of 1801 x 1203 cells with three materials: 2.2 ms then, 0.9 now).
constexpr int GEO_TY = 8;

__global__ void __launch_bounds__(32 * GEO_TY) geometry_kernel(uint8_t* __restrict__ geom, const Layout L,
                                                               const mfd_shape* __restrict__ shapes, const int nshape,
                                                               const double* __restrict__ xs, const double* __restrict__ ys,
                                                               const double* __restrict__ zs, int* box, int* count, const int nmat) {
    __shared__ int sb[6 * 255], sc[255];
    const int lane = threadIdx.x, tid = threadIdx.x + 32 * threadIdx.y;
    for (int i = tid; i < 6 * nmat; i += 32 * GEO_TY) sb[i] = (i & 1) ? -1 : 0x7fffffff;
    for (int i = tid; i < nmat; i += 32 * GEO_TY) sc[i] = 0;
    __syncthreads();
    const long long rows = (long long)L.ny * L.nz;
    for (long long row = (long long)blockIdx.x * GEO_TY + threadIdx.y; row < rows; row += (long long)gridDim.x * GEO_TY) {
        const int iz = (int)(row / L.ny), iy = (int)(row - (long long)iz * L.ny);
        const double y = ys ? ys[iy] : 0.0, z = zs[iz];
        for (int x0 = 0; x0 < L.nx; x0 += 32) {
            const int ix = x0 + lane;
            int g = 0;
            if (ix < L.nx) {
                const double x = xs ? xs[ix] : 0.0;
                for (int s = 0; s < nshape; ++s)
                    if (shape_covers(shapes[s], x, y, z)) g = shapes[s].material;
                g = (uint8_t)g;   // what the map holds
                geom[ix + (long long)L.px * iy + (long long)L.sz * iz] = (uint8_t)g;
            }
            unsigned todo = __ballot_sync(0xffffffffu, g != 0);
            while (todo) {
                const int first = __ffs((int)todo) - 1;
                const int gl = __shfl_sync(0xffffffffu, g, first);
                const unsigned m = __ballot_sync(0xffffffffu, g == gl);
                if (lane == first) {
                    int* b = sb + 6 * (gl - 1);
                    const int hi = x0 + 31 - __clz((int)m);
                    if (ix < b[0]) atomicMin(b + 0, ix);
                    if (hi > b[1]) atomicMax(b + 1, hi);
                    if (iy < b[2]) atomicMin(b + 2, iy);
                    if (iy > b[3]) atomicMax(b + 3, iy);
                    if (iz < b[4]) atomicMin(b + 4, iz);
                    if (iz > b[5]) atomicMax(b + 5, iz);
                    atomicAdd(&sc[gl - 1], __popc(m));
                }
                todo &= ~m;
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < 6 * nmat; i += 32 * GEO_TY) {
        if (i & 1) { if (sb[i] >= 0) atomicMax(box + i, sb[i]); }
        else if (sb[i] != 0x7fffffff) atomicMin(box + i, sb[i]);
    }
    for (int i = tid; i < nmat; i += 32 * GEO_TY)
        if (sc[i]) atomicAdd(count + i, sc[i]);
}

}  // namespace mfd
