// footprint.cuh -- the device arrays of a model, from its descriptor (host code).
//
// One list serves two uses: the engine reserves the memory of a model's small arrays as one block
// of exactly their size, and the server's admission estimate (desc_footprint in serve.cuh) adds the
// same arrays up before anything is allocated.
#pragma once

#include "aux.cuh"

namespace mfd {

// Every array starts on a 256-byte boundary of its block.
static int64_t array_room(int64_t bytes) { return (std::max<int64_t>(bytes, 1) + 255) / 256 * 256; }

static int64_t padded_nx(const mfd_desc* d) { return d->ndim == 1 ? d->nx : ((int64_t)d->nx + 31) / 32 * 32; }
static int64_t padded_cells(const mfd_desc* d) { return padded_nx(d) * d->ny * d->nz; }
static int64_t desc_tsize(const mfd_desc* d) { return d->dtype == MFD_F64 ? 8 : 4; }

// Read-backs of rows below PACK_ROW bytes are packed on the device, PACK_BYTES at a time at most:
// the size of a model's buffer for it (0: its rows are long, or dense already).
constexpr int64_t PACK_ROW = 1024, PACK_BYTES = 8 << 20;
static int64_t pack_bytes(int64_t nx, int64_t px, int64_t cells, int64_t tsize) {
    if (nx == px || nx * tsize >= PACK_ROW) return 0;
    return std::min(std::max(cells * tsize, 8 * nx), PACK_BYTES);   // a row of any element type
}

// f(bytes) for every array that mfd_create makes of a descriptor, but for the TFSF replay's and those
// that depend on where the materials lie (each_material_array).
template <typename F>
static void each_array(const mfd_desc* d, F&& f) {
    const int64_t T = desc_tsize(d), nt = d->nt, px = padded_nx(d), Np = padded_cells(d);
    const int nd = d->ndim;
    static const int ncomp[4] = {0, 3, 5, 9}, ncm[4] = {0, 2, 3, 6};
    const bool ey2 = nd == 2 && d->polarization == MFD_POL_EY;   // Hx, Hz, Dy, Ey
    for (int k = 0; k < (ey2 ? 4 : ncomp[nd]) + 1; ++k) f(Np * T);   // fields, running sum
    f(nt * 4);                                                       // per-step flags
    if (!d->geometry && d->nshape > 0) {   // the map made from shapes
        f(Np);
        f((int64_t)d->nshape * (int64_t)sizeof(mfd_shape));
        f(d->nx * 8ll);
        f(d->ny * 8ll);
        f(d->nz * 8ll);
        f(7 * 4 * (int64_t)d->nmat);
    }
    if (d->nmat > 0) {
        f(d->nmat * T);
        f(d->nmat * (int64_t)sizeof(MatDev<double, double>));
    }
    for (int k = 0; k < 6; ++k) {
        const int64_t nb = d->pml[k].nb;
        const int axis = k / 2;
        if (nb <= 0 || !(nd == 3 || (nd == 2 && axis != 1) || (nd == 1 && axis == 2))) continue;
        f(nb * 8 * T);   // divisors
        f(nb * T);
        f(nb * T);
        const int64_t cnt = nd == 1 ? nb : nd == 2 ? (axis == 0 ? nb * d->nz : px * nb)
                                                   : axis == 0 ? nb * d->ny * d->nz : axis == 1 ? px * nb * d->nz : px * d->ny * nb;
        for (int j = 0; j < (nd == 3 ? 4 : 2); ++j) f(cnt * T);
    }
    for (int i = 0; i < d->nsrc; ++i) {
        const mfd_source& s = d->srcs[i];
        if (s.npts < 1) continue;
        f(s.npts * 8);
        if (s.wave) f(nt * s.npts * 8);
        else {
            f(s.npts * 8);
            f(nt * 8);
        }
    }
    int64_t ring_vals = 0;
    for (int i = 0; i < d->nmon; ++i) {
        const mfd_monitor& m = d->mons[i];
        if (m.npts < 1) continue;
        if (m.kind != MFD_MON_FIELD || m.sum) ring_vals += ncm[nd] * m.npts;
    }
    const int64_t slots = ring_vals ? std::max<int64_t>(1, std::min<int64_t>(MFD_DFT_MAXSLOTS, (512ll << 20) / (T * ring_vals))) : 0;
    for (int i = 0; i < d->nmon; ++i) {
        const mfd_monitor& m = d->mons[i];
        if (m.npts < 1) continue;
        f(m.npts * 4);
        if (m.kind == MFD_MON_FIELD) f(ncm[nd] * nt * (m.sum ? 1 : m.npts) * T);
        else if (m.nw > 0) {
            f(ncm[nd] * (int64_t)m.nw * (m.sum ? 1 : m.npts) * 16);
            f(nt * (int64_t)m.nw * 16);
        }
        if (m.kind != MFD_MON_FIELD || m.sum) f(slots * ncm[nd] * m.npts * T);
    }
    if (d->nmon > 0) {
        f(d->nmon * (int64_t)sizeof(MonDev<double>));
        f(4);   // the fold's status
    }
}

// f(bytes) for the arrays of a model whose material m (0-based) fills a box of box_cells[m] cells, 0 where
// no cell holds it.
template <typename F>
static void each_material_array(const mfd_desc* d, const std::vector<int64_t>& box_cells, F&& f) {
    const int64_t T = desc_tsize(d), R = (T == 8 || d->rho_fp64) ? 8 : 4, Np = padded_cells(d);
    const int nc = d->ndim;
    bool any = false;
    for (int m = 0; m < d->nmat; ++m) {
        const mfd_material& s = d->mats[m];
        const int64_t bs = box_cells[m];
        if (s.plasma && s.rate_kind == MFD_RATE_TABLE) {   // present or not
            f(s.rate_n * T);
            f(s.rate_n * T);
        }
        if (!bs) continue;
        any = true;
        if (s.nq > 0) f(2 * s.nq * nc * bs * T);
        if (s.plasma) {
            f(2 * nc * bs * T);
            f(nc * bs * T);
            f(bs * R);
            f(bs * R);
            f(bs * T);
        }
    }
    if (!any) return;
    if (d->geometry) f(Np);
    f(Np * T);   // the second running sum
}

}  // namespace mfd
