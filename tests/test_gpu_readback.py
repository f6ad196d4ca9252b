"""Reads of fields, running sums and the material map on a device that has no memory left: they copy
arrays that are there, so they must work, and give the values that they give with memory to spare
(tolerance zero).  So must the steps of a small model, which build their point lists at its first run
and take the separate launches without them.  The device's allocations are taken from a small pool of the test's own while it
is full, through the driver API: no memory of the device is filled."""
import ctypes as C

import numpy as np
import pytest

import cases
import maxwellfdtd_b200 as M
from maxwellfdtd_b200 import _abi
from maxwellfdtd_b200.sources import comp_index, field_components

pytestmark = pytest.mark.gpu


class _PoolProps(C.Structure):   # CUmemPoolProps
    _fields_ = [("allocType", C.c_int), ("handleTypes", C.c_int), ("locType", C.c_int), ("locId", C.c_int),
                ("win32", C.c_void_p), ("maxSize", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


class _FullPool:
    """Within the block every cudaMallocAsync of 512 bytes or more fails: the device's pool is one of
    `size` bytes at most, filled."""

    def __init__(self, size=4 << 20):
        self.cu = C.CDLL("libcuda.so.1")
        for f, a in {"cuMemPoolCreate": [C.POINTER(C.c_void_p), C.POINTER(_PoolProps)], "cuDeviceGetMemPool": [C.POINTER(C.c_void_p), C.c_int],
                     "cuDeviceSetMemPool": [C.c_int, C.c_void_p], "cuMemPoolDestroy": [C.c_void_p],
                     "cuMemAllocFromPoolAsync": [C.POINTER(C.c_uint64), C.c_size_t, C.c_void_p, C.c_void_p],
                     "cuMemFreeAsync": [C.c_uint64, C.c_void_p], "cuStreamSynchronize": [C.c_void_p]}.items():
            getattr(self.cu, f).argtypes = a
        self.size = size

    def __enter__(self):
        cu, self.old, self.pool, self.held = self.cu, C.c_void_p(), C.c_void_p(), []
        props = _PoolProps(allocType=1, handleTypes=0, locType=1, locId=0, maxSize=self.size)   # pinned, no handles, device 0
        assert cu.cuDeviceGetMemPool(C.byref(self.old), 0) == 0
        assert cu.cuMemPoolCreate(C.byref(self.pool), C.byref(props)) == 0
        for piece in (64 << 10, 512):   # at most 256 MiB, should the limit be rounded up
            for _ in range(4096):
                p = C.c_uint64()
                if cu.cuMemAllocFromPoolAsync(C.byref(p), piece, self.pool, None) != 0:
                    break
                self.held.append(p.value)
            else:
                raise AssertionError("the pool has no limit")
        assert cu.cuDeviceSetMemPool(0, self.pool) == 0
        return self

    def __exit__(self, *exc):
        cu = self.cu
        cu.cuDeviceSetMemPool(0, self.old)
        for p in self.held:
            cu.cuMemFreeAsync(p, None)
        cu.cuStreamSynchronize(None)
        cu.cuMemPoolDestroy(self.pool)


def _reads(st, model):
    out = {c: st.read_field(comp_index(c)) for c in field_components(model.grid.ndim)}
    out["Sa"], out["E2"] = st.read_integral(_abi.MFD_INT_SA), st.read_integral(_abi.MFD_INT_E2)
    out["geometry"] = st.read_geometry()
    return out


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [(37, 1, 211), (255, 1, 700), (61, 48, 55), (300, 1, 301)])
def test_reads_without_device_memory(n, dtype, gpu_lib):
    nd = 3 if n[1] > 1 else 2
    g = cases.grid3(n) if nd == 3 else cases.grid2((n[0], n[2]))
    src = M.SoftSource(geometry=(0.0,) * nd, waveform=lambda *a: cases.pulse(a[-1], t0=2e-15), component="Ez")
    mat = M.Material(geometry=lambda *c: c[-1] > 100e-9, eps=2.25)
    model = M.Model(g, src, tmax=30.5 * M.model.time_step(g, 0.5), pml=0, material=mat)
    b, _ = model.build_desc(dtype, None)
    steppers = [_abi.Stepper(gpu_lib, b, dtype) for _ in range(2)]
    try:
        for st in steppers:
            st.run(1, model.Nt)
        ref = _reads(steppers[0], model)
        with _FullPool():
            got = _reads(steppers[1], model)   # its first reads
        again = _reads(steppers[1], model)
    finally:
        for st in steppers:
            st.close()
    for k in ref:
        assert np.array_equal(ref[k], got[k]) and np.array_equal(ref[k], again[k]), k
    assert np.abs(ref["Ez"]).max() > 0 and ref["geometry"].max() == 1


@pytest.mark.parametrize("n", [(1, 1, 2001), (201, 1, 149), (67, 61, 59)])
def test_first_run_without_device_memory(n, gpu_lib):
    nd = 3 if n[1] > 1 else 2 if n[0] > 1 else 1
    g = cases.grid3(n) if nd == 3 else cases.grid2((n[0], n[2])) if nd == 2 else cases.grid1(n[2])
    src = M.SoftSource(geometry=(0.0,) * nd, waveform=lambda *a: cases.pulse(a[-1], t0=2e-15), component="Ex")
    model = M.Model(g, src, tmax=40.5 * M.model.time_step(g, 0.5), pml=0)
    mons = [M.FieldMonitor(lambda *c: np.abs(c[-1]) < 60e-9)]
    b, _ = model.build_desc(np.float32, mons)
    out, launches = [], []
    for full in (False, True):
        st = _abi.Stepper(gpu_lib, b, np.float32)
        try:
            st.set_profiling(False)
            if full:
                with _FullPool():
                    st.run(1, 7)
                st.run(8, model.Nt)
            else:
                st.run(1, 7)
                st.run(8, model.Nt)
            launches.append(sum(v[1] for v in st.kernel_times().values()))
            shape = (model.Nt, int(b.desc.mons[0].npts))
            out.append([st.read_field(comp_index(c)) for c in field_components(nd)] + [st.read_integral(_abi.MFD_INT_SA)] +
                       [st.read_monitor(0, comp_index(c), shape, False) for c in field_components(nd) if c[0] != "D"])
        finally:
            st.close()
    assert launches[0] < launches[1] / 4
    for a, c in zip(*out):
        assert np.array_equal(a, c)
    assert np.abs(out[0][-1]).max() > 0
