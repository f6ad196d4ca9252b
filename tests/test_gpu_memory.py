"""Device memory that a model takes, as the device's memory pool counts it (driver API), against what
mfd_device_bytes reports and what the admission estimates allow for: after mfd_create, and after the
reads that follow.  The pool rounds each allocation up to its granularity, which is measured here; a
model's arrays below 4 MiB come in at most 8 allocations."""
import ctypes as C

import numpy as np
import pytest

import cases
import maxwellfdtd_b200 as M
from maxwellfdtd_b200 import _abi, serve
from maxwellfdtd_b200.sources import comp_index, field_components
from test_zz_no_alloc import _default_pool

pytestmark = pytest.mark.gpu

D = 50e-9


def _granularity(used):
    cu = C.CDLL("libcuda.so.1")
    cu.cuMemAllocAsync.argtypes = [C.POINTER(C.c_uint64), C.c_size_t, C.c_void_p]
    cu.cuMemFreeAsync.argtypes = [C.c_uint64, C.c_void_p]
    p, base = C.c_uint64(), used()
    assert cu.cuMemAllocAsync(C.byref(p), 1, None) == 0
    g = used() - base
    assert cu.cuMemFreeAsync(p, None) == 0 and cu.cuStreamSynchronize(None) == 0
    return g


def _model(n):
    nd = 3 if n[1] > 1 else 2 if n[0] > 1 else 1
    g = cases.grid3(n, D) if nd == 3 else cases.grid2((n[0], n[2]), D) if nd == 2 else cases.grid1(n[2], D)
    src = M.SoftSource(geometry=(0.0,) * nd, waveform=lambda *a: cases.pulse(a[-1], t0=2e-15), component="Ex")
    r = 0.2 * min(k for k in n if k > 1) * D
    mats = [M.Material(geometry=cases._ball(nd, r), eps=2.25, chi=[M.DrudeSusceptibility(wp=1.37e16, gamma=1.07e14),
                                                                    M.LorentzSusceptibility(deps=1.1, w0=4.2e15, delta=5e14)]),
            M.Material(geometry=lambda *c: c[-1] > 2 * r, eps=2.0)]
    model = M.Model(g, src, tmax=20.5 * M.model.time_step(g, 0.5), pml=8 * D, material=mats)
    return model, [M.FieldMonitor((0.0,) * nd), M.SpectralMonitor(lambda *c: np.abs(c[-1]) < 0.6 * D, w=[1.5e15, 2e15])]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [(1, 1, 2001), (33, 1, 40), (256, 1, 256), (200, 1, 201), (400, 1, 400), (700, 1, 700), (48, 48, 48),
                               (61, 48, 55), (127, 90, 60)])
def test_device_bytes_are_what_the_pool_gave(n, dtype, gpu_lib):
    model, mons = _model(n)
    b, _ = model.build_desc(dtype, mons)
    estimates = (gpu_lib.server_footprint(C.byref(b.desc)), serve.footprint(b, model, dtype))
    _abi.Stepper(gpu_lib, b, dtype).close()   # the process's first use of these divisors, of the device
    used, _, _ = _default_pool()
    g, base = _granularity(used), used()
    st = _abi.Stepper(gpu_lib, b, dtype)
    try:
        own = 12 * (n[0] * n[1] * n[2] * np.dtype(dtype).itemsize > 3 << 20)   # arrays above 4 MiB, padded
        made, said = used() - base, st.device_bytes()
        assert said <= made <= said + (8 + own) * g, (n, said, made, g)
        for c in field_components(model.grid.ndim):
            st.read_field(comp_index(c))
        st.read_integral(_abi.MFD_INT_SA)
        read, said = used() - base, st.device_bytes()
        assert said <= read <= said + (9 + own) * g, (n, said, read, g)
        for est in estimates:
            assert read <= est + (8 + own) * g and est <= 1.1 * read + (1 << 20), (n, read, est)
    finally:
        st.close()
