"""Sources that write H in the resident steps (TFSF replay, soft and hard point sources on H) against
the separate launches of the same library, which a profiled run always takes: bit for bit (tolerance
zero), on grids of one block, one cluster and many blocks of one and of several rounds of cells per
thread.  The sources cover whole runs of cells, so both sides of block boundaries are among them, and
a dispersive half-space makes the blocks' E updates differ in length: a block that is done must not
change an H that a slower one has yet to read.  H monitors lie on the same cells."""
import numpy as np
import pytest

import cases as C
import maxwellfdtd_b200 as M
from maxwellfdtd_b200 import _abi
from maxwellfdtd_b200.sources import comp_index, field_components
from test_gpu_resident import _outputs, _same

pytestmark = pytest.mark.gpu

D = 50e-9
# threads of a block at most: 640 (float), 512 (double); a cluster of 8 blocks up to 5120 / 4096 cells
SIZES = [(1, 1, 128), (1, 1, 129), (1, 1, 4097), (1, 1, 5121), (1, 1, 60013), (64, 1, 64), (331, 1, 577), (806, 1, 805),
         (16, 16, 20), (67, 61, 59), (90, 91, 79)]


def _grid(n):
    nd = 3 if n[1] > 1 else 2 if n[0] > 1 else 1
    return nd, (C.grid3(n, D) if nd == 3 else C.grid2((n[0], n[2]), D) if nd == 2 else C.grid1(n[2], D))


def _steps(n):
    return 60 if n[0] * n[1] * n[2] > 500000 else 150


def _half_space(z0):
    return M.Material(geometry=lambda *c: c[-1] > z0, eps=2.25,
                      chi=[M.DrudeSusceptibility(wp=1.37e16, gamma=1.07e14), M.LorentzSusceptibility(deps=1.1, w0=4.2e15, delta=5e14)])


def _compare(model, mons, lib, dtype, mode):
    ref, n2 = _outputs(model, lib, dtype, mons, mode, True, [])
    one, n1 = _outputs(model, lib, dtype, mons, mode, False, [])
    cut, _ = _outputs(model, lib, dtype, mons, mode, False, [1, 2, 31])
    assert n1 < n2 / 4, "the model must have taken the resident steps"
    _same(ref, one)
    _same(ref, cut)
    for c in ("Hy", "Hx", "Ex", "Ey"):
        if c in ref:
            assert np.isfinite(ref[c]).all() and np.abs(ref[c]).max() > 0


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("pol", ["Hy", "Ey"])
@pytest.mark.parametrize("n", SIZES)
def test_h_point_sources(n, pol, dtype, mode, gpu_lib):
    nd, g = _grid(n)
    if pol == "Ey" and nd != 2:
        pytest.skip("the second field set is 2-D")
    half = (n[2] - 1) / 2 * D
    band = lambda *c: np.abs(c[-1]) < 0.2 * half          # a fifth of the rows: whole runs of cells
    point = lambda f: tuple([f * float(a[-1]) for a in ((g.x, g.y, g.z) if nd == 3 else (g.x, g.z) if nd == 2 else (g.z,))])
    hs = [c for c in field_components(nd, pol) if c[0] == "H"]
    e0 = "Ey" if pol == "Ey" else "Ex"

    def wave(*a):
        return 1e-3 * C.pulse(a[-1], t0=3e-15) * np.cos(sum(x / (3.7 * D) for x in a[:-1]))
    src = [M.SoftSource(geometry=point(0.05), waveform=lambda *a: C.pulse(a[-1], t0=3e-15), component=e0)]
    for k, c in enumerate(hs):
        src.append(M.SoftSource(geometry=band, component=c,
                                waveform=M.SeparableWaveform(lambda *x, k=k: np.cos(sum(v / ((3.3 + k) * D) for v in x)),
                                                             lambda t: 1e-3 * C.pulse(t, t0=3e-15))))
        src.append(M.HardSource(geometry=lambda *x, k=k: band(*x) & (np.abs(np.sin(x[-1] / D * 0.9 + k)) < 0.2) if nd == 1 else
                                band(*x) & (np.abs(x[0] - 2.2 * k * D) < 0.6 * D), waveform=wave, component=c))
        src.append(M.SoftSource(geometry=point(-0.1), waveform=wave, component=e0, explicit=True))
    plane = lambda *c: np.abs(c[-1]) < 0.6 * D
    mons = [M.FieldMonitor(plane), M.SpectralMonitor(plane, sum=True), M.FieldMonitor(point(-0.1))]
    model = M.Model(g, src, tmax=(_steps(n) - 0.5) * M.model.time_step(g, 0.5), pml=5 * D if min(k for k in n if k > 1) > 30 else 0,
                    material=_half_space(0.0), polarization=pol)
    _compare(model, mons, gpu_lib, dtype, mode)


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [(1, 1, 2001), (1, 1, 60013), (64, 1, 64), (331, 1, 577), (61, 48, 55), (67, 61, 59)])
def test_tfsf(n, dtype, mode, gpu_lib):
    nd, g = _grid(n)
    steps = 150
    dt = M.model.time_step(g, 0.5)
    ext = [0.3 * (k - 1) * D for k in n if k > 1]          # the box spans 0.6 of each axis
    z0 = -ext[-1] - 4 * D
    rec = M.Model(g, M.SoftSource(geometry=lambda *c: np.abs(c[-1] - z0) < 0.6 * D, waveform=lambda *a: C.pulse(a[-1], t0=3e-15),
                                  component="Ex"), tmax=(steps - 0.5) * dt, pml=(0,) * (2 * nd - 2) + (5 * D, 5 * D))
    sol = M.solve(rec, backend=M.B200(dtype, library=gpu_lib), tfsf_record=True, tfsf_box=tuple(s * e for e in ext for s in (-1, 1)),
                  tfsf_fname=C._tmp_name())
    plane = lambda *c: np.abs(c[-1] + ext[-1]) < 1.6 * D    # the box's first face, H on both sides of it
    model = M.Model(g, M.TFSFSource(data=sol.out["tfsf_record"]), tmax=(steps - 0.5) * dt, pml=5 * D,
                    material=_half_space(-ext[-1] + 6 * D))
    _compare(model, [M.FieldMonitor(plane), M.SpectralMonitor(plane, sum=True)], gpu_lib, dtype, mode)


@pytest.mark.parametrize("n", [(1, 1, 2001), (201, 1, 149), (61, 48, 55)])
def test_point_lists_at_the_first_run_that_uses_them(n, gpu_lib):
    """A model that is stepped otherwise (profiled here; by a batch) makes no lists: device memory grows
    at the first resident run only, and runs before it in another way change nothing."""
    nd, g = _grid(n)
    src = M.SoftSource(geometry=(0.0,) * nd, waveform=lambda *a: C.pulse(a[-1], t0=3e-15), component="Ex")
    model = M.Model(g, src, tmax=40.5 * M.model.time_step(g, 0.5), pml=5 * D)
    b, _ = model.build_desc(np.float32, [M.FieldMonitor((0.0,) * nd)])
    fields = []
    for profiled in (0, 9):
        st = _abi.Stepper(gpu_lib, b, np.float32)
        made = st.device_bytes()
        if profiled:
            st.set_profiling(True)
            st.run(1, profiled)
            assert st.device_bytes() == made
            st.set_profiling(False)
        st.run(profiled + 1, model.Nt)
        assert st.device_bytes() > made
        fields.append([st.read_field(comp_index(c)) for c in field_components(nd)])
        st.close()
    assert all(np.array_equal(a, c) for a, c in zip(*fields))


# around one block (128 cells), one cluster (8 blocks of 640 or 512 threads) and one round of 148 blocks
SMALL = [("float32", n) for n in ((1, 1, 128), (1, 1, 129), (1, 1, 5120), (1, 1, 5121), (64, 1, 80), (61, 1, 84), (320, 1, 296), (313, 1, 303))] + \
        [("float64", n) for n in ((1, 1, 128), (1, 1, 129), (1, 1, 4096), (1, 1, 4097), (256, 1, 296), (257, 1, 295))]
# the largest models that step so and the next: (type, mode, field set, medium, H source, the larger of the two sizes)
LIMITS = [("float32", "exact", "Hy", "response", False, (807, 1, 806)), ("float32", "fast", "Hy", "map", True, (807, 1, 806)),
          ("float32", "exact", "Hy", "light", True, (709, 1, 706)), ("float64", "fast", "Hy", "light", True, (709, 1, 706)),
          ("float64", "exact", "Hy", "light", False, (807, 1, 806)), ("float64", "fast", "Ey", "light", False, (895, 1, 894)),
          ("float32", "fast", "Ey", "light", False, (1001, 1, 1000)), ("float32", "exact", "Ey", "map", False, (1001, 1, 1000)),
          ("float64", "exact", "Hy", "map", False, (922, 1, 922)), ("float64", "exact", "Hy", "response", False, (1001, 1, 1000)),
          ("float32", "exact", "", "map", True, (100, 100, 76)), ("float64", "exact", "", "response", False, (100, 100, 76)),
          ("float64", "exact", "", "map", True, (100, 100, 66)), ("float64", "fast", "", "response", True, (100, 100, 66)),
          ("float64", "fast", "", "light", False, (100, 100, 66)), ("float64", "fast", "", "light", True, (100, 100, 36)),
          ("float64", "fast", "", "map", False, (100, 100, 36))]


def _threshold(dtype, mode, pol, medium, hsrc, n, small, lib):
    nd, g = _grid(n)
    dt = np.dtype(dtype).type
    at = tuple(0.11 * float(a[-1]) for a in ((g.x, g.y, g.z) if nd == 3 else (g.x, g.z) if nd == 2 else (g.z,)))
    src = [M.SoftSource(geometry=at, waveform=lambda *a: C.pulse(a[-1], t0=3e-15), component="Ey" if pol == "Ey" else "Ex")]
    if hsrc:
        src.append(M.SoftSource(geometry=at, waveform=lambda *a: 1e-3 * C.pulse(a[-1], t0=2e-15), component="Hy"))
    plane = lambda *c: np.abs(c[-1] - at[-1]) < 0.6 * D
    mons = [M.FieldMonitor(at), M.SpectralMonitor(plane, sum=True)]
    mat = {"light": None, "map": M.Material(geometry=lambda *c: c[-1] > at[-1], eps=2.25), "response": _half_space(at[-1])}[medium]
    model = M.Model(g, src, tmax=40.5 * M.model.time_step(g, 0.5), pml=5 * D, material=mat, polarization=pol or "Hy")
    ref, n2 = _outputs(model, lib, dt, mons, mode, True, [])
    got, n1 = _outputs(model, lib, dt, mons, mode, False, [5])
    assert (n1 < n2 / 4) == small
    _same(ref, got)
    assert np.abs(got["Ey" if pol == "Ey" else "Ex"]).max() > 0


@pytest.mark.parametrize("dtype,n", SMALL)
def test_sizes_around_blocks_and_clusters(dtype, n, gpu_lib):
    _threshold(dtype, "exact", "", "response", False, n, True, gpu_lib)


@pytest.mark.parametrize("dtype,mode,pol,medium,hsrc,n", LIMITS)
def test_largest_resident_models(dtype, mode, pol, medium, hsrc, n, gpu_lib):
    below = n[:2] + (n[2] - 1,) if n[1] > 1 else (n[0] - 1, 1, n[2])
    _threshold(dtype, mode, pol, medium, hsrc, n, False, gpu_lib)
    _threshold(dtype, mode, pol, medium, hsrc, below, True, gpu_lib)
