"""The resident steps (many steps of a small model in one cooperative launch) against the
separate launches of the same library, which a profiled run always takes, and against the
oracle.  Both run the same cell code, so every output is bit-identical (tolerance zero)."""
import numpy as np
import pytest

import cases as C
import maxwellfdtd_b200 as M
from maxwellfdtd_b200 import _abi
from maxwellfdtd_b200.sources import comp_index, field_components

pytestmark = pytest.mark.gpu


def _outputs(model, lib, dtype, mons, mode, profiled, cuts):
    """Every output, the run cut into mfd_run calls after the given steps."""
    b, meta = model.build_desc(dtype, mons, mode=mode)
    st = _abi.Stepper(lib, b, dtype)
    if profiled is not None:
        st.set_profiling(profiled)
    a = 1
    for c in list(cuts) + [model.Nt]:
        st.run(a, c)
        a = c + 1
    n = sum(v[1] for v in st.kernel_times().values()) if profiled is not None else None
    out = {c: st.read_field(comp_index(c)) for c in field_components(model.grid.ndim, model.polarization)}
    out["Sa"], out["E2"] = st.read_integral(_abi.MFD_INT_SA), st.read_integral(_abi.MFD_INT_E2)
    for k, ms in enumerate(meta["monitors"]):
        spectral = ms["kind"] == 1
        rows = ms["dft"].Nw if spectral else model.Nt
        for c in field_components(model.grid.ndim, model.polarization):
            if c[0] != "D":
                out[f"mon{k}.{c}"] = st.read_monitor(k, comp_index(c), (rows,) if ms["sum"] else (rows, len(ms["cells"])), spectral)
    st.close()
    return out, n


def _same(a, b):
    assert set(a) == set(b)
    bad = [k for k in a if not np.array_equal(a[k], b[k], equal_nan=True)]
    assert not bad, bad


@pytest.mark.parametrize("mode", ["exact", "fast"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("builder", ["vacuum", "bcs", "materials", "sources"])
def test_equals_separate_launches(builder, ndim, dtype, mode, gpu_lib):
    model = getattr(C, "model_" + builder)(ndim)
    mons = C.monitors(ndim)
    one, n1 = _outputs(model, gpu_lib, dtype, mons, mode, False, [])
    cut, _ = _outputs(model, gpu_lib, dtype, mons, mode, False, [1, 2, 20])
    ref, n2 = _outputs(model, gpu_lib, dtype, mons, mode, True, [])
    assert n1 < n2 / 4, "the model must have taken the resident steps"
    _same(ref, one)
    _same(ref, cut)
    assert np.abs(one["Ex"]).max() > 0


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("ndim", [1, 2, 3])
def test_tfsf_replay(ndim, dtype, gpu_lib):
    sol = M.solve(C.model_tfsf_record(ndim), backend=M.B200(dtype, library=gpu_lib), tfsf_record=True,
                  tfsf_box=C.tfsf_box(ndim), tfsf_fname=C._tmp_name())
    model = C.model_tfsf_replay(ndim, sol.out["tfsf_record"])
    ref, _ = _outputs(model, gpu_lib, dtype, C.monitors(ndim), "exact", True, [])
    got, _ = _outputs(model, gpu_lib, dtype, C.monitors(ndim), "exact", False, [7])
    _same(ref, got)
    assert np.abs(got["Ex"]).max() > 0


# cells at the edges of a block's run (512 threads, one cell each): one less, equal, one more;
# two and a half blocks; a prime row length so rows straddle blocks; several cells per thread
SIZES = [(1, 1, 511), (1, 1, 512), (1, 1, 513), (16, 1, 32), (16, 1, 33), (127, 1, 11), (8, 8, 8), (13, 7, 17),
         (1, 1, 40007), (331, 1, 577), (67, 61, 59)]


@pytest.mark.parametrize("n", SIZES)
def test_block_edges_against_oracle(n, gpu_lib, oracle_lib):
    nd = 3 if n[1] > 1 else 2 if n[0] > 1 else 1
    g = C.grid3(n) if nd == 3 else C.grid2((n[0], n[2])) if nd == 2 else C.grid1(n[2])
    at = tuple(float(c[len(c) // 2]) for c in ((g.x, g.y, g.z) if nd == 3 else (g.x, g.z) if nd == 2 else (g.z,)))
    src = M.SoftSource(geometry=at, waveform=lambda *a: 1e3 * C.pulse(a[-1], t0=4e-15), component="Ex")
    mat = M.Material(geometry=lambda *c: c[-1] > 0, eps=2.25, chi=M.DrudeSusceptibility(wp=1.37e16, gamma=1.07e14))
    model = M.Model(g, src, tmax=39.5 * M.model.time_step(g, 0.5), pml=0, material=mat)
    mons = [M.FieldMonitor(at)]
    ref, _ = _outputs(model, oracle_lib, np.float32, mons, "exact", None, [])
    got, _ = _outputs(model, gpu_lib, np.float32, mons, "exact", False, [5])
    _same(ref, got)
