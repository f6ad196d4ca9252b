"""The 2-D updates with four cells of a row per thread against the oracle, bit for bit: rows of
every remainder by 4 and around a warp's 128 cells, every boundary condition, CPML layers (kappa
1 and not 1, overlapping ones too) that begin and end inside a group, materials with 0 to 5 poles
and Kerr, in the separate launches (a profiled run takes them at any size) and in a batch."""
import numpy as np
import pytest

import cases as C
import maxwellfdtd_b200 as M
from maxwellfdtd_b200 import _abi
from maxwellfdtd_b200.sources import comp_index, field_components

pytestmark = pytest.mark.gpu


def _model(nx, bc, kmax, poles):
    d = 50e-9
    g = C.grid2((nx, 13), d)
    at = (float(g.x[-1]), float(g.z[6]))
    src = [M.SoftSource(geometry=at, waveform=lambda x, z, t: 1e3 * C.pulse(t, t0=3e-15), component="Ez"),
           M.SoftSource(geometry=(float(g.x[0]), float(g.z[12])), waveform=lambda x, z, t: 5e2 * C.pulse(t, t0=2e-15), component="Ex")]
    chi = [M.LorentzSusceptibility(deps=0.5 + 0.2 * i, w0=(3 + i) * 1e15, delta=(1 + i) * 1e14) for i in range(poles)]
    mats = [M.Material(geometry=lambda x, z: x > g.x[-1] / 3, eps=2.25, mu=1.3, sigma=2e4),
            M.Material(geometry=lambda x, z: np.abs(z) < 130e-9, eps=3.0, chi=chi or None, chi3=1e-19 if poles % 2 == 0 else None)]
    cp = M.CPML(thickness=3 * d, kmax=kmax) if kmax else 0
    return M.Model(g, src, tmax=25.5 * M.model.time_step(g, 0.5), pml=(cp,) * 4, bc=bc, material=mats)


def _read(st, model):
    out = {c: st.read_field(comp_index(c)) for c in field_components(2, "Hy")}
    out["Sa"], out["E2"] = st.read_integral(_abi.MFD_INT_SA), st.read_integral(_abi.MFD_INT_E2)
    return out


CASES = [(nx, bc, kmax, poles) for nx, bc in zip((2, 3, 4, 5, 6, 7, 31, 33, 34, 127, 128, 129, 131),
                                                  ("periodic", "dirichlet", "neumann") * 5)
         for kmax, poles in ((0, 1), (1.0, 2), (4.0, 3))] + [(35, "periodic", 1.0, p) for p in (0, 5)]


@pytest.mark.parametrize("nx,bc,kmax,poles", CASES)
def test_rows_against_oracle(nx, bc, kmax, poles, oracle_lib, gpu_lib):
    if kmax and nx < 4:
        kmax = 0                      # no room for layers
    model = _model(nx, bc, kmax, poles)
    b, _ = model.build_desc(np.float32, None)
    ref = _abi.Stepper(oracle_lib, b, np.float32)
    ref.run(1, model.Nt)
    ref_out = _read(ref, model)
    ref.close()
    solo = _abi.Stepper(gpu_lib, b, np.float32)
    solo.set_profiling(True)          # separate launches
    solo.run(1, model.Nt)
    member = _abi.Stepper(gpu_lib, b, np.float32)
    batch = _abi.Batch(gpu_lib)
    batch.add(member, model.Nt)
    batch.run_all()
    for st in (solo, member):
        got = _read(st, model)
        bad = [k for k in ref_out if not np.array_equal(ref_out[k], got[k])]
        assert not bad, (bad, "solo" if st is solo else "batch")
    batch.close()
    solo.close()
    member.close()
    assert np.abs(ref_out["Ez"]).max() > 0
