"""The double-precision constant division (two correction steps inside a band of magnitudes,
IEEE division outside) against the oracle's IEEE division: bit for bit, for fields in the middle
of the band, at both of its ends, below the normal range and near overflow; grids with layers
whose kappa is and is not 1, so that both divisor kinds occur."""
import numpy as np
import pytest

import cases as C
import maxwellfdtd_b200 as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kmax", [1.0, 4.0])
@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("amp", [0.0, 1e-318, 1e-296, 1e-271, 1e-262, 1.0, 1e264, 1e270, 1e290])
def test_double_division_magnitudes(amp, ndim, kmax, oracle_lib, gpu_lib):
    g = C._grid(ndim)
    src = M.SoftSource(geometry=C._plane(ndim, 0.0), waveform=lambda *a: amp * C.pulse(a[-1], t0=2e-15), component="Ex",
                       explicit=True)
    cp = M.CPML(thickness=150e-9, kmax=kmax)
    model = M.Model(g, src, tmax=30.5 * M.model.time_step(g, 0.5), pml=(cp,) * (2 * ndim))
    ref = C.run_all(model, oracle_lib, np.float64)
    got = C.run_all(model, gpu_lib, np.float64)
    assert set(ref) == set(got)
    bad = [k for k in ref if not np.array_equal(ref[k], got[k], equal_nan=True)]
    assert not bad, bad
    assert amp == 0.0 or np.abs(got["field/Ex"]).max() > 0
