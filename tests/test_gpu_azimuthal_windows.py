"""The float-pair azimuthal pass's windows (csrc/kernels_azimuthal.cu: 128
cells per warp, the inner 120 written, four per lane) against the oracle at
the ring lengths where they can go wrong: the shortest ring (several turns of
it in one window), one window short of, exactly and past 120 cells, one whole
warp, two windows and their remainders, lengths that are and are not whole
lanes (aligned and single loads); both limiters, FARGO and standard transport,
with and without the energy equation.  Bar: the FP64 form's relative
L-infinity of 1e-10 per evolved field.  The FP32-mixed form's window pass
(azimuthal_window, csrc/fp32_device.cuh) at the same lengths against its
strided ring kernel, whose arithmetic per cell is the same: equal bits."""
import numpy as np
import pytest

from gpu_cases import initial_state, load, make_params
from golden_runner import EVOLVED, rel_linf
from test_gpu_vs_oracle import TOL, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("naz", [8, 11, 116, 119, 120, 121, 124, 128, 239, 240, 243, 8192])
@pytest.mark.parametrize("adiabatic,mc,fargo", [(True, 0, 1), (False, 1, 1), (True, 1, 0)])
def test_window_edges(naz, adiabatic, mc, fargo):
    params, d = make_params(8, naz, adiabatic=adiabatic, flux_limiter=mc, fast_transport=fargo)
    (o, _), (g, _) = run_both(params, d, steps=3, planet=False)
    for f in EVOLVED:
        assert rel_linf(g.get_field(f), o.get_field(f)) <= TOL, f


@pytest.mark.parametrize("naz", [8, 11, 116, 119, 120, 121, 124, 128, 239, 240, 243, 6144])
@pytest.mark.parametrize("adiabatic,mc,fargo", [(True, 0, 1), (False, 1, 1), (True, 1, 0)])
def test_fp32_windows_match_the_ring_kernel(naz, adiabatic, mc, fargo, monkeypatch):
    from fargocpt_gb300.engine import Engine, grid_radii

    params, d = make_params(8, naz, adiabatic=adiabatic, precision=1, flux_limiter=mc,
                            fast_transport=fargo)
    radii = grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"])
    st = initial_state(d, radii, seed=5)
    out = []
    for variant in ("strided", None):
        if variant:
            monkeypatch.setenv("FARGO_GB300_AZIMUTHAL", variant)
        else:
            monkeypatch.delenv("FARGO_GB300_AZIMUTHAL", raising=False)
        e = Engine(params, radii)
        load(e, st, [(0.0, 0.0, 1.0, 0.0, 0.0)])
        t = 0.0
        for _ in range(4):
            dt = e.condition_cfl()
            e.step_euler(dt, t)
            t += dt
        out.append({f: e.get_field(f) for f in EVOLVED})
        e.close()
    for f in EVOLVED:
        assert np.array_equal(out[0][f], out[1][f]), f
