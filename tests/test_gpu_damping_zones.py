"""Damping of rings that lie in both zones (a narrow disk: the inner zone ends
beyond the outer one's begin), against the oracle: both edges' damping applies to
such a ring in turn, inner edge first, whatever the kinds and however many blocks
share the ring (1024 cells each).  Both forms; the ring mean at either edge or at
both.

Bars: FP64 1e-13 (a sum of 2100 terms, an exponential and three operations),
FP32-mixed 1e-6 (the same to 2^-24)."""
import numpy as np
import pytest

from gpu_cases import initial_state, load, make_params
from golden_runner import EVOLVED, rel_linf

pytestmark = pytest.mark.gpu

REFERENCE, MEAN = 1, 3


@pytest.mark.parametrize("naz", [96, 1024, 1025, 2100])
@pytest.mark.parametrize("kinds", [(MEAN, REFERENCE), (REFERENCE, MEAN), (MEAN, MEAN),
                                   (REFERENCE, REFERENCE)])
def test_rings_in_both_zones(naz, kinds):
    from fargocpt_gb300.abi import params_from_dict
    from fargocpt_gb300.engine import Engine, grid_radii
    from oracle.oracle_py import OracleState

    params, d = make_params(12, naz, adiabatic=True, rmin=0.9, rmax=1.1,
                            damping_inner=[kinds[0]] * 4, damping_outer=[kinds[1]] * 4,
                            damping_inner_limit=1.15, damping_outer_limit=0.85)
    radii = grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"])
    st = initial_state(d, radii, seed=17, noise=0.1)
    reference = initial_state(d, radii, seed=18, noise=0.1)

    def run(backend):
        load(backend, st, [(0.0, 0.0, 1.0, 0.0, 0.0)])
        for f, a in reference.items():
            backend.set_field(f + "0", a)
        backend.apply_boundary_condition(0.0, 30.0, True)
        return {f: backend.get_field(f) for f in EVOLVED}

    want = run(OracleState(params, radii))
    # (the damping reaches the middle of the disk)
    assert not np.allclose(want["SIGMA"][6], st["SIGMA"][6], rtol=1e-2, atol=0)
    for precision, bar in ((0, 1e-13), (1, 1e-6)):
        got = run(Engine(params_from_dict(dict(d, precision=precision)), radii))
        for f in EVOLVED:
            assert rel_linf(got[f], want[f]) <= bar, (precision, f)
