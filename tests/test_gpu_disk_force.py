"""The disk's force on the bodies (csrc/kernels_force.cu and the FP32-mixed
form's in csrc/kernels_fp32.cu: two adjacent cells per lane, 256 cells per block
and pass, four bodies per pass) against the oracle at ring lengths where a lane
lacks its second cell, a block its last lanes or a pass its full width; one to
five bodies, one of them with Klahr's smoothing over several cells, with and
without the ring mean removed.

Bars, of the force's magnitude: the FP64 form 1e-10 (pairs carry 2^-46 of each
term, the terms cancel to a few percent of their sum at the least), the
FP32-mixed form 1e-5 (terms rounded to 2^-24)."""
import math

import numpy as np
import pytest

from gpu_cases import initial_state, load, make_params

pytestmark = pytest.mark.gpu

STAR = (0.0, 0.0, 1.0, 0.0, 0.0)
BODIES = [STAR] + [(x, y, 1e-4, rsm, math.hypot(x, y))
                   for x, y, rsm in ((1.0, 0.05, 0.0), (-0.6, 0.8, 0.3), (0.2, -1.9, 0.0),
                                     (0.5, 0.1, 0.0))]


@pytest.mark.parametrize("nrad,naz", [(6, 8), (6, 59), (9, 255), (9, 256), (8, 257), (12, 514),
                                      (7, 1031)])
@pytest.mark.parametrize("nbodies,mean", [(1, 1), (2, 0), (4, 1), (5, 1)])
def test_force_at_block_edges(nrad, naz, nbodies, mean):
    from fargocpt_gb300.abi import params_from_dict
    from fargocpt_gb300.engine import Engine, grid_radii
    from oracle.oracle_py import OracleState

    params, d = make_params(nrad, naz, adiabatic=True, correct_disk_selfgravity=mean)
    radii = grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"])
    st = initial_state(d, radii, seed=31, noise=0.2)
    o = OracleState(params, radii)
    load(o, st, BODIES[:nbodies])
    want = np.array([o.disk_on_planet_accel(k) for k in range(nbodies)])
    size = np.hypot(want[:, 0], want[:, 1])
    for precision, bar in ((0, 1e-10), (1, 1e-5)):
        g = Engine(params_from_dict(dict(d, precision=precision)), radii)
        load(g, st, BODIES[:nbodies])
        got = np.array(g.disk_on_nbody_accel(nbodies)).reshape(want.shape)
        err = np.hypot(*(got - want).T) / size
        assert np.all(err <= bar), (precision, err)
