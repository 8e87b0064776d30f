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


@pytest.mark.parametrize("naz", [8, 59, 257])
@pytest.mark.parametrize("mean", [0, 1])
def test_force_without_smoothing(naz, mean):
    """ThicknessSmoothing 0: the force on the central object, at the origin, where
    only a cell's own distance keeps the inverse cube finite, also in the lane of
    an odd ring that lacks its second cell.  Bars, of the sum of the terms'
    magnitudes (a smooth disk's cancel to a thousandth of it): 1e-12 and 1e-6,
    some ten roundings of a pair (2^-46) and of a float (2^-24)."""
    from fargocpt_gb300.abi import params_from_dict
    from fargocpt_gb300.engine import Engine, grid_radii
    from oracle.oracle_py import OracleState

    params, d = make_params(9, naz, adiabatic=True, thickness_smoothing=0.0,
                            correct_disk_selfgravity=mean)
    radii = np.asarray(grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"]))
    st = initial_state(d, radii, seed=5, noise=0.2)
    bodies = [STAR, (0.1, 0.05, 1e-3, 0.0, math.hypot(0.1, 0.05))]
    o = OracleState(params, radii)
    load(o, st, bodies)
    want = np.array([o.disk_on_planet_accel(k) for k in range(2)])
    lo, hi = radii[:9, None], radii[1:10, None]
    mid, phi = 2 / 3 * (hi ** 3 - lo ** 3) / (hi ** 2 - lo ** 2), 2 * np.pi * np.arange(naz) / naz
    term = (np.pi / naz * (hi ** 2 - lo ** 2) * st["SIGMA"])[1:-1]
    size = np.array([(term / np.abs(mid * np.exp(1j * phi) - complex(x, y))[1:-1] ** 2).sum()
                     for x, y, *_ in bodies])
    for precision, bar in ((0, 1e-12), (1, 1e-6)):
        g = Engine(params_from_dict(dict(d, precision=precision)), radii)
        load(g, st, bodies)
        got = np.array(g.disk_on_nbody_accel(2)).reshape(want.shape)
        err = np.hypot(*(got - want).T) / size
        assert np.all(err <= bar), (precision, err)
