"""The FP32-mixed form's substeps of four cells per thread (Quad in
csrc/fp32_device.cuh) against the oracle at the ring lengths where they can go
wrong: multiples of four (16-byte accesses, neighbours across lanes, blocks and
the ring's ends) and the lengths between (scalar accesses, fours cut short by the
ring's end), one and several blocks per ring; SN and TW, both equations of state,
single and batched.

Bars: the FP32 form rounds each operation to 6e-8; some twenty per step and field
over three steps, relative to each field's largest value, stay below 1e-5; v_r and
the fields formed from velocity differences, which are 1e-3 to 1e-2 of the
velocities they come from, below 1e-3.  A neighbour taken from the wrong cell is
off by the noise of the state, 2e-2 and more."""
import math

import numpy as np
import pytest

from gpu_cases import initial_state, load, make_params
from golden_runner import rel_linf

pytestmark = pytest.mark.gpu

BODIES = [(0.0, 0.0, 1.0, 0.0, 0.0), (1.0, 0.05, 1e-3, 0.0, math.hypot(1.0, 0.05))]
FINE = ["SIGMA", "V_AZIMUTHAL", "POTENTIAL"]
COARSE = ["V_RADIAL", "TAU_R_R", "TAU_PHI_PHI", "TAU_R_PHI"]


def step(b, st):
    load(b, st, BODIES)
    b.apply_boundary_condition(0.0, 0.0, False)
    t = 0.0
    for _ in range(3):
        dt = b.condition_cfl()
        b.step_euler(dt, t)
        t += dt
    return b


SHORT = [8, 9, 10, 11, 12, 126, 127, 128, 129]
LONG = [508, 511, 512, 513, 516, 1025]


# (TW with the short rings only: its viscosity, whose length is the larger cell side,
# is unstable on nine rings of the long ones, v_r grows 1e4-fold in a step)
@pytest.mark.parametrize("naz,adiabatic,art", [(n, True, 1) for n in SHORT + LONG] +
                         [(n, False, 2) for n in SHORT] + [(n, False, 1) for n in LONG])
def test_substeps_at_ring_lengths(naz, adiabatic, art):
    from fargocpt_gb300.abi import params_from_dict
    from fargocpt_gb300.batch import Batch
    from fargocpt_gb300.engine import Engine, grid_radii
    from oracle.oracle_py import OracleState

    params, d = make_params(9, naz, adiabatic=adiabatic, art_visc=art)
    p32 = params_from_dict(dict(d, precision=1))
    radii = grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"])
    st = initial_state(d, radii, seed=41, noise=2e-2)
    o = step(OracleState(params, radii), st)
    g = step(Engine(p32, radii), st)
    fine = FINE + (["ENERGY", "QMINUS"] if adiabatic else [])
    for f in fine:
        assert rel_linf(g.get_field(f), o.get_field(f)) <= 1e-5, f
    for f in COARSE:
        assert rel_linf(g.get_field(f), o.get_field(f)) <= 1e-3, f
    # a batch of this disk alone: the same bits
    b = Batch([p32], [radii])
    e = b.disks[0]
    load(e, st, BODIES)
    e.apply_boundary_condition(0.0, 0.0, False)
    t = np.zeros(1)
    for _ in range(3):
        dt = np.array([e.condition_cfl()])
        b.step(dt, t)
        t += dt
    for f in fine + COARSE:
        assert np.array_equal(e.get_field(f), g.get_field(f)), f
    b.close()


def sheared(st):
    # alternating ring speeds: the shear of neighbouring rings limits
    st["V_AZIMUTHAL"][:] *= 1.0 + 0.9 * (np.arange(len(st["V_AZIMUTHAL"])) % 2)[:, None]


@pytest.mark.parametrize("nrad,naz", [(6, 8), (9, 59), (9, 128), (40, 511), (7, 516), (300, 64)])
@pytest.mark.parametrize("change", [None, sheared])
@pytest.mark.parametrize("adiabatic,art", [(True, 1), (False, 2)])
def test_step_limit(nrad, naz, change, adiabatic, art):
    """The CFL step of the FP32-mixed form (cells, and the shear limit that the last
    ring to finish takes) against the oracle's to 1e-5, and in a batch bit for bit,
    for any tile and after the autotuner has run other states through it."""
    from fargocpt_gb300.abi import params_from_dict
    from fargocpt_gb300.batch import Batch
    from fargocpt_gb300.engine import Engine, grid_radii
    from oracle.oracle_py import OracleState

    params, d = make_params(nrad, naz, adiabatic=adiabatic, art_visc=art)
    p32 = params_from_dict(dict(d, precision=1))
    radii = grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"])
    st = initial_state(d, radii, seed=43, noise=2e-2)
    if change:
        change(st)
    o, g, b = OracleState(params, radii), Engine(p32, radii), Batch([p32], [radii])
    for x in (o, g, b.disks[0]):
        load(x, st, BODIES)
    dt = g.condition_cfl()
    assert dt == pytest.approx(o.condition_cfl(), rel=1e-5)
    assert b.disks[0].condition_cfl() == dt
    b.autotune(reps=1)
    assert b.disks[0].condition_cfl() == dt
    g.step_euler(0.1 * dt, 0.0)
    b.step(np.array([0.1 * dt]), np.zeros(1))
    assert b.disks[0].condition_cfl() == g.condition_cfl()
    b.close()
