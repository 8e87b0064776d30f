"""The float-pair gas kick's marching windows (csrc/kernels_kick.cu: 64 cells
per warp, the inner 60 written, two per lane; marches of 1 to 16 rings) against
the oracle at the ring lengths and ring counts where they can go wrong: the
shortest ring, one cell short of, exactly and past a window, odd lengths
(single loads), several windows; few rings, ring counts that leave a short last
march.  SN and TW artificial viscosity, both equations of state, the
potential with Klahr-smoothed planets and a rotating frame, and a central
object off the origin (the kernels of the general potential).  Bar: the FP64
form's relative L-infinity of 1e-10 per evolved field; the intermediate fields
they leave (potential, artificial pressures, stress tensor) to 1e-9."""
import math

import pytest

from gpu_cases import initial_state, load, make_params
from golden_runner import EVOLVED, rel_linf
from test_gpu_vs_oracle import TOL

pytestmark = pytest.mark.gpu

PLANET = (1.0, 0.05, 1e-3, 0.0, math.hypot(1.0, 0.05))
KLAHR = (0.7, -0.9, 5e-4, 0.08, math.hypot(0.7, 0.9))


def run(nrad, naz, bodies, omega=0.0, steps=3, **over):
    from fargocpt_gb300.engine import Engine, grid_radii
    from oracle.oracle_py import OracleState

    params, d = make_params(nrad, naz, **over)
    radii = grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"])
    st = initial_state(d, radii, seed=17)
    out = []
    for cls in (OracleState, Engine):
        b = cls(params, radii)
        load(b, st, bodies)
        b.set_bodies(bodies, 1e-4, -2e-4, omega)
        b.apply_boundary_condition(0.0, 0.0, False)
        t = 0.0
        for _ in range(steps):
            dt = b.condition_cfl()
            b.step_euler(dt, t)
            t += dt
        out.append(b)
    return out


# (2300 rings of 64 cells, for the longest marches' remainders, with SN only: TW's
# viscosity, whose length is the larger cell side, is unstable on such cells, v_r
# grows 1e5-fold in three steps)
@pytest.mark.parametrize("nrad,naz,adiabatic,art",
                         [(n, z, a, v) for n, z in ((8, 8), (8, 59), (9, 60), (7, 61), (6, 62),
                                                    (11, 120), (40, 121))
                          for a, v in ((True, 1), (False, 2), (True, 2), (False, 1))] +
                         [(2300, 64, True, 1), (2300, 64, False, 1)])
def test_window_and_march_edges(nrad, naz, adiabatic, art):
    o, g = run(nrad, naz, [(0.0, 0.0, 1.0, 0.0, 0.0), PLANET], adiabatic=adiabatic, art_visc=art)
    for f in EVOLVED:
        assert rel_linf(g.get_field(f), o.get_field(f)) <= TOL, f
    fields = ["POTENTIAL", "Q_R", "Q_PHI", "DIV_V", "TAU_R_R", "TAU_PHI_PHI", "TAU_R_PHI"]
    for f in fields:
        assert rel_linf(g.get_field(f), o.get_field(f)) <= 1e-9, f


@pytest.mark.parametrize("star", [(0.0, 0.0, 1.0, 0.0, 0.0), (1e-3, -2e-3, 1.0, 0.0, 2.2e-3)])
@pytest.mark.parametrize("naz", [96, 127])
def test_potential_options(star, naz):
    o, g = run(24, naz, [star, PLANET, KLAHR], omega=0.3, adiabatic=True)
    for f in EVOLVED:
        assert rel_linf(g.get_field(f), o.get_field(f)) <= TOL, f
    assert rel_linf(g.get_field("POTENTIAL"), o.get_field("POTENTIAL")) <= 1e-12
