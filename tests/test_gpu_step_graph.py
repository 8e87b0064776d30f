"""A step captured from the engine's stream into a CUDA graph and launched again
and again is that many steps: it reads and writes the same buffers every time, and
the CFL step that follows is the last launch's.  Against the same steps called one
by one: equal bits, with every number of passes the gas kick can take (energy
equation or not, artificial viscosity, StabilizeViscosity's own viscous kernel)."""
import math

import numpy as np
import pytest

from gpu_cases import initial_state, load, make_params
from golden_runner import EVOLVED

pytestmark = pytest.mark.gpu

BODIES = [(0.0, 0.0, 1.0, 0.0, 0.0), (1.0, 0.05, 1e-3, 0.0, math.hypot(1.0, 0.05))]


@pytest.mark.parametrize("adiabatic,over", [
    (True, {}), (False, {}), (False, dict(art_visc=0)), (True, dict(art_visc=2)),
    (True, dict(stabilize_viscosity=1)), (False, dict(stabilize_viscosity=1, art_visc=0)),
    (True, dict(stabilize_viscosity=2)), (True, dict(precision=1)), (False, dict(precision=1)),
])
@pytest.mark.parametrize("arith", ["pair", "fp64"])
def test_replayed_step(adiabatic, over, arith, monkeypatch):
    torch = pytest.importorskip("torch")
    from fargocpt_gb300.engine import Engine, grid_radii

    monkeypatch.setenv("FARGO_GB300_FP64_ARITH", arith)
    params, d = make_params(20, 62, adiabatic=adiabatic, **over)
    radii = grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"])
    st = initial_state(d, radii, seed=41)
    steps, out = 3, []
    for replay in (False, True):
        g = Engine(params, radii)
        load(g, st, BODIES)
        g.apply_boundary_condition(0.0, 0.0, False)
        dt = 0.2 * g.condition_cfl()
        if replay:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(g.stream)):
                g.step_euler(dt, 0.0)
        dts = []
        for _ in range(steps):
            if replay:
                with torch.cuda.stream(torch.cuda.ExternalStream(g.stream)):
                    graph.replay()
            else:
                g.step_euler(dt, 0.0)
            dts.append(g.condition_cfl())
        out.append((dts, {f: g.get_field(f) for f in EVOLVED}))
    assert out[0][0] == out[1][0]
    assert len(set(out[0][0])) == steps  # (the CFL step differs from step to step)
    for f in EVOLVED:
        assert np.array_equal(out[0][1][f], out[1][1][f]), f


def test_state_read_and_set_between_steps():
    """SIGMA and ENERGY read, changed and set back between single steps: as in a run
    that steps on without."""
    from fargocpt_gb300.engine import Engine, grid_radii

    params, d = make_params(20, 62, adiabatic=True)
    radii = grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"])
    st = initial_state(d, radii, seed=43)
    out = []
    for touch in (False, True):
        g = Engine(params, radii)
        load(g, st, BODIES)
        dt = 0.2 * g.condition_cfl()
        for _ in range(3):
            if touch:
                for f in ("SIGMA", "ENERGY"):
                    a = g.get_field(f)
                    g.set_field(f, 2.0 * a)
                    assert np.array_equal(g.get_field(f), 2.0 * a)
                    g.set_field(f, a)
            g.step_euler(dt, 0.0)
        out.append({f: g.get_field(f) for f in EVOLVED})
    for f in EVOLVED:
        assert np.array_equal(out[0][f], out[1][f]), f
