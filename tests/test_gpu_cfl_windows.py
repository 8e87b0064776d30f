"""The float-pair CFL kernel (csrc/kernels_cfl.cu: 60 cells per warp and ring,
marches through the rings, an FP32 bound in front of the float-pair sums, the
ring means of v_phi by the ghost kernel or a kernel of their own) against the
oracle: the step and the derived quantities at the edges of windows and marches,
SN and TW, both equations of state, with and without fast transport, LeapFrog's
limits, and disks where the limit lies elsewhere than in a smooth one: v_phi that
crosses a power of two and zero within a ring, a v_r of exact zeros with one cell
that differs, the rings' shear.

Bars: on equal fields the step and the derived quantities 1e-12 (float pairs,
2^-45 relative per operation, are well inside); after a step 1e-9 (the fields agree
to 1e-10); the step formed by the call against the one formed by the kernel after
the transport, from the same fields, 1e-13."""
import math

import numpy as np
import pytest

from gpu_cases import initial_state, load, make_params
from golden_runner import rel_linf

pytestmark = pytest.mark.gpu

STAR = (0.0, 0.0, 1.0, 0.0, 0.0)
PLANET = (1.0, 0.05, 1e-3, 0.0, math.hypot(1.0, 0.05))


def pair(nrad, naz, change=None, **over):
    from fargocpt_gb300.engine import Engine, grid_radii
    from oracle.oracle_py import OracleState

    params, d = make_params(nrad, naz, **over)
    radii = grid_radii(d["radial_spacing"], d["rmin"], d["rmax"], d["nrad"])
    st = initial_state(d, radii, seed=23)
    if change:
        change(st)
    out = []
    for cls in (OracleState, Engine):
        b = cls(params, radii)
        load(b, st, [STAR, PLANET])
        out.append(b)
    return out


def check(o, g, adiabatic):
    dt = o.condition_cfl()
    assert g.condition_cfl() == pytest.approx(dt, rel=1e-12)
    fields = ["PRESSURE", "VISCOSITY"]
    if adiabatic:
        fields += ["SOUNDSPEED", "SCALE_HEIGHT", "TEMPERATURE"]
    for f in fields:
        assert rel_linf(g.get_field(f), o.get_field(f)) <= 1e-12, f
    return dt


@pytest.mark.parametrize("nrad,naz", [(6, 8), (8, 59), (9, 60), (7, 61), (40, 121), (700, 64)])
@pytest.mark.parametrize("adiabatic,art,over", [
    (True, 1, {}), (False, 1, {}), (True, 2, {}), (False, 2, dict(fast_transport=0)),
    (True, 1, dict(integrator=1, viscous_alpha=0.0, constant_viscosity=1e-4)),
])
def test_step_at_window_edges(nrad, naz, adiabatic, art, over):
    o, g = pair(nrad, naz, adiabatic=adiabatic, art_visc=art, **over)
    dt = check(o, g, adiabatic)
    for b in (o, g):
        b.apply_boundary_condition(0.0, 0.0, False)
        b.step_euler(0.2 * dt, 0.0)
    dt1 = g.condition_cfl()  # formed by the step
    assert dt1 == pytest.approx(o.condition_cfl(), rel=1e-9)
    g.set_field("V_RADIAL", g.get_field("V_RADIAL"))
    assert g.condition_cfl() == pytest.approx(dt1, rel=1e-13)  # formed by the call


def crossing(st):
    # v_phi around 1, with both signs and zeros in some rings
    rng = np.random.default_rng(3)
    v = st["V_AZIMUTHAL"]
    v[:] = 1.0 + 0.02 * rng.uniform(-1, 1, v.shape)
    v[5] -= 1.0
    v[6, ::2] = 0.0
    v[7] *= -1.0


def lone_radial(st):
    st["V_RADIAL"][:] = 0.0
    st["V_RADIAL"][9, 31] = 2.0


def sheared(st):
    # alternating ring speeds: the shear of neighbouring rings limits
    st["V_AZIMUTHAL"][:] *= 1.0 + 0.9 * (np.arange(len(st["V_AZIMUTHAL"])) % 2)[:, None]


@pytest.mark.parametrize("change", [crossing, lone_radial, sheared])
@pytest.mark.parametrize("naz", [90, 1031])
@pytest.mark.parametrize("art", [1, 2])
def test_step_of_other_limits(change, naz, art):
    o, g = pair(24, naz, change, adiabatic=True, art_visc=art)
    check(o, g, True)


@pytest.mark.parametrize("scale", [2.0 ** -46, 2.0 ** 100])
@pytest.mark.parametrize("art", [1, 2])
def test_step_near_the_ends_of_the_pairs_range(scale, art):
    """Sigma and energy near the smallest and the largest values a float pair holds
    (2^-74, 2^126), the limit in one cell's heating: the bound in front of the pairs,
    formed from truncated values, lets that cell through."""
    def scaled(st):
        for f in ("SIGMA", "ENERGY"):
            st[f] *= scale

    o, g = pair(24, 90, scaled, adiabatic=True, art_visc=art)
    heat = np.zeros((24, 90))
    cool = 0.125 * o.get_field("ENERGY")
    heat[9, 31] = 4.0e4 * cool[9, 31]
    for b in (o, g):
        b.set_field("QPLUS", heat)
        b.set_field("QMINUS", cool)
    dt = check(o, g, True)
    heat[9, 31] = 0.0
    o.set_field("QPLUS", heat)
    assert o.condition_cfl() > 1.5 * dt  # (the cell does limit)
