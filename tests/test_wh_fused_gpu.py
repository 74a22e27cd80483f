"""Wisdom-Holman steps whose interaction is formed inside the drift kernel (at
most 64 massive bodies, FP64) against the oracle, at the limit and past it, and
the shorter Kepler iteration on eccentric orbits and long steps. Tolerances as
test_wh_gpu.py: 1e-11 relative L2."""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, Params
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planets,particles", [(1, 0), (1, 1), (8, 255), (8, 256), (62, 700), (63, 700), (64, 700)])
@pytest.mark.parametrize("eps2", [0.0, 1e-6])
def test_fused_interaction_matches_oracle(ctx, orc, planets, particles, eps2):
    pos, vel, m = gen.planetary_system(planets, particles, 31 + planets, planet_mass=(1e-7, 1e-5))
    p = Params(G=1.0, eps2=eps2, dt=0.03)
    ctx.upload(pos, vel, m)
    for k in (1, 2, 7):
        ctx.wh_steps(p, k, FP64)
    gp, gv, _ = ctx.download()
    op, ov = pos, vel
    for k in (1, 2, 7):
        op, ov = orc.wh(op, ov, m, p.dt, k, eps2=eps2)
    assert rel_l2(gp, op) < 1e-11 and rel_l2(gv, ov) < 1e-11


@pytest.mark.parametrize("dt", [1e-4, 0.02, 0.5, 3.0])
def test_kepler_drift_on_conics(ctx, orc, dt):
    """Elliptic, near-parabolic and hyperbolic orbits through steps short and long against them."""
    pos, vel, m, e = gen.kepler_orbits(3000, 9)
    p = Params(G=1.0, dt=dt)
    ctx.upload(pos, vel, m)
    ctx.wh_steps(p, 3, FP64)
    gp, gv, _ = ctx.download()
    # (massless bodies only: drifts compose, and the oracle takes the longest steps in thirty parts)
    op, ov = orc.wh(pos, vel, m, dt, 3) if dt < 1.0 else orc.wh(pos, vel, m, dt / 30, 90)
    ep = np.linalg.norm(gp[1:] - op[1:], axis=1) / np.linalg.norm(op[1:], axis=1)
    near = (e > 0.96) & (e < 1.04)
    assert ep[~near].max() < 1e-11 and ep[near].max() < 1e-9
