"""The team walk (a block of warps per group, lbvh.cu:k_walk_team) against the
oracle's walk over the same lists: list lengths equal, forces FP64 1e-12
(relative L2) as for the one-warp walk, mixed within FP32's resolution of the
groups. Sizes: one body, groups at the
one- and two-body-per-lane limits (32, 33, 48, 49, 64), lists shorter and
longer than a batch (the last chunk full, odd and empty), and both sides of the
sizes at which either walk takes over.
"""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, MIXED, NEWTON, PN1, PN2, PN25, SOLVER_LBVH, AsterError, Context, Params
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _check(ctx, orc, n, prec, eps2, theta):
    pos, vel, m = gen.plummer(n, 900 + n, masses="lognormal")
    if n > 40:
        m[7:30] = 0.0  # massless bodies among the others
    o = orc.lbvh(pos, m, theta)
    ref, cnt = orc.lbvh_forces(o, o["perm"], pos, 1.0, eps2)
    ctx.upload(pos, vel, m)
    acc, c = ctx.lbvh_forces(Params(eps2=eps2, theta=theta), prec, list_counts=True)
    np.testing.assert_array_equal(c, cnt)
    if n == 1:
        assert np.all(acc == 0.0)
    elif prec == FP64:
        assert rel_l2(acc, ref) < 1e-12
    else:
        # FP32 positions relative to a group's centre resolve a close pair to 2^-24 of the group's extent over its
        # separation, three times that in the force: 3 * 2^-24 * 20 / 0.02 for the widest groups and closest pairs here
        assert np.abs(acc - ref).max() < 2e-4 * np.abs(ref).max()


@pytest.mark.parametrize("n", [1, 2, 32, 33, 48, 49, 64, 65, 129, 700, 3001])
@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("eps2,theta", [(1e-4, 0.5), (0.0, 0.5), (1e-4, 0.05)])
def test_team_walk_matches_oracle(ctx, orc, n, prec, eps2, theta):
    _check(ctx, orc, n, prec, eps2, theta)


# a post-Newtonian batch: 3 chunks of 64 entries mixed, 4 of 64 FP64, velocities fetched by the evaluating warps
@pytest.mark.parametrize("n", [1, 2, 33, 49, 64, 65, 129, 193, 257, 700, 3001])
@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("law", [NEWTON | PN1, NEWTON | PN1 | PN2 | PN25])
def test_pn_team_walk_matches_oracle(ctx, orc, n, prec, law):
    pos, vel, m = gen.plummer(n, 950 + n, masses="lognormal")
    vel = vel * 5.0
    if n > 40:
        m[7:30] = 0.0
    o = orc.lbvh(pos, m, 0.5)
    ref, cnt = orc.lbvh_forces_pn(o, o["perm"], pos, vel, 1.0, 1e-4, 0.1, law)
    ctx.upload(pos, vel, m)
    acc, c = ctx.lbvh_forces(Params(eps2=1e-4, theta=0.5, c=10.0, force_law=law), prec, list_counts=True)
    np.testing.assert_array_equal(c, cnt)
    if n == 1:
        assert np.all(acc == 0.0)
    elif prec == FP64:
        assert rel_l2(acc, ref) < 1e-12
    else:  # as _check, up to the fifth power of the separation in place of the third
        assert np.abs(acc - ref).max() < 3.3e-4 * np.abs(ref).max()


@pytest.mark.parametrize("n", [120000, 120001, 200000, 200001])
def test_either_side_of_the_team_limits(ctx, n):
    """Mixed and FP64 walks of one tree, at the sizes where one of them changes from the team to one warp per group:
    the same lists, forces 1e-6 apart (relative L2), and the FP64 sums of all bodies 1e-12 from the direct sum of a
    theta = 0 tree for a sample would be too long: the lists fix the terms, the precisions their sums."""
    pos, vel, m = gen.plummer(n, 900 + n, masses="lognormal")
    ctx.upload(pos, vel, m)
    p = Params(eps2=2.5e-5, theta=0.5)
    a, ca = ctx.lbvh_forces(p, MIXED, list_counts=True)
    b, cb = ctx.lbvh_forces(p, FP64, list_counts=True)
    np.testing.assert_array_equal(ca, cb)
    assert rel_l2(a, b) < 1e-6


@pytest.mark.parametrize("scale", [1e-105, 1e105])
def test_fp64_walk_at_extreme_scales(ctx, scale):
    """Squared distances outside the range of the inverse cube's series step: with masses scaled as the coordinates,
    accelerations go as their inverse (a power of two, so the trees and lists are the same)."""
    pos, _, m = gen.plummer(1500, 31)
    k = 2.0 ** round(np.log2(scale))
    ctx.upload(pos, None, m)
    ref = ctx.lbvh_forces(Params(theta=0.0), FP64)
    ctx.upload(pos * k, None, m * k)
    acc = ctx.lbvh_forces(Params(theta=0.0), FP64)
    assert np.isfinite(acc).all()
    assert rel_l2(acc * k, ref) < 1e-12


def test_team_stack_overflow_is_reported(monkeypatch):
    monkeypatch.setenv("ASTER_WALK_STACK_LIMIT", "64")
    pos, vel, m = gen.plummer(20000, 5)
    with Context(0) as c:
        c.upload(pos, vel, m)
        for prec in (MIXED, FP64):
            with pytest.raises(AsterError) as e:
                c.lbvh_forces(Params(theta=0.1, eps2=1e-4), prec)
            assert e.value.status == 5
        acc = c.lbvh_forces(Params(theta=3.0, eps2=1e-4), MIXED)  # shallow stacks: the context is usable
        assert np.isfinite(acc).all()


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_team_steps_repeat_exactly(ctx, prec):
    pos, vel, m = gen.plummer(15001, 6, masses="lognormal")
    p = Params(eps2=2.5e-5, dt=5e-4)
    out = []
    for split in ((6,), (1, 2, 3)):
        ctx.upload(pos, vel, m)
        for k in split:
            ctx.kdk_steps(p, k, SOLVER_LBVH, prec)
        out.append(ctx.download())
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
