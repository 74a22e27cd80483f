"""The walk with one warp per group (lbvh.cu:k_walk), which serves trees beyond
the limits of the team walk, on small trees: against the oracle's sums over the
same lists, and against the team walk. Sizes, tolerances and their reasons as
test_team_walk_gpu.py, with every force law, unsoftened as well, the kick and
drift fused into the walk against single steps, and the stack's overflow."""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, MIXED, NEWTON, PN1, PN2, PN25, SOLVER_LBVH, AsterError, Context, Params
from conftest import rel_l2

pytestmark = pytest.mark.gpu
EVERY = NEWTON | PN1 | PN2 | PN25


@pytest.fixture(scope="module")
def one(request):
    """A context whose trees all take the one-warp walk."""
    mp = pytest.MonkeyPatch()
    mp.setenv("ASTER_WALK_TEAM_LIMIT", "0")
    c = Context(0)
    mp.undo()
    yield c
    c.close()


def _bodies(n, seed):
    pos, vel, m = gen.plummer(n, seed + n, masses="lognormal")
    if n > 40:
        m[7:30] = 0.0  # massless bodies among the others
    return pos, vel, m


def _close(acc, ref, prec, mixed_tol):
    if prec == FP64:
        assert rel_l2(acc, ref) < 1e-12
    else:
        assert np.abs(acc - ref).max() < mixed_tol * np.abs(ref).max()


@pytest.mark.parametrize("n", [1, 2, 32, 33, 48, 49, 64, 65, 129, 700, 3001])
@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("eps2,theta", [(1e-4, 0.5), (0.0, 0.5), (1e-4, 0.05)])
def test_newton_matches_oracle(one, orc, n, prec, eps2, theta):
    pos, vel, m = _bodies(n, 900)
    o = orc.lbvh(pos, m, theta)
    ref, cnt = orc.lbvh_forces(o, o["perm"], pos, 1.0, eps2)
    one.upload(pos, vel, m)
    acc, c = one.lbvh_forces(Params(eps2=eps2, theta=theta), prec, list_counts=True)
    np.testing.assert_array_equal(c, cnt)
    if n == 1:
        assert np.all(acc == 0.0)
    else:
        _close(acc, ref, prec, 2e-4)


@pytest.mark.parametrize("n", [1, 2, 33, 49, 64, 65, 129, 193, 700, 3001])
@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("law", [NEWTON | PN1, EVERY])
@pytest.mark.parametrize("eps2", [1e-4, 0.0])
def test_post_newton_matches_oracle(one, ctx, orc, n, prec, law, eps2):
    pos, vel, m = _bodies(n, 950)
    vel = vel * 5.0
    o = orc.lbvh(pos, m, 0.5)
    ref, cnt = orc.lbvh_forces_pn(o, o["perm"], pos, vel, 1.0, eps2, 0.1, law)
    p = Params(eps2=eps2, theta=0.5, c=10.0, force_law=law)
    one.upload(pos, vel, m)
    acc, c = one.lbvh_forces(p, prec, list_counts=True)
    np.testing.assert_array_equal(c, cnt)
    if n == 1:
        assert np.all(acc == 0.0)
    elif eps2 > 0.0 or prec == FP64:
        _close(acc, ref, prec, 3.3e-4)
    else:
        # unsoftened, mixed: the closest pair's terms go as the fifth power of a separation that FP32 may resolve to a
        # few parts in 1e3 only; the team walk forms the same terms in another order of addition
        ctx.upload(pos, vel, m)
        team = ctx.lbvh_forces(p, prec)
        assert np.abs(acc - team).max() < 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("scale", [1e-105, 1e105])
def test_extreme_scales(one, scale):
    pos, _, m = gen.plummer(1500, 31)
    k = 2.0 ** round(np.log2(scale))
    one.upload(pos, None, m)
    ref = one.lbvh_forces(Params(theta=0.0), FP64)
    one.upload(pos * k, None, m * k)
    acc = one.lbvh_forces(Params(theta=0.0), FP64)
    assert np.isfinite(acc).all()
    assert rel_l2(acc * k, ref) < 1e-12


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("law", [NEWTON, NEWTON | PN1, EVERY])
def test_fused_steps_repeat_single_ones(one, prec, law):
    """Runs whose walks apply the next kick and drift, in one call and cut into shorter ones: the same bits; and the
    team walk's states, apart by the order of addition (FP64) or by FP32's resolution of it (mixed)."""
    pos, vel, m = gen.plummer(5001, 6, masses="lognormal")
    p = Params(eps2=2.5e-5, dt=5e-4, c=100.0, force_law=law)
    out = []
    for split in ((6,), (1, 2, 3), (1,) * 6):
        one.upload(pos, vel, m)
        for k in split:
            one.kdk_steps(p, k, SOLVER_LBVH, prec)
        out.append(one.download())
    for o in out[1:]:
        for a, b in zip(out[0], o):
            np.testing.assert_array_equal(a, b)
    with Context(0) as c:
        c.upload(pos, vel, m)
        c.kdk_steps(p, 6, SOLVER_LBVH, prec)
        for a, b in zip(out[0], c.download()):
            assert rel_l2(a, b) < (1e-12 if prec == FP64 else 1e-6)


def test_stack_overflow_is_reported(monkeypatch):
    monkeypatch.setenv("ASTER_WALK_STACK_LIMIT", "64")
    monkeypatch.setenv("ASTER_WALK_TEAM_LIMIT", "0")
    pos, vel, m = gen.plummer(20000, 5)
    with Context(0) as c:
        c.upload(pos, vel, m)
        for prec in (MIXED, FP64):
            with pytest.raises(AsterError) as e:
                c.lbvh_forces(Params(theta=0.1, eps2=1e-4), prec)
            assert e.value.status == 5
        acc = c.lbvh_forces(Params(theta=3.0, eps2=1e-4), MIXED)  # shallow stacks: the context is usable
        assert np.isfinite(acc).all()


@pytest.mark.parametrize("n", [120001, 200000])
def test_large_fp64_trees_match_the_team(n, monkeypatch):
    """FP64 forces of the largest trees of the team walk, by both walks: 1e-12."""
    pos, vel, m = gen.plummer(n, 60, masses="lognormal")
    out = []
    for lim in ("0", str(n)):
        monkeypatch.setenv("ASTER_WALK_TEAM_LIMIT", lim)
        with Context(0) as c:
            c.upload(pos, vel, m)
            out.append(c.lbvh_forces(Params(eps2=2.5e-5, theta=0.7), FP64, list_counts=True))
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert not np.array_equal(out[0][0], out[1][0])  # (two walks)
    assert rel_l2(out[0][0], out[1][0]) < 1e-12
