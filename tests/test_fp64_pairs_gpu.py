"""FP64 all-pairs with every unordered pair formed once (allpairs_sym.cu) and
its inverse distances (fp64_pair.cuh).

Tolerances: against the oracle 1e-12 relative L2, as every FP64 all-pairs
check; one pair's acceleration to 8 ulp (1.8e-15): r^-3 carries the roundings
of r^2 (3/2 of at most 2 ulp), of the cube and its series step (2 ulp) and two
products, and each separation is exact to one rounding of its own.
"""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, NEWTON, PN1, SOLVER_ALLPAIRS, Params
from conftest import rel_l2

pytestmark = pytest.mark.gpu


# the smallest size of the path and the one below, tile and set edges (64, 128, 256 bodies), the small-tile limit,
# sizes with more than one set per tile (128 slots of 128 or 256 bodies end at 16384 and 32768)
@pytest.mark.parametrize("n", [127, 128, 129, 191, 193, 3999, 4000, 4097, 16385, 33001])
@pytest.mark.parametrize("law,eps2", [(NEWTON, 1e-4), (NEWTON, 0.0), (NEWTON | PN1, 0.0), (NEWTON | PN1, 1e-4)])
def test_symmetric_pairs_match_oracle(ctx, orc, n, law, eps2):
    pos, vel, m = gen.plummer(n, 300 + n, masses="lognormal")
    vel = vel * 5.0
    pos[-1] = pos[n // 2]  # two bodies in one place: no pull without softening
    vel[-1] = vel[n // 2]
    p = Params(eps2=eps2, c=20.0, force_law=law)
    ctx.upload(pos, vel, m)
    acc = ctx.allpairs(p, FP64)
    if n <= 4097:
        ref = orc.allpairs(pos, m, 1.0, eps2, vel=vel, inv_c=1.0 / 20.0, pn=law)
        # (without softening the oracle, as the reference, has no value for the two bodies in one place)
        ok = np.isfinite(ref).all(1)
        assert ok.sum() >= n - (2 if eps2 == 0.0 else 0)
        assert rel_l2(acc[ok], ref[ok]) < 1e-12
    # and the directed kernel (an explicit target list), body by body
    t = np.unique(np.r_[0, 1, 63, 64, 126, n // 2, n - 2, n - 1, np.arange(0, n, 97)])
    d = ctx.allpairs_targets(p, t, FP64)
    scale = np.linalg.norm(d, axis=1).max()
    assert np.abs(acc[t] - d).max() < 1e-12 * scale


def test_large_tiles_match_directed_kernel(ctx):
    """140,001 bodies: tiles of two source parts; sampled targets against the directed kernel."""
    pos, vel, m = gen.exponential_disk(140001, 7)
    p = Params(eps2=4e-6)
    ctx.upload(pos, vel, m)
    acc = ctx.allpairs(p, FP64)
    t = np.arange(0, 140001, 1111)
    assert rel_l2(acc[t], ctx.allpairs_targets(p, t, FP64)) < 1e-12


def test_one_pair_to_a_few_ulp(ctx):
    """A unit mass (the last body, so that every body counts as a source) and 600 massless bodies at distances from
    1e-3 to 1e3: each acceleration against extended precision."""
    rng = np.random.default_rng(5)
    u = rng.normal(size=(601, 3))
    pos = u / np.linalg.norm(u, axis=1)[:, None] * np.exp(rng.uniform(np.log(1e-3), np.log(1e3), 601))[:, None]
    pos[-1] = 0.0
    m = np.zeros(601)
    m[-1] = 1.0
    ctx.upload(pos, None, m)
    acc = ctx.allpairs(Params(), FP64)[:-1]
    x = pos[:-1].astype(np.longdouble)
    r2 = (x * x).sum(1)
    ref = -x / (r2 * np.sqrt(r2))[:, None]
    assert float((np.abs(acc - ref) / np.abs(ref)).max()) < 1.8e-15


@pytest.mark.parametrize("scale", [1e-105, 1e-60, 1e60, 1e105])
def test_extreme_scales(ctx, scale):
    """Coordinates whose squared distances leave the series step's range (and ones that stay inside), against the same
    system at unit scale: with masses scaled as the coordinates, accelerations go as their inverse."""
    pos, _, m = gen.plummer(700, 11)
    ctx.upload(pos, None, m)
    ref = ctx.allpairs(Params(), FP64)
    k = 2.0 ** round(np.log2(scale))  # a power of two: the scaled problem has the same roundings
    ctx.upload(pos * k, None, m * k)
    acc = ctx.allpairs(Params(), FP64)
    assert np.isfinite(acc).all()
    assert rel_l2(acc * k, ref) < 1e-12


def test_repeated_evaluations_are_identical(ctx):
    pos, vel, m = gen.plummer(9001, 12)
    p = Params(eps2=1e-4)
    ctx.upload(pos, vel, m)
    a = ctx.allpairs(p, FP64)
    np.testing.assert_array_equal(a, ctx.allpairs(p, FP64))
    ctx.upload(pos, vel, m)
    ctx.kdk_steps(p, 0, SOLVER_ALLPAIRS, FP64)
    np.testing.assert_array_equal(a, ctx.download()[2])
