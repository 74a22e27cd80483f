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
from aster_b200.api import FP64, MIXED, NEWTON, PN1, PN2, PN25, SOLVER_ALLPAIRS, Params
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


@pytest.mark.parametrize("n", [1, 2, 127, 129, 256, 257, 7999, 8000, 8193])
@pytest.mark.parametrize("ref_form", [False, True])
@pytest.mark.parametrize("eps2", [0.0, 1e-4])
def test_energy_of_every_pair_once(ctx, n, ref_form, eps2):
    """Block and slice edges of the energy sum (2 and 4 bodies per thread), 1e-12 against numpy's sum over i < j."""
    pos, vel, m = gen.plummer(n, 60 + n, masses="lognormal")
    pot = 0.0
    for i in range(n - 1):
        r2 = ((pos[i + 1:] - pos[i]) ** 2).sum(1)
        pot -= (m[i] * m[i + 1:] / (np.sqrt(r2) + eps2 if ref_form else np.sqrt(r2 + eps2))).sum()
    ke = 0.5 * (m * (vel * vel).sum(1)).sum()
    ctx.upload(pos, vel, m)
    e, mom = ctx.energy(Params(eps2=eps2), ref_form=ref_form)
    assert abs(e - (ke + pot)) <= 1e-12 * (ke + abs(pot))
    np.testing.assert_allclose(mom, (m[:, None] * vel).sum(0), rtol=0, atol=1e-14)


def test_energy_of_bodies_in_one_place(ctx):
    """1 / r of two bodies in one place: infinite without softening, 1 / eps2 in the reference formula, 1 / eps
    otherwise; and squared distances far outside the series step's range."""
    pos = np.array([[0.5, 0.25, 0.0], [0.5, 0.25, 0.0], [1.5, 0.25, 0.0]])
    m = np.array([2.0, 3.0, 1.0])
    ctx.upload(pos, None, m)
    assert ctx.energy(Params(eps2=0.0))[0] == -np.inf
    assert abs(ctx.energy(Params(eps2=0.25), ref_form=True)[0] + 6.0 / 0.25 + 5.0 / 1.25) < 1e-14 * 28
    assert abs(ctx.energy(Params(eps2=0.25))[0] + 6.0 / 0.5 + 5.0 / np.sqrt(1.25)) < 1e-14 * 16
    for k in (2.0 ** 400, 2.0 ** -400):
        ctx.upload(np.array([[0.0, 0.0, 0.0], [k, 0.0, 0.0]]), None, np.array([1.0, 1.0]))
        assert abs(ctx.energy(Params())[0] * k + 1.0) < 1e-14
        assert abs(ctx.energy(Params(), ref_form=True)[0] * k + 1.0) < 1e-14


# every path that ends in a kernel adding partial sums: symmetric FP64 (small and large tiles, 1PN), directed FP64
# (below the symmetric size, every PN term), mixed slices, mixed with PN terms; and mixed without slices
@pytest.mark.parametrize("n,prec,law", [(100, FP64, NEWTON), (1000, FP64, NEWTON), (5000, FP64, NEWTON),
                                        (5000, FP64, NEWTON | PN1), (700, FP64, NEWTON | PN1 | PN2),
                                        (3000, MIXED, NEWTON), (3000, MIXED, NEWTON | PN1), (40, MIXED, NEWTON)])
def test_fused_drift_equals_single_steps(ctx, n, prec, law):
    """A multi-step run applies each next step's opening kick and drift where the forces are added up; single-step
    calls run the kick-drift kernel. The same state bit for bit."""
    pos, vel, m = gen.plummer(n, 70 + n, masses="lognormal")
    p = Params(eps2=1e-4, dt=1e-3, c=50.0, force_law=law)
    out = []
    for split in ((7,), (1,) * 7, (2, 5)):
        ctx.upload(pos, vel, m)
        for k in split:
            ctx.kdk_steps(p, k, SOLVER_ALLPAIRS, prec)
        out.append(ctx.download())
    for o in out[1:]:
        for a, b in zip(out[0], o):
            np.testing.assert_array_equal(a, b)


# the gathered post-Newtonian pair (pn.cuh: newton_pn_f64), every set of terms, all-pairs and the tree with every node opened
@pytest.mark.parametrize("terms", [PN2, PN25, PN1 | PN2, PN1 | PN25, PN2 | PN25, PN1 | PN2 | PN25])
@pytest.mark.parametrize("n,eps2", [(1, 1e-4), (97, 0.0), (700, 1e-4)])
def test_gathered_pn_terms(ctx, orc, n, eps2, terms):
    pos, vel, m = gen.plummer(n, 500 + n, masses="lognormal")
    vel = vel * 5.0
    ref = orc.allpairs(pos, m, 1.0, eps2, vel=vel, inv_c=0.1, pn=NEWTON | terms)
    ctx.upload(pos, vel, m)
    p = Params(eps2=eps2, theta=0.0, c=10.0, force_law=NEWTON | terms)
    for acc in (ctx.allpairs(p, FP64), ctx.lbvh_forces(p, FP64)):
        if n == 1:
            assert np.all(acc == 0.0)
        else:
            assert rel_l2(acc, ref) < 1e-12
