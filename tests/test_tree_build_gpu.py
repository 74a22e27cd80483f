"""The bottom-up tree build (lbvh.cu: k_tree_local, k_tree_merge) against the
oracle's Karras tree, every array bit for bit: sizes around a block of 64 leaves,
one and several merge launches, and bodies clustered so that subtrees left over
by a block exceed a merge's shared memory."""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import MIXED, NEWTON, PN1, Params
from conftest import rel_l2

pytestmark = pytest.mark.gpu

KEYS = (("codes", "codes"), ("sorted_codes", "sorted_codes"), ("perm", "perm"), ("left", "left"), ("right", "right"),
        ("parent", "parent"), ("range_lo", "range_lo"), ("range_hi", "range_hi"), ("node_mass", "node_mass"),
        ("node_com", "node_com"), ("node_bmin", "bmin"), ("node_bmax", "bmax"), ("node_rcrit2", "rcrit2"))


def _same(ctx, orc, pos, m, bits=30):
    ctx.upload(pos, None, m)
    t = ctx.lbvh_build(Params(theta=0.5, morton_bits=bits))
    o = orc.lbvh(pos, m, 0.5, bits=bits)
    for a, b in KEYS:
        np.testing.assert_array_equal(t[a], o[b], err_msg=a)


# sort: a cluster's block of 1024 bodies, its 16 blocks with one and with two bodies a thread, the sort of many launches;
# tree: one block, two, the last merge alone (up to 13k bodies), one middle merge, two middle merges (above 450k)
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 128, 129, 1024, 1025, 4095, 12500, 14500, 16384, 16385, 32768,
                               32769, 100001, 470001])
@pytest.mark.parametrize("bits", [30, 63])
def test_tree_bit_exact(ctx, orc, n, bits):
    pos, _, m = gen.plummer(n, 40 + n, masses="lognormal")
    if n > 200:
        pos[100:130] = pos[50]   # equal codes
        m[10:100] = 0.0          # nodes without mass
    _same(ctx, orc, pos, m, bits)


@pytest.mark.parametrize("n", [5000, 60000])
@pytest.mark.parametrize("bits", [30, 63])
def test_clustered_bodies(ctx, orc, n, bits):
    """Distances from the origin falling by powers of two down to 2^-60, so that subtrees hang off one long spine and
    the blocks leave most of their leaves over; and every body in one place."""
    rng = np.random.default_rng(8)
    u = rng.normal(size=(n, 3))
    pos = u / np.linalg.norm(u, axis=1)[:, None] * 2.0 ** -rng.uniform(0, 60, n)[:, None]
    _same(ctx, orc, pos, rng.uniform(0.5, 1.5, n), bits)
    _same(ctx, orc, np.full((n, 3), 0.25), rng.uniform(0.5, 1.5, n), bits)


def test_spines_cut_by_every_block(ctx, orc):
    """1024 runs of the 21 codes prefix | {0, 2^0 .. 2^19}: each run is a spine of 21 leaves, and a block of 64 leaves
    cuts one at either end, so that it leaves some 20 subtrees over: 64 blocks' items pass the shared memory of a
    middle merge, and the last merge's too."""
    codes = np.array([(r << 20) | c for r in range(1024) for c in [0] + [1 << k for k in range(20)]], dtype=np.int64)
    q = np.zeros((len(codes), 3), dtype=np.int64)
    for b in range(10):
        for k in range(3):
            q[:, k] |= ((codes >> (3 * b + k)) & 1) << b
    pos = np.vstack([(q + 0.5) / 512.0 - 1.0, -np.ones(3)])  # the last body spans the cube
    t = orc.lbvh(pos, np.ones(len(pos)), 0.5)
    left_over = [_frontier(t["left"], t["right"], t["range_lo"], t["range_hi"], b0, len(pos))
                 for b0 in range(0, len(pos), 64)]
    assert sum(left_over[:64]) > 512 and sum(left_over) > 1344
    _same(ctx, orc, pos, np.random.default_rng(4).uniform(0.5, 1.5, len(pos)))


def _frontier(left, right, lo, hi, b0, n):
    """Maximal subtrees inside the leaves [b0, b0 + 64)."""
    b1, count, stack = min(b0 + 64, n) - 1, 0, [n]
    while stack:
        v = stack.pop()
        if lo[v] > b1 or hi[v] < b0:
            continue
        if lo[v] >= b0 and hi[v] <= b1:
            count += 1
        else:
            stack += [left[v], right[v]]
    return count


@pytest.mark.parametrize("scale", [1e-130, 1e130])
def test_divisions_outside_the_middle_range(ctx, orc, scale):
    """Centres of mass whose sums leave [2^-400, 2^400) take the plain division."""
    pos, _, m = gen.plummer(3000, 77, masses="lognormal")
    _same(ctx, orc, pos * scale, m)


def test_pn_walk_after_newtonian_walk(ctx, orc):
    """The parents and siblings that the node velocities need are written again when a PN law asks for them."""
    pos, vel, m = gen.plummer(9000, 5, masses="lognormal")
    ctx.upload(pos, vel, m)
    p = Params(eps2=1e-4, c=30.0, theta=0.5, force_law=NEWTON | PN1)
    ctx.lbvh_forces(Params(eps2=1e-4, theta=0.5), MIXED)
    a = ctx.lbvh_forces(p, MIXED)
    o = orc.lbvh(pos, m, 0.5)
    ref, _ = orc.lbvh_forces_pn(o, o["perm"], pos, vel, 1.0, 1e-4, 1.0 / 30.0, NEWTON | PN1)
    assert rel_l2(a, ref) < 1e-6
