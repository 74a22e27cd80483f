"""FP64 sums over directed pairs (allpairs.cu:k_allpairs_fp64), four sources at a
time: source counts around multiples of four and of a tile, the body itself among
its sources softened and not, separations outside the series step's range, and
target lists. Tolerance as test_fp64_pairs_gpu.py: 1e-13 relative L2 to the
oracle, whose terms differ by a few roundings each."""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, Context, Params
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def directed():
    """A context without room for partial sums: every evaluation takes the directed kernel, in one slice."""
    mp = pytest.MonkeyPatch()
    mp.setenv("ASTER_SUMS_LIMIT", "0")
    c = Context(0)
    mp.undo()
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 127, 128, 129, 131, 132, 255, 257, 1001, 3003])
@pytest.mark.parametrize("eps2", [1e-4, 0.0])
def test_all_on_all_matches_oracle(directed, orc, n, eps2):
    pos, vel, m = gen.plummer(n, 700 + n, masses="lognormal")
    directed.upload(pos, vel, m)
    acc = directed.allpairs(Params(eps2=eps2, G=1.25), FP64)
    assert directed.stats()["kernels"] == 1
    ref = orc.allpairs(pos, m, 1.25, eps2)
    if n == 1:
        assert np.all(acc == 0.0)
    else:
        assert rel_l2(acc, ref) < 1e-13


@pytest.mark.parametrize("n,nt", [(130, 1), (1001, 7), (5003, 300), (20003, 129)])
@pytest.mark.parametrize("eps2", [1e-4, 0.0])
def test_targets_match_oracle(ctx, orc, n, nt, eps2):
    pos, vel, m = gen.plummer(n, 800 + n, masses="lognormal")
    m[n - n // 3:] = 0.0  # the sources end in the middle of a tile
    tg = np.random.default_rng(n).permutation(n)[:nt].astype(np.int32)
    ctx.upload(pos, vel, m)
    acc = ctx.allpairs_targets(Params(eps2=eps2), tg, FP64)
    assert rel_l2(acc, orc.allpairs(pos, m, 1.0, eps2, targets=tg)) < 1e-13


@pytest.mark.parametrize("scale", [1e-105, 1e105])
@pytest.mark.parametrize("n", [50, 515])
def test_extreme_scales(directed, scale, n):
    """With masses scaled as the coordinates, accelerations go as their inverse (a power of two)."""
    pos, _, m = gen.plummer(n, 33)
    k = 2.0 ** round(np.log2(scale))
    ref = directed.upload(pos, None, m).allpairs(Params(), FP64)
    acc = directed.upload(pos * k, None, m * k).allpairs(Params(), FP64)
    assert np.isfinite(acc).all()
    assert rel_l2(acc * k, ref) < 1e-13


def test_one_far_body_among_ordinary_ones(directed, orc):
    """A body so far off that its squared distances leave the range: its group of sources takes the other branch."""
    pos, vel, m = gen.plummer(203, 34)
    pos[77] = [1e120, -1e120, 1e119]
    acc = directed.upload(pos, vel, m).allpairs(Params(eps2=1e-4), FP64)
    ref = orc.allpairs(pos, m, 1.0, 1e-4)
    keep = np.arange(203) != 77
    assert rel_l2(acc[keep], ref[keep]) < 1e-13
