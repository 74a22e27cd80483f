"""The adjoint's step structure (adjoint.cu): checkpoints, segments and fused kicks and drifts."""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, MIXED, Params
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps,every", [(40, 9, 4), (300, 8, 4), (1000, 7, 1), (1000, 1, 4), (3001, 9, 5)])
@pytest.mark.parametrize("prec,tol", [(FP64, 1e-10), (MIXED, 1e-5)])
def test_adjoint_segments_match_oracle(ctx, orc, n, steps, every, prec, tol):
    """The adjoint with its steps' kicks and drifts applied where forces are added, checkpoints at, before and after the
    last step, one step per segment, and the short last segment; without slices (40 bodies) and with. Relative L2
    against the oracle's reverse mode, as the adjoint's tests: FP64 1e-10, mixed 1e-5."""
    pos, vel, m = gen.plummer(n, 80 + n)
    p = Params(eps2=1e-4, dt=1e-3)
    target = pos + np.random.default_rng(n).normal(0.0, 1e-2, pos.shape)
    ctx.upload(pos, vel, m)
    loss, gx, gv, gm = ctx.adjoint(p, steps, target, prec, every)
    rl, rx, rv, rm = orc.adjoint(pos, vel, m, target, p.dt, steps, eps2=p.eps2)
    assert abs(loss - rl) < tol * abs(rl)
    assert rel_l2(gx, rx) < tol and rel_l2(gv, rv) < tol
    assert rel_l2(gm, rm) < tol
    x, v, _ = ctx.download()  # the uploaded state is unchanged
    np.testing.assert_array_equal(x, pos)
    np.testing.assert_array_equal(v, vel)
