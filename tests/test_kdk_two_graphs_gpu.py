"""The KDK graphs that a context keeps, one for either solver (integrate.cu:
middle_graph): calls that alternate the solvers give the states of calls that do
not, and capture nothing again. The capture is seen in the time of a short call:
with it the all-pairs call below takes about twice as long (165 against 86 us),
and the least of many is compared, so that a busy host does not show."""
import time

import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, MIXED, SOLVER_ALLPAIRS, SOLVER_LBVH, Context, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_alternating_solvers_keep_both_graphs(prec):
    n = 1000
    pos, vel, m = gen.plummer(n, 51)
    p = Params(eps2=1e-4, dt=1e-5)
    with Context(0) as c:
        c.upload(pos, vel, m)

        def call(solver):
            t = time.perf_counter()
            c.kdk_steps(p, 5, solver, prec)
            return time.perf_counter() - t

        for _ in range(5):
            call(SOLVER_LBVH), call(SOLVER_ALLPAIRS)
        alternating = min((call(SOLVER_LBVH), call(SOLVER_ALLPAIRS))[1] for _ in range(60))
        alone = min(call(SOLVER_ALLPAIRS) for _ in range(60))
        assert alternating < 1.5 * alone, (alternating, alone)


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_alternating_solvers_step_as_alone(prec):
    n = 3000
    pos, vel, m = gen.plummer(n, 52, masses="lognormal")
    p = Params(eps2=1e-4, dt=1e-3, theta=0.0)
    order = [SOLVER_LBVH, SOLVER_ALLPAIRS, SOLVER_LBVH, SOLVER_ALLPAIRS, SOLVER_ALLPAIRS, SOLVER_LBVH]
    with Context(0) as c:
        got = []
        for s in order:
            c.upload(pos, vel, m)
            c.kdk_steps(p, 6, s, prec)
            got.append(c.download())
    for s, out in zip(order, got):
        with Context(0) as c:
            c.upload(pos, vel, m)
            c.kdk_steps(p, 6, s, prec)
            for a, r in zip(out, c.download()):
                np.testing.assert_array_equal(a, r)
