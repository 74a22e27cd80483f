"""The KDK graph kept across calls (integrate.cu: middle_graph, step_key) with the
all-pairs solver: states of one size whose massless bodies at the end differ
take different kernels and source ranges, so one's graph must not serve the
other."""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, MIXED, SOLVER_ALLPAIRS, Context, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_kept_graph_follows_the_sources(ctx, prec):
    n = 3000
    pos, vel, m = gen.plummer(n, 1033, masses="lognormal")
    tail = m.copy()
    tail[n // 3:] = 0.0

    def run(c, masses, dt):
        c.upload(pos, vel, masses)
        c.kdk_steps(Params(G=1.0, eps2=1e-4, dt=dt), 6, SOLVER_ALLPAIRS, prec)
        return c.download()

    # the first run allocates; of the others each would find the graph of the one before it (other contexts come last:
    # their buffers' release advances the generation that a kept graph is bound to)
    calls = [(m, 1e-3), (tail, 1e-3), (tail, 5e-4), (m, 5e-4), (tail, 5e-4)]
    got = [run(ctx, *call) for call in calls]
    for call, out in zip(calls, got):
        with Context(0) as other:
            ref = run(other, *call)
        for a, r in zip(out, ref):
            np.testing.assert_array_equal(a, r)
