"""The ensemble's default unrolling, chosen by the force law and the number of
systems (aster_ensemble_run), gives the bits of every unrolling."""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import EIH, FP64, MIXED, NEWTON, PN1, PN2, PN25, YOSHIDA4, Context, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsys", [5, 2400])  # either side of sixteen systems an SM
@pytest.mark.parametrize("law", [NEWTON, NEWTON | PN1, NEWTON | PN1 | PN2 | PN25, NEWTON | PN1 | EIH])
@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_default_unrolling_gives_the_same_bits(nsys, law, prec):
    pos, vel, m, off = gen.hierarchical_ensemble(nsys, 71, 3, 64 if nsys < 100 else 9)
    p = Params(dt=1e-4, c=100.0, force_law=law)
    out = []
    with Context(0) as c:
        for unroll in (0, 1, 2, 4):
            c.ensemble_upload(off, pos, vel, m)
            c.ensemble_run(p, 5, YOSHIDA4, prec, config=dict(unroll=unroll))
            out.append(c.ensemble_download())
    for o in out[1:]:
        for a, b in zip(out[0], o):
            np.testing.assert_array_equal(a, b)
