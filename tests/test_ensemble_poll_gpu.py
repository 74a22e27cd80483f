"""The ensemble's cancel flag, read by one warp for all: a flag set before the
systems are taken, while short systems are going through and late in a run;
and a run after a cancelled one."""
import threading
import time

import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import ERR_CANCELLED, FP64, MIXED, AsterError, Context, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsys,steps,delay", [(1, 4000000, 0.05), (300, 400000, 0.02), (4000, 100000, 0.05)])
@pytest.mark.parametrize("prec", [MIXED, FP64])
def test_cancel_reaches_every_warp(nsys, steps, delay, prec):
    pos, vel, m, off = gen.hierarchical_ensemble(nsys, 21, 3, 12)
    p = Params(dt=1e-5)
    with Context(0) as c:
        c.ensemble_upload(off, pos, vel, m)
        t = threading.Timer(delay, c.ensemble_cancel)
        t.start()
        t0 = time.perf_counter()
        with pytest.raises(AsterError) as e:
            c.ensemble_run(p, steps, precision=prec)
        took = time.perf_counter() - t0
        t.join()
        assert e.value.status == ERR_CANCELLED
        assert took < 20.0
        c.ensemble_upload(off, pos, vel, m)
        c.ensemble_run(p, 20, precision=prec)  # the flag does not outlast the run
        a = c.ensemble_download()
        c.ensemble_upload(off, pos, vel, m)
        c.ensemble_run(p, 20, precision=prec, config=dict(check_every=1, use_graph=0))
        for x, y in zip(a, c.ensemble_download()):
            np.testing.assert_array_equal(x, y)
