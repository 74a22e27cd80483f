"""A cancel that comes while the systems are being taken: another thread calls it
without pause from before the run on (a run clears the flag as it begins, so a
single earlier call is of no effect; the next one ends the run). And that single
earlier call."""
import threading
import time

import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import ERR_CANCELLED, FP64, MIXED, AsterError, Context, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsys,steps,check", [(1, 4000000, 1), (300, 400000, 64), (4000, 100000, 1), (4000, 100000, 0)])
@pytest.mark.parametrize("prec", [MIXED, FP64])
def test_cancel_from_the_start(nsys, steps, check, prec):
    pos, vel, m, off = gen.hierarchical_ensemble(nsys, 22, 3, 12)
    with Context(0) as c:
        c.ensemble_upload(off, pos, vel, m)
        over = threading.Event()

        def keep_cancelling():
            while not over.is_set():
                c.ensemble_cancel()

        t = threading.Thread(target=keep_cancelling)
        t.start()
        t0 = time.perf_counter()
        try:
            with pytest.raises(AsterError) as e:
                c.ensemble_run(Params(dt=1e-5), steps, precision=prec, config=dict(check_every=check))
        finally:
            over.set()
            t.join()
        assert e.value.status == ERR_CANCELLED
        assert time.perf_counter() - t0 < 10.0


def test_cancel_before_the_run_is_dropped():
    pos, vel, m, off = gen.hierarchical_ensemble(100, 23, 3, 12)
    out = []
    with Context(0) as c:
        for cancel in (False, True):
            c.ensemble_upload(off, pos, vel, m)
            if cancel:
                c.ensemble_cancel()
            c.ensemble_run(Params(dt=1e-5), 50)
            out.append(c.ensemble_download())
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
