"""Results of several megabytes through page-locked staging (context.cu)."""
import threading

import numpy as np
import pytest

from aster_b200.api import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [87381, 87382, 262153])
def test_staged_download_is_whole(n):
    """Results on either side of the size from which they come through page-locked staging (6 MB), from two contexts
    at once (one of them finds the staging in use)."""
    rng = np.random.default_rng(n)
    data = [(rng.normal(size=(n, 3)), rng.normal(size=(n, 3)), rng.uniform(1, 2, n)) for _ in range(2)]
    ctxs = [Context(0).upload(p, v, m) for p, v, m in data]
    bad = []

    def fetch(c, d):
        for _ in range(5):
            p, v, a = c.download()
            if not (np.array_equal(p, d[0]) and np.array_equal(v, d[1]) and not a.any()):
                bad.append(n)

    team = [threading.Thread(target=fetch, args=x) for x in zip(ctxs, data)]
    for t in team:
        t.start()
    for t in team:
        t.join()
    for c in ctxs:
        c.close()
    assert not bad
    with Context(0).upload(*data[0]) as c:  # after the last context took the staging with it
        assert np.array_equal(c.download()[0], data[0][0])
