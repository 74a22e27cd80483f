"""Accelerations that a download gives after Wisdom-Holman steps: the planets'
interaction at the final positions, whichever launch formed it (inside the drift
kernel up to 64 massive bodies in FP64, a force launch otherwise). Tolerances: a
sum of 65 FP64 terms of a few roundings each, 1e-13 of the largest; mixed 1e-6."""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, MIXED, Context, Params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planets,particles", [(1, 0), (8, 0), (8, 1000), (63, 700), (64, 700)])
@pytest.mark.parametrize("eps2", [0.0, 1e-4])
@pytest.mark.parametrize("prec", [FP64, MIXED])
def test_download_gives_the_interaction(planets, particles, eps2, prec):
    pos, vel, m = gen.planetary_system(planets, particles, 77 + planets, planet_mass=(1e-7, 1e-5))
    with Context(0) as c:
        c.upload(pos, vel, m)
        c.wh_steps(Params(G=1.5, eps2=eps2, dt=0.02), 3, prec)
        x, _, a = c.download()
    ref = np.zeros_like(x)
    for j in range(1, 1 + planets):
        d = x[j] - x
        r2 = (d * d).sum(1) + eps2
        r2[j] = 1.0
        ref += 1.5 * m[j] * d / r2[:, None] ** 1.5
    # (the central body takes no part in the interaction; its entry is taken at its position before the steps)
    scale = np.abs(ref[1:]).max()
    assert np.abs(a[1:] - ref[1:]).max() <= (1e-13 if prec == FP64 else 1e-6) * scale
    x0 = x[0]
    q = np.concatenate([pos[:1], x[1:1 + planets] - x0])  # as the steps hold them: the others relative to the centre
    d = q[1:] - q[0]
    r2 = (d * d).sum(1) + eps2
    r0 = (1.5 * m[1:1 + planets, None] * d / r2[:, None] ** 1.5).sum(0)
    assert np.abs(a[0] - r0).max() <= (1e-13 if prec == FP64 else 1e-6) * max(scale, np.abs(r0).max())
