"""The staging of large results on the host (aster_b200/csrc/staged_copy.cuh),
compiled alone with copies and allocations of its own: memory that runs out while
the threads start, and copies that fail, end in a whole result or in an error,
never in the process's end."""
import subprocess
from pathlib import Path

import pytest

SRC = Path(__file__).with_name("host") / "staged_copy_harness.cpp"


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    out = tmp_path_factory.mktemp("staged") / "harness"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", str(SRC), "-o", str(out)], check=True)
    return out


@pytest.mark.parametrize("what", ["memory", "device"])
@pytest.mark.parametrize("pieces", [1, 7, 16, 17, 40])
def test_staged_copy(harness, what, pieces):
    r = subprocess.run([str(harness), what, str(pieces)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)


def test_slab_is_asked_for_again_by_later_contexts(harness):
    r = subprocess.run([str(harness), "slab", "0"], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)


def test_only_pageable_destinations_are_staged(harness):
    r = subprocess.run([str(harness), "pieces", "0"], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)


@pytest.mark.gpu
@pytest.mark.parametrize("locked", [(), (0,), (1, 2), (0, 1, 2)])
@pytest.mark.parametrize("n", [1000, 262153])
def test_mixed_destinations_arrive_whole(locked, n):
    import ctypes

    import numpy as np
    import torch

    from aster_b200.api import Context
    rng = np.random.default_rng(5)
    pos, vel, m = rng.normal(size=(n, 3)), rng.normal(size=(n, 3)), rng.uniform(1, 2, n)
    out = [torch.full((n, 3), float("nan"), dtype=torch.float64, pin_memory=k in locked).numpy() for k in range(3)]
    with Context(0) as c:
        c.upload(pos, vel, m)
        assert c.lib.aster_state_download(c.h, *[ctypes.c_void_p(o.ctypes.data) for o in out]) == 0
    np.testing.assert_array_equal(out[0], pos)
    np.testing.assert_array_equal(out[1], vel)
    assert not out[2].any()
