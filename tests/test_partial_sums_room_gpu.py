"""Force and adjoint calls when the device has little memory left: the kernels'
partial sums find no room and the sums are made in one piece.

The other tensors take the memory (torch allocations); what is left free is a
fixed number of megabytes, enough for everything but the partial sums. Last, the
limit on the sums of a context that has all the room it could want."""
import numpy as np
import pytest

from aster_b200 import gen
from aster_b200.api import FP64, MIXED, NEWTON, PN1, PN2, SOLVER_ALLPAIRS, AsterError, Context, Params
from conftest import rel_l2

pytestmark = pytest.mark.gpu
MB = 1 << 20
ERR_OOM = 3


class Crowd:
    """Takes all device memory but `leave` bytes while it lasts."""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        import torch
        torch.cuda.empty_cache()
        self.held = []
        while True:
            free = torch.cuda.mem_get_info()[0]
            if free <= self.leave + 32 * MB:
                return self
            size = min(free - self.leave, 8192 * MB) // (2 * MB) * (2 * MB)
            self.held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))

    def __exit__(self, *exc):
        import torch
        self.held = None
        torch.cuda.empty_cache()


def test_adjoint_without_room_is_an_error_or_right():
    """131,072 bodies: 32 slices of sums take 134 MB, the call's other arrays 60."""
    n = 131072
    pos, vel, m = gen.plummer(n, 41)
    target = pos + 0.01
    p = Params(eps2=1e-4, dt=1e-3)
    with Context(0) as roomy:  # (and every kernel has been loaded)
        ref = roomy.upload(pos, vel, m).adjoint(p, 3, target, MIXED, 2)
        small = Context(0).upload(pos[:70], vel[:70], m[:70])  # one slice
        small.adjoint(p, 3, target[:70], MIXED, 2)
        small.close()
    with Context(0) as c:
        c.upload(pos, vel, m)
        with Crowd(100 * MB):
            try:
                got = c.adjoint(p, 3, target, MIXED, 2)
            except AsterError as e:
                assert e.status == ERR_OOM
                got = None
        if got is not None:
            assert abs(got[0] - ref[0]) <= 1e-9 * ref[0]
            for g, r in zip(got[1:], ref[1:]):
                assert rel_l2(g, r) < 1e-5
        again = c.upload(pos, vel, m).adjoint(p, 3, target, MIXED, 2)
        assert again[0] == ref[0]
        for g, r in zip(again[1:], ref[1:]):
            np.testing.assert_array_equal(g, r)


@pytest.mark.parametrize("prec,tol", [(MIXED, 1e-6), (FP64, 1e-12)])
@pytest.mark.parametrize("steps", [1, 2, 3, 6])
def test_steps_without_room_run_in_one_piece(prec, tol, steps):
    """All-pairs steps, the later ones captured: a step that finds no room for its sums looks for it once, before the
    capture. 131,072 bodies need 134 MB (slices) or 403 MB (tile pairs), 64 are free. Accelerations as far apart as
    two orders of one sum (mixed: FP32 pair terms)."""
    n = 131072
    pos, vel, m = gen.plummer(n, 42)
    p = Params(eps2=1e-4, dt=1e-3)
    with Context(0) as roomy:
        roomy.upload(pos, vel, m).kdk_steps(p, steps, SOLVER_ALLPAIRS, prec)
        ref = roomy.download()
        kernels = roomy.stats()["kernels"]
    with Context(0) as c:
        c.upload(pos, vel, m)
        with Crowd(64 * MB):
            c.kdk_steps(p, steps, SOLVER_ALLPAIRS, prec)
            assert c.stats()["kernels"] == kernels - 2  # a kick-drift in every step, and no reductions
            got = c.download()
    for g, r in zip(got, ref):
        assert rel_l2(g, r) < tol


@pytest.mark.parametrize("steps", [1, 4])
def test_room_for_slices_alone_takes_slices(steps):
    """FP64, 180,000 bodies: 381 MB of tile-pair sums do not fit into 260, 184 MB of slices' sums do."""
    n = 180000
    pos, vel, m = gen.plummer(n, 48)
    p = Params(eps2=1e-4, dt=1e-3)
    out = []
    for leave in (None, 260 * MB):
        with Context(0) as c:
            c.upload(pos, vel, m)
            if leave is None:
                c.kdk_steps(p, steps, SOLVER_ALLPAIRS, FP64)
                kernels = c.stats()["kernels"]
            else:
                with Crowd(leave):
                    c.kdk_steps(p, steps, SOLVER_ALLPAIRS, FP64)
                    assert c.stats()["kernels"] == kernels  # reductions, and the drifts in them
            out.append(c.download())
    assert not np.array_equal(out[0][2], out[1][2])
    for a, b in zip(*out):
        assert rel_l2(b, a) < 1e-12


def test_room_that_comes_free_is_used():
    """FP64 forces of 300,000 bodies: 706 MB of tile-pair sums do not fit into 600; once the memory is free again the
    same context takes the tile pairs (the sums of a fresh context, bit for bit)."""
    n = 300000
    pos, vel, m = gen.plummer(n, 43)
    p = Params(eps2=1e-4)
    with Context(0) as roomy:
        ref = roomy.upload(pos, vel, m).allpairs(p, FP64)
    with Context(0) as c:
        c.upload(pos, vel, m)
        with Crowd(600 * MB):
            tight = c.allpairs(p, FP64)
            np.testing.assert_array_equal(c.allpairs(p, FP64), tight)
        assert not np.array_equal(tight, ref) and rel_l2(tight, ref) < 1e-12
        np.testing.assert_array_equal(c.allpairs(p, FP64), ref)


@pytest.mark.parametrize("prec,tol", [(MIXED, 1e-5), (FP64, 1e-10)])
def test_adjoint_without_room_runs_in_one_piece(prec, tol):
    """Gradients as far from those with room as test_adjoint_steps_gpu.py lets either be from the oracle."""
    n = 131072
    pos, vel, m = gen.plummer(n, 44)
    target = pos + 0.01
    p = Params(eps2=1e-4, dt=1e-3)
    with Context(0) as roomy:
        ref = roomy.upload(pos, vel, m).adjoint(p, 3, target, prec, 2)
        kernels = roomy.stats()["kernels"]
    with Context(0) as c:
        c.upload(pos, vel, m)
        with Crowd(100 * MB):
            got = c.adjoint(p, 3, target, prec, 2)
            assert c.stats()["kernels"] < kernels  # no reductions
        assert abs(got[0] - ref[0]) <= tol * ref[0]
        for g, r in zip(got[1:], ref[1:]):
            assert rel_l2(g, r) < tol


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("limit,n,law", [(8, 12500, NEWTON), (8, 12500, NEWTON | PN1), (2, 20000, NEWTON), (2, 3900, NEWTON | PN1),
                                         (0, 5000, NEWTON), (0, 130, NEWTON)])
@pytest.mark.parametrize("prec,tol", [(MIXED, 1e-6), (FP64, 1e-12)])
def test_limited_sums_give_the_same_results(monkeypatch, limit, n, law, prec, tol):
    """Fewer tiles than without a limit (12,500 bodies: 25), the directed kernel with one slice (20,000; 3900), and no
    sums at all: forces, steps and gradients, and the memory that the first of them takes."""
    pos, vel, m = gen.plummer(n, 45 + n)
    p = Params(eps2=1e-4, dt=1e-3, c=50.0, force_law=law)
    out = []
    for lim in (None, limit):
        if lim is not None:
            monkeypatch.setenv("ASTER_SUMS_LIMIT", str(lim))
        with Context(0) as c:
            c.upload(pos, vel, m)
            free = _free()
            a = c.allpairs(p, prec)
            if lim is not None:
                assert free - _free() <= (lim + 2) * MB  # (the device hands out 2 MB at a time)
            c.kdk_steps(p, 5, SOLVER_ALLPAIRS, prec)
            state = c.download()
            grads = () if law != NEWTON else c.upload(pos, vel, m).adjoint(p, 3, pos + 0.01, prec, 2)[1:]
        out.append((a, *state, *grads))
    for k, (x, y) in enumerate(zip(*out)):
        assert rel_l2(y, x) < (tol if k < 4 else 10 * tol), k


def test_sums_of_a_large_system_stay_within_the_limit():
    n = 1 << 20
    pos, vel, m = gen.plummer(n, 46)
    with Context(0) as c:
        c.upload(pos, vel, m)
        free = _free()
        c.allpairs(Params(eps2=1e-4), FP64)
        assert free - _free() <= 1026 * MB


@pytest.mark.parametrize("n,law,kernels", [(2432, NEWTON, 1), (2433, NEWTON, 2), (2750, NEWTON, 2), (2750, NEWTON | PN1, 2),
                                           (2750, NEWTON | PN1 | PN2, 1), (1700, NEWTON, 2)])
def test_middle_sizes_take_slices_of_two_tiles(monkeypatch, n, law, kernels):
    """Mixed forces, 2433 to 3072 bodies: the sums of 256-source slices fit into 1 MB, those of 128-source slices,
    which the sizes below and the longer force laws take, do not (one launch less: no reduction)."""
    pos, vel, m = gen.plummer(n, 47)
    p = Params(eps2=1e-4, c=50.0, force_law=law)
    with Context(0) as c:
        ref = c.upload(pos, vel, m).allpairs(p, FP64)
    monkeypatch.setenv("ASTER_SUMS_LIMIT", "1")
    with Context(0) as c:
        acc = c.upload(pos, vel, m).allpairs(p, MIXED)
        assert c.stats()["kernels"] == kernels
    assert rel_l2(acc, ref) < 1e-6
