"""The second population buffer of the single phase's multi-step kernel: taken by
the first call that uses it, given back when memory runs out, and done without
when there is none.  The values do not depend on it.  Memory failures are the
engine's host-side injection."""
import numpy as np
import pytest

from flowlb_b200 import cases
from flowlb_b200 import engine as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu

NX, NY = 2048, 1024
BYTES = 9 * NX * NY * 4
FIELDS = (E.FIELD_F, E.FIELD_RHO, E.FIELD_U)


@pytest.fixture
def free():
    """Free device bytes, with every kernel of the case loaded."""
    import torch

    w = solver()
    w.step(4)
    w.step(1)
    w.close()

    def read():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info(0)[0]

    return read


def solver(**kw):
    return E.Solver(cases.plain_channel(NX, NY).flags, precision=32, tau=0.6, fx=1e-5, device=0, **kw)


def launches_of(s, n):
    before = s.launches
    s.step(n)
    return s.launches - before


def same(a, b):
    return all(np.array_equal(a.read(f), b.read(f)) for f in FIELDS)


def test_taken_by_the_first_call_of_several_steps(free):
    start = free()
    s = solver()
    made = free()
    assert start - made < 2 * BYTES  # one population buffer, density, velocity, flags
    s.step(1)
    assert abs(free() - made) <= 2 << 20
    s.step(8)
    assert abs(made - free() - BYTES) <= 4 << 20
    s.close()
    assert abs(free() - start) <= 2 << 20


def test_without_it_one_step_per_launch_and_the_same_values(free, monkeypatch):
    a, b = solver(), solver()
    a.step(21)
    monkeypatch.setenv("FLB_FAIL_ALLOC_AT", "second")
    assert launches_of(b, 21) == 21
    assert same(a, b)
    monkeypatch.delenv("FLB_FAIL_ALLOC_AT")
    for _ in range(64):
        a.step(2)
        b.step(2)
    a.step(22)
    assert launches_of(b, 22) < 22  # asked for again
    assert same(a, b)
    a.close()
    b.close()


def test_given_back_when_a_creation_runs_out_of_memory(free, monkeypatch):
    a, ref = solver(), solver(kernel_variant=1)
    a.step(13)  # an odd number of launches: the buffers have changed places
    ref.step(13)
    held = free()
    monkeypatch.setenv("FLB_FAIL_ALLOC_AT", "1")
    c = cases.plain_channel(64, 32)
    b = E.Solver(c.flags, precision=32, tau=0.6, fx=1e-5, device=0)  # the first allocation fails once
    monkeypatch.delenv("FLB_FAIL_ALLOC_AT")
    assert abs(free() - held - BYTES) <= 8 << 20
    a.step(1)
    ref.step(1)
    assert same(a, ref)
    assert launches_of(a, 13) == 13
    ref.step(13)
    for _ in range(63):
        a.step(2)
    ref.step(126)
    assert abs(free() - held) <= 8 << 20  # and taken again
    assert same(a, ref)
    for s in (a, ref, b):
        s.close()


def test_reset_without_inlets_takes_several_steps_per_launch():
    closed = cases.plain_channel(90, 26).flags
    flags = closed.copy()
    flags[1:-1, 0] = cases.INLET
    flags[1:-1, -1] = cases.OUTLET
    s = E.Solver(flags, precision=32, tau=0.7, fx=1e-5, device=0)
    assert launches_of(s, 16) == 16
    s.reset(closed)
    o = O.Oracle(closed, O.OracleConfig(variant=O.F32, bb=O.BB_HALFWAY, arithmetic=O.ARITH_FUSED, tau=0.7, fx=1e-5))
    assert launches_of(s, 16) < 16
    o.step(16)
    assert np.array_equal(s.f, o.f64().astype(np.float32)) and np.array_equal(s.u, o.u)
    s.close()


def test_batch_without_them_gives_the_same_values(monkeypatch):
    cs = [cases.plain_channel(64 + 9 * k, 30 + k) for k in range(6)]

    def batch():
        b = E.Batch([(c.flags, 0.6, 1e-5, 0.0) for c in cs], autotune=0)
        b.set_launch("streams", 1, 4, 0)
        b.step(45)
        return [b.read(k, f) for k in range(len(cs)) for f in FIELDS]

    want = batch()
    monkeypatch.setenv("FLB_FAIL_ALLOC_AT", "second")
    assert all(np.array_equal(x, y) for x, y in zip(want, batch()))
