"""The single-phase multi-step kernel (several time steps per launch) against
the CPU oracle: every value of the population array, density and velocity equal."""
import numpy as np
import pytest

from flowlb_b200 import cases
from flowlb_b200 import engine as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def pair(flags, variant, bb, arith, **kw):
    prec = {O.F64: 64, O.F32: 32, O.F16S: 16}[variant]
    s = E.Solver(flags, precision=prec, bounce_back=bb, arithmetic=arith, **kw)
    o = O.Oracle(flags, O.OracleConfig(variant=variant, bb=bb, arithmetic=arith, **kw))
    return s, o


def check(s, o, variant, what):
    f = o.f64() if variant == O.F64 else o.f64().astype(np.float32)
    for name, a, b in (("f", s.f, f), ("rho", s.rho, o.rho), ("u", s.u, o.u)):
        assert np.array_equal(a, b), f"{what}: {name} differs at {np.flatnonzero(a != b)[:5]}"


# widths and heights below, at and beyond a window, whole vectors and not; one
# grid per window size the dispatch picks
@pytest.mark.parametrize("nx,ny", [(3, 5), (17, 9), (64, 40), (101, 61), (256, 64), (517, 131), (1024, 136)],
                         ids=lambda v: str(v))
@pytest.mark.parametrize("variant", [O.F32, O.F64, O.F16S], ids=["f32", "f64", "f16s"])
@pytest.mark.parametrize("bb,arith", [(E.BB_HALFWAY, E.ARITH_FUSED), (E.BB_IMPLICIT, E.ARITH_REFERENCE)],
                         ids=["halfway-fused", "implicit-ref"])
def test_multi_step_matches_oracle(nx, ny, variant, bb, arith):
    w = max(1, nx // 5)
    flags = cases.channel_with_block(nx, ny, nx // 3, nx // 3 + w, max(2, ny // 3))
    flags[ny // 2, nx // 2] = cases.GAS  # not updated, not a wall
    s, o = pair(flags, variant, bb, arith, tau=0.58, fx=2e-5, fy=-1e-5)
    for n in (1, 2, 21, 8, 3):  # odd and even starts, whole launches and remainders
        s.step(n)
        o.step(n)
        check(s, o, variant, f"t={o.t}")
    s.close()


@pytest.mark.parametrize("kw", [dict(u_max=0.01), dict(subgrid=True), dict(collision=1, use_force=False)],
                         ids=["limiter", "subgrid", "trt"])
def test_multi_step_options_match_oracle(kw):
    c = cases.plain_channel(200, 48)
    s, o = pair(c.flags, O.F32, E.BB_HALFWAY, E.ARITH_FUSED, tau=0.55, fx=1e-4, **kw)
    s.step(67)
    o.step(67)
    check(s, o, O.F32, str(kw))
    s.close()


def test_multi_step_large_grid_equals_one_step_per_launch():
    """A grid on the large-grid window (several windows wide and high), against the one-step kernels."""
    c = cases.plain_channel(2052, 600)
    for prec in (32, 64, 16):
        a = E.Solver(c.flags, precision=prec, tau=0.6, fx=1e-5)
        b = E.Solver(c.flags, precision=prec, tau=0.6, fx=1e-5, kernel_variant=1)
        for n in (37, 6):
            a.step(n)
            b.step(n)
        for fid in (E.FIELD_F, E.FIELD_RHO, E.FIELD_U):
            assert np.array_equal(a.read(fid), b.read(fid)), (prec, fid)
        a.close()
        b.close()


def test_inlet_outlet_buffers_over_odd_calls_writes_checkpoint_and_reset(tmp_path):
    """Inlet/outlet cells read density and velocity of the step before, which
    two pairs of buffers hold in turn: calls of odd and even lengths, a write-back
    of both fields, a checkpoint and a reset, against the oracle."""
    flags = cases.plain_channel(90, 26).flags.copy()
    flags[1:-1, 0] = cases.INLET
    flags[1:-1, -1] = cases.OUTLET
    kw = dict(tau=0.7, inlet_ux=0.04, use_force=False)
    s, o = pair(flags, O.F32, E.BB_HALFWAY, E.ARITH_FUSED, **kw)
    for n in (1, 2, 3, 33, 5):
        s.step(n)
        o.step(n)
        check(s, o, O.F32, f"t={o.t}")
    s.write(E.FIELD_RHO, s.rho)
    s.write(E.FIELD_U, s.u)
    s.step(3)
    o.step(3)
    check(s, o, O.F32, "after the write-back")
    path = str(tmp_path / "state.bin")
    s.save_checkpoint(path)
    b = E.Solver(flags, precision=32, bounce_back=E.BB_HALFWAY, arithmetic=E.ARITH_FUSED, **kw)
    b.step(7)
    b.load_checkpoint(path)
    for n in (1, 36):
        b.step(n)
        o.step(n)
        check(b, o, O.F32, f"checkpoint, t={o.t}")
    b.close()
    s.reset(flags)
    o = O.Oracle(flags, O.OracleConfig(variant=O.F32, bb=E.BB_HALFWAY, arithmetic=E.ARITH_FUSED, **kw))
    s.step(35)
    o.step(35)
    check(s, o, O.F32, "after the reset")
    s.close()


def one_step(flags, **kw):
    return E.Solver(flags, kernel_variant=1, **kw)


def same_state(a, b):
    return all(np.array_equal(a.read(f), b.read(f)) for f in (E.FIELD_F, E.FIELD_RHO, E.FIELD_U))


FUSED, REF = dict(arithmetic=E.ARITH_FUSED), dict(arithmetic=E.ARITH_REFERENCE)
TRT, LES = dict(collision=1, use_force=False), dict(subgrid=True)
# every row of the window tables of long calls, with rows of whole vectors and
# not, and the grids for which they name none (several: whether steps share a launch)
LONG = [(32, FUSED, nx, ny, True) for nx, ny in [(129, 128), (128, 64), (201, 200), (200, 200), (601, 301), (600, 300),
                                                 (1401, 401), (1400, 360), (45, 1800), (5001, 20), (10001, 4)]]
LONG += [(32, FUSED, 60001, 4, False)]
LONG += [(32, REF, nx, ny, True) for nx, ny in [(150, 150), (152, 150), (201, 200), (300, 301), (301, 301), (40, 2700),
                                                (41, 2401)]]
LONG += [(32, REF, nx, ny, False) for nx, ny in [(20000, 3), (400, 400)]]
LONG += [(32, TRT, 181, 200, True), (32, LES, 201, 201, True), (32, TRT, 256, 256, False), (32, LES, 301, 230, False), (32, LES, 301, 240, True),
         (32, TRT, 384, 256, True), (32, LES, 4164, 24, False)]
LONG += [(64, FUSED, nx, ny, True) for nx, ny in [(129, 128), (201, 200), (200, 200), (249, 249), (248, 250), (401, 301),
                                                  (400, 300), (1401, 401), (1400, 400), (16664, 6)]]
LONG += [(64, FUSED, nx, ny, False) for nx, ny in [(256, 256), (50001, 3)]]
LONG += [(16, FUSED, nx, ny, True) for nx, ny in [(129, 128), (201, 200), (200, 200), (400, 300), (301, 301), (529, 529),
                                                  (33, 3030)]]
LONG += [(16, TRT, 201, 200, True), (16, TRT, 401, 301, False), (16, LES, 400, 300, True)]
LONG += [(16, FUSED, nx, ny, False) for nx, ny in [(249, 249), (1549, 96), (1877, 117)]]


@pytest.mark.parametrize("prec,kw,nx,ny,several", LONG, ids=lambda v: "-".join(v) if isinstance(v, dict) else str(v))
def test_window_tables_of_long_calls(prec, kw, nx, ny, several):
    flags = cases.channel_with_block(nx, ny, nx // 3, nx // 2, max(2, ny // 3))
    kw = dict(precision=prec, tau=0.6, fx=1e-5, fy=-2e-6, **kw)
    a, b = E.Solver(flags, **kw), one_step(flags, **kw)
    for n in (35, 40):  # from an even and an odd step
        before = a.launches
        a.step(n)
        assert (a.launches - before < n) == several
        b.step(n)
        assert same_state(a, b), n
    a.close()
    b.close()


# calls of fewer steps than the tables of long calls are for: the sizes that the
# first test of this file leaves out
@pytest.mark.parametrize("prec,kw,nx,ny", [(32, REF, 301, 301), (16, FUSED, 201, 200), (16, FUSED, 200, 200),
                                           (32, FUSED, 1023, 255), (64, FUSED, 1023, 255), (16, FUSED, 301, 301),
                                           (32, FUSED, 1401, 401), (64, FUSED, 1401, 401)],
                         ids=lambda v: "-".join(v) if isinstance(v, dict) else str(v))
def test_window_tables_of_short_calls(prec, kw, nx, ny):
    flags = cases.channel_with_block(nx, ny, nx // 3, nx // 2, max(2, ny // 3))
    kw = dict(precision=prec, tau=0.6, fx=1e-5, fy=-2e-6, **kw)
    a, b = E.Solver(flags, **kw), one_step(flags, **kw)
    for n in (13, 2, 33, 4):
        before = a.launches
        a.step(n)
        assert n == 2 or a.launches - before < n
        b.step(n)
        assert same_state(a, b), n
    a.close()
    b.close()


@pytest.mark.parametrize("streams,sizes", [(2, [(64, 40), (61, 39)]), (4, [(101, 61), (96, 48), (33, 20), (200, 64)]),
                                           (8, [(256 + 31 * k, 90 + 7 * k) for k in range(10)])], ids=str)
@pytest.mark.parametrize("arith", [E.ARITH_FUSED, E.ARITH_REFERENCE], ids=["fused", "reference"])
def test_batch_graphs_of_windows(streams, sizes, arith):
    """Streams form: calls long enough to launch a case's graph of windows several
    times, from even and odd steps, against handles of one step per launch."""
    flags = [cases.plain_channel(nx, ny).flags for nx, ny in sizes]
    b = E.Batch([(g, 0.6, 1e-5, 0.0) for g in flags], arithmetic=arith, autotune=0)
    b.set_launch("streams", 1, streams, 0)
    ref = [one_step(g, precision=32, tau=0.6, fx=1e-5, arithmetic=arith) for g in flags]
    for n in (230, 201, 222, 5):
        b.step(n)
        for k, r in enumerate(ref):
            r.step(n)
            for f in (E.FIELD_F, E.FIELD_RHO, E.FIELD_U):
                assert np.array_equal(b.read(k, f), r.read(f)), (n, k, f)
    b.close()
    for r in ref:
        r.close()
