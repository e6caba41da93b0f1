"""Single-phase steps that the caller captures into a CUDA graph of their own and
replays between direct calls, against the CPU oracle: every value of the
population array, density and velocity equal."""
import numpy as np
import pytest

from flowlb_b200 import cases
from flowlb_b200 import engine as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("captured", [2, 34])
@pytest.mark.parametrize("prec,io", [(32, False), (64, False), (16, False), (32, True)],
                         ids=["f32", "f64", "f16s", "f32-inlet"])
def test_replays_between_direct_calls_match_oracle(prec, io, captured):
    import torch

    flags = cases.channel_with_block(101, 45, 30, 44, 15)
    kw = dict(tau=0.58, fx=2e-5, fy=-1e-5)
    if io:
        flags[1:-1, 0] = cases.INLET
        flags[1:-1, -1] = cases.OUTLET
        flags[20, 20] = cases.GAS  # never written: its density and velocity stay
        kw = dict(tau=0.7, inlet_ux=0.04, use_force=False)
    variant = {64: O.F64, 32: O.F32, 16: O.F16S}[prec]
    cfg = O.OracleConfig(variant=variant, bb=O.BB_HALFWAY, arithmetic=O.ARITH_FUSED, **kw)
    st = torch.cuda.Stream()
    s = E.Solver(flags, precision=prec, bounce_back=E.BB_HALFWAY, arithmetic=E.ARITH_FUSED, stream=st.cuda_stream, **kw)
    o = O.Oracle(flags, cfg)
    graph = torch.cuda.CUDAGraph()

    def direct(n):
        s.step(n)
        o.step(n)

    def replay():
        with torch.cuda.stream(st):
            graph.replay()
        o.step(captured)

    def check(what):
        f = o.f64() if variant == O.F64 else o.f64().astype(np.float32)
        for name, a, b in (("f", s.f, f), ("rho", s.rho, o.rho), ("u", s.u, o.u)):
            assert np.array_equal(a, b), f"{what}: {name} differs at {np.flatnonzero(a != b)[:5]}"

    direct(20)
    with torch.cuda.graph(graph, stream=st):
        s.step(captured)
    replay()
    check("first replay")
    for n in (20, 2, 36):  # an odd and an even number of launches of several steps
        direct(n)
        check(f"direct {n}")
        replay()
        replay()
        check(f"replays after direct {n}")
    rho = s.rho
    rho[flags.ravel() != cases.FLUID] += 0.25  # the cells that no step writes among them
    s.write(E.FIELD_RHO, rho)
    o.rho[:] = rho
    replay()
    check("replay after a write")
    direct(3)
    direct(1)
    check("direct after a write")
    s.reset(flags)
    o = O.Oracle(flags, cfg)
    replay()
    check("replay after a reset")
    del graph
    s.close()
