"""Free-surface super-tile lists against the CPU oracle on grids whose last
super-tile column or row is one or two cells wide, and on grids with super-tiles
of plain fluid, with liquid that crosses the periodic edges: every field equal."""
import numpy as np
import pytest

from conftest import exact_equal, first_mismatch
from flowlb_b200 import cases
from flowlb_b200 import engine as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("f", "rho", "u", "flags", "mass", "excess", "phi")


def blobs(nx, ny, walls):
    """Liquid around the periodic corner and in the middle, gas elsewhere."""
    y, x = np.mgrid[0:ny, 0:nx]
    dx, dy = np.minimum(x, nx - x) / nx, np.minimum(y, ny - y) / ny
    flags = np.full((ny, nx), cases.GAS, np.uint8)
    flags[(dx < 0.3) & (dy < 0.35)] = cases.FLUID
    flags[(np.abs(x - 0.55 * nx) < 0.08 * nx) & (np.abs(y - 0.6 * ny) < 0.2 * ny)] = cases.FLUID
    if walls:
        flags[0, :] = cases.WALL
        flags[ny // 3:ny // 3 + 2, nx // 4:nx // 4 + 3] = cases.WALL
    return flags


def oracle_fields(o, prec):
    f = o.f64()
    return dict(f=f if prec == 64 else f.astype(np.float32), rho=o.rho, u=o.u, flags=o.flags, mass=o.mass,
                excess=o.excess, phi=o.phi)


# thin in x, in y, in both, in neither; up to 512, 1024 and more super-tiles
@pytest.mark.parametrize("nx,ny", [(65, 10), (130, 21), (66, 9), (3, 17), (96, 3), (321, 402), (1601, 265),
                                   (2113, 266), (2176, 520)], ids=lambda v: str(v))
@pytest.mark.parametrize("prec,walls,mode", [(32, False, E.STEP_KERNELS), (64, True, E.STEP_KERNELS),
                                             (16, True, E.STEP_KERNELS), (32, True, E.STEP_PERSISTENT)],
                         ids=["f32", "f64-walls", "f16s-walls", "f32-walls-persistent"])
def test_lists_match_oracle(nx, ny, prec, walls, mode):
    flags = blobs(nx, ny, walls)
    kw = dict(tau=0.56, fx=3e-4, fy=-2e-4, u_max=0.25)
    s = E.Solver(flags, free_surface=True, precision=prec, mass_precision=64, bounce_back=E.BB_HALFWAY,
                 fs_mode=E.FS_CONSERVATIVE, arithmetic=E.ARITH_FUSED, **kw)
    s.set_step_mode(mode)
    variant = {32: O.F32, 64: O.F64, 16: O.F16S}[prec]
    o = O.Oracle(flags, O.OracleConfig(variant=variant, free_surface=True, bb=O.BB_HALFWAY,
                                       fs_mode=O.FS_CONSERVATIVE, arithmetic=O.ARITH_FUSED, **kw))
    for n in (1, 2, 5, 60):
        s.step(n)
        o.step(n)
        want = oracle_fields(o, prec)
        for name in FIELDS:
            a = getattr(s, name)
            assert exact_equal(a, want[name]), f"t={o.t} {name}: {first_mismatch(a, want[name])}"
    if mode == E.STEP_KERNELS:
        s.set_step_mode(E.STEP_PERSISTENT)  # the other form takes over the lists
        s.step(34)
        o.step(34)
        want = oracle_fields(o, prec)
        for name in FIELDS:
            a = getattr(s, name)
            assert exact_equal(a, want[name]), f"t={o.t} {name}: {first_mismatch(a, want[name])}"
    s.close()
    o.close()


# plain-fluid super-tiles (grids of more than 1,024) under the options that the
# cases above leave out: FlowLB's free-surface rules, implicit walls, FP32 mass,
# the reference arithmetic, the subgrid model
@pytest.mark.parametrize("variant,kw", [
    (O.F32_M32, dict(fs_mode=E.FS_REFERENCE, bb=E.BB_IMPLICIT, arith=E.ARITH_REFERENCE)),
    (O.F32_M32, dict(fs_mode=E.FS_REFERENCE, bb=E.BB_IMPLICIT, arith=E.ARITH_REFERENCE, subgrid=True)),
    (O.F32, dict(fs_mode=E.FS_CONSERVATIVE, bb=E.BB_HALFWAY, arith=E.ARITH_FUSED, subgrid=True)),
    (O.F32_M32, dict(fs_mode=E.FS_CONSERVATIVE, bb=E.BB_IMPLICIT, arith=E.ARITH_FUSED)),
    (O.F64, dict(fs_mode=E.FS_REFERENCE, bb=E.BB_IMPLICIT, arith=E.ARITH_REFERENCE)),
    (O.F16S, dict(fs_mode=E.FS_REFERENCE, bb=E.BB_IMPLICIT, arith=E.ARITH_FUSED)),
], ids=["ref-m32", "ref-m32-subgrid", "f32-subgrid", "implicit-m32", "ref-f64", "ref-f16s"])
@pytest.mark.parametrize("nx,ny", [(2113, 266), (2176, 520)], ids=str)
def test_plain_fluid_super_tiles_under_other_options(variant, kw, nx, ny):
    kw = dict(kw)
    bb, arith = kw.pop("bb"), kw.pop("arith")
    kw.update(tau=0.56, fx=3e-4, fy=-2e-4, u_max=0.25)
    flags = blobs(nx, ny, True)
    prec = {O.F64: 64, O.F16S: 16}.get(variant, 32)
    s = E.Solver(flags, free_surface=True, precision=prec, mass_precision=32 if variant == O.F32_M32 else 64,
                 bounce_back=bb, arithmetic=arith, **kw)
    s.set_step_mode(E.STEP_KERNELS)
    o = O.Oracle(flags, O.OracleConfig(variant=variant, free_surface=True, bb=bb, arithmetic=arith, **kw))
    for n in (1, 2, 5, 40):
        s.step(n)
        o.step(n)
        want = oracle_fields(o, prec)
        for name in FIELDS:
            a = getattr(s, name)
            assert exact_equal(a, want[name]), f"t={o.t} {name}: {first_mismatch(a, want[name])}"
    s.close()
    o.close()


def test_fp16_listed_paths_agree_on_a_large_grid():
    """FP16 storage above 8,192 super-tiles: the default stream-collide against the vector one."""
    flags = blobs(4160, 1040, True)
    kw = dict(free_surface=True, precision=16, tau=0.56, fx=3e-4, fy=-2e-4, u_max=0.25)
    a, b = E.Solver(flags, **kw), E.Solver(flags, kernel_variant=2, **kw)
    for n in (3, 40):
        a.step(n)
        b.step(n)
        for name in FIELDS:
            assert exact_equal(getattr(a, name), getattr(b, name)), name
    a.close()
    b.close()
