"""Element counts that no tile divides: the 2D Picard pass runs 4 x 4 (above
p = 3: 4 x 2) element tiles that hang over the domain's high edges, the 3D pass
blocks of 8, 4, 2 or 1 consecutive elements, the fallback its own tiles, and
spacings that are no power of two take the division by h from its reciprocal.
The plain form against the oracle, bit for bit; the precision form against
the plain form."""
import zlib

import numpy as np
import pytest

from helpers import gpu_config, oracle_active, oracle_config, rel_l1, same_bits
from test_gpu_parity import load_oracle_state, random_state, solver

pytestmark = pytest.mark.gpu

# one element past a tile, one short of it, less than one tile, whole tiles
SIZES = [(2, 2), (3, 5), (5, 3), (4, 6), (9, 7)]
EDGES = ["periodic", "gradfree", "reflective"]


def overrides(p, nx, ny, bc, fallback=True, integrator="ader"):
    return [f"mesh/p={p}", f"mesh/nx1={nx}", f"mesh/nx2={ny}", "mesh/nx3=1", f"mesh/x1_bc={bc[0]}",
            f"mesh/x2_bc={bc[1]}", f"job/fallback={str(fallback).lower()}", f"time/integrator={integrator}"]


def against_oracle(ov, mine, ref5, D, steps=2):
    from oracle import oracle as O
    g, o = solver(ov), O.Oracle(oracle_config(ov))
    g.write_u(mine)
    load_oracle_state(o, ref5, D)
    dt = o.compute_dt()
    assert g.dt() == dt
    for step in range(steps):
        o.step(dt)
        g.step()
        dt = o.compute_dt()
        assert g.dt() == dt, step
        for name, field in (("U_sp", 0), ("W_cv", 1)):
            wo, wg = oracle_active(o, name), g.to_reference_slots(g.field_array(field))
            assert same_bits(wg, wo), (step, name, rel_l1(wo, wg))
    g.close()


@pytest.mark.parametrize("p", range(1, 8))
@pytest.mark.parametrize("size", SIZES)
def test_ragged_counts_match_the_oracle(p, size):
    k = zlib.crc32(repr((p, size)).encode())
    bc = (EDGES[k % 3], EDGES[(k // 3) % 3])
    integrator = ["ader", "ader", "rk2"][(k // 9) % 3]
    ov = overrides(p, *size, bc, fallback=k % 2 == 0, integrator=integrator)
    if integrator == "ader" and k % 5 == 0:
        ov.append("hydro/g2=-0.3")
    against_oracle(ov, *random_state(gpu_config(ov), seed=k))


# what the draws above leave out: gravity where a thread finishes two variables
# (p <= 3) and where one does (above), the fallback's RK stages at every kind
# of tile, and the viscous pass on odd counts
EXPLICIT = ([(p, size, fb, "ader", "hydro/g2=-0.3") for p in (2, 3) for size in ((5, 3), (9, 7)) for fb in (False, True)] +
            [(p, (5, 6), fb, "ader", "hydro/g2=-0.3") for p in (1, 5, 6, 7) for fb in (False, True)] +
            [(p, (7, 5), True, "rk2", "hydro/g1=0.2") for p in (1, 2, 3, 5)] +
            [(p, size, fb, "ader", "hydro/nu=0.01") for p, fb in ((1, True), (2, False), (3, True), (5, False), (7, True))
             for size in ((5, 3), (3, 7))] +
            [(3, (7, 9), True, "rk3", "hydro/nu=0.01")])


@pytest.mark.parametrize("p,size,fallback,integrator,extra", EXPLICIT)
def test_gravity_viscosity_and_stages_on_ragged_counts(p, size, fallback, integrator, extra):
    ov = overrides(p, *size, ("gradfree", "reflective"), fallback=fallback, integrator=integrator) + [extra]
    against_oracle(ov, *random_state(gpu_config(ov), seed=zlib.crc32(repr((p, size, extra)).encode())))


@pytest.mark.parametrize("p", range(1, 6))
@pytest.mark.parametrize("size", [(2, 2, 2), (3, 2, 5), (5, 3, 2)])
def test_ragged_counts_match_the_oracle_3d(p, size):
    k = zlib.crc32(repr((p, size)).encode())
    ov = overrides(p, size[0], size[1], (EDGES[k % 3], EDGES[(k // 3) % 3]), fallback=k % 2 == 0,
                   integrator=["ader", "ader", "rk2"][(k // 9) % 3])
    ov[3] = f"mesh/nx3={size[2]}"
    ov.append(f"mesh/x3_bc={EDGES[(k // 27) % 3]}")
    if k % 5 < 2:
        ov.append("hydro/g3=-0.3")
    against_oracle(ov, *random_state(gpu_config(ov), seed=k), steps=1 if p == 5 else 2)


# both sides of the switch to one block per SM in 3D (148 elements)
@pytest.mark.parametrize("p,size,integrator,extra", [(5, (6, 5, 5), "ader", "hydro/g3=-0.3"), (5, (7, 7, 3), "rk2", "hydro/nu=0.01"),
                                                     (5, (5, 5, 5), "rk3", "hydro/g1=0.2"), (5, (3, 4, 5), "ader", "hydro/nu=0.01")])
def test_both_3d_launches(p, size, integrator, extra):
    ov = overrides(p, size[0], size[1], ("gradfree", "reflective"), fallback=False, integrator=integrator) + [extra]
    ov[3] = f"mesh/nx3={size[2]}"
    against_oracle(ov, *random_state(gpu_config(ov), seed=p), steps=1)


# both sides of the switches between the detection's tiles at p = 4 (148 blocks of
# 2 x 2 elements)
@pytest.mark.parametrize("size", [(24, 24), (25, 24)])
def test_both_detection_tiles(size):
    ov = overrides(4, *size, ("gradfree", "periodic"))
    against_oracle(ov, *random_state(gpu_config(ov), seed=size[0]), steps=1)


# both sides of the switches between the 2D passes' kernels: small tiles up to 64
# of them (above p = 4), correctors for few blocks up to 296 (above p = 4: 128)
LAUNCHES = [(5, (16, 16), "ader"), (5, (17, 16), "ader"), (5, (16, 17), "rk2"), (7, (16, 16), "rk2"), (6, (17, 15), "rk3"),
            (7, (33, 31), "rk2"), (6, (31, 34), "ader"), (5, (33, 32), "rk2"), (3, (72, 66), "rk2"), (2, (73, 69), "rk3"),
            (2, (68, 68), "rk2"), (1, (69, 72), "ader"), (4, (46, 50), "ader"), (4, (51, 49), "rk2")]


@pytest.mark.parametrize("p,size,integrator", LAUNCHES)
def test_both_sides_of_every_kernel_switch(p, size, integrator):
    ov = overrides(p, *size, ("reflective", "periodic"), fallback=False, integrator=integrator)
    against_oracle(ov, *random_state(gpu_config(ov), seed=p), steps=1)


@pytest.mark.parametrize("scale", [1e-160, 1e-300, 1e80])
def test_fluxes_too_small_or_large_for_the_reciprocal(scale):
    """momenta (and with them flux values) of this size leave the range in
    which a quotient from 1/h is exact: the tile divides"""
    ov = overrides(3, 5, 6, ("periodic", "gradfree"), fallback=False)
    mine, ref5, D = random_state(gpu_config(ov), seed=3)
    mine[:, :, :, 1:3] *= scale
    ref5[1:3] *= scale
    against_oracle(ov, mine, ref5, D, steps=1)


@pytest.mark.parametrize("p,size", [(2, (7, 6)), (3, (6, 5)), (5, (5, 7)), (5, (17, 18)), (7, (5, 6)),
                                    (2, (63, 63)), (2, (66, 62)), (3, (65, 63))])
def test_precision_form_on_ragged_counts(p, size):
    """FP32 round-off only (as the aligned counts): smooth flow, 4 steps"""
    ov = overrides(p, *size, ("periodic", "periodic"), fallback=False) + ["time/cfl=0.4"]
    g64, g32 = solver(ov, precision="fp64"), solver(ov, precision="fp32")
    for _ in range(4):
        g64.step()
        g32.step()
    a, b = g64.field_array(0), g32.field_array(0)
    assert max(np.abs(b[v] - a[v]).sum() / np.abs(a[v]).sum() for v in range(4)) < 3e-6
    g64.close()
    g32.close()


@pytest.mark.parametrize("p,size", [(1, (5, 3)), (2, (5, 7)), (3, (6, 5)), (4, (3, 6)), (5, (5, 3)), (7, (3, 5)),
                                    (2, (3, 2, 5)), (3, (5, 3, 2)), (4, (3, 2, 3)), (5, (2, 3, 3)), (4, (5, 6, 5))])
def test_precision_form_does_not_see_where_a_tile_ends(p, size):
    """FP32 with the fallback, from a random state: a periodic box on counts that
    hang over its tiles against the same box repeated to whole tiles, whose
    elements then sit elsewhere in theirs. Spacings are 1/8, so that only the
    sub-cell widths round differently (the last FP64 bit of a difference of
    faces, seldom one of its FP32 value): a flux difference of relative 6e-8 a
    step, on values of order one."""
    D = len(size)
    reps = (4,) * D if D == 2 else (2,) * D

    def run(N, u):
        ov = [f"mesh/p={p}", "time/cfl=0.4", "job/fallback=true"]
        for d in range(3):
            ov += [f"mesh/nx{d + 1}={N[d] if d < D else 1}", f"mesh/x{d + 1}_bc=periodic",
                   f"mesh/x{d + 1}len={N[d] / 8 if d < D else 1}"]
        g = solver(ov, precision="fp32")
        if u is None:
            from test_gpu_precision import random_u
            u = random_u(g, seed=p).astype(np.float32).astype(np.float64)
        g.write_u(u)
        for _ in range(2):
            g.step()
        out = g.read(0).reshape(*N[::-1], -1)
        flagged = g.read(4).any()
        g.close()
        return u.reshape(*N[::-1], -1), out, flagged
    start, small, flagged = run(size, None)
    k = reps[::-1] + (1,)
    _, large, _ = run(tuple(n * r for n, r in zip(size, reps)), np.tile(start, k))
    assert flagged
    assert np.abs(large - np.tile(small, k)).max() <= 2 * 16 * 6e-8 * np.abs(small).max()
