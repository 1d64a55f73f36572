"""The 2D induction solver (spdk_induction2d_*): 2D field-loop advection.

Parity: the reference built with the loop's velocity and centre
(oracle/patch_loop2d.py) and run quasi-2D (nx3 = 2, periodic, B_z = 0) gives
B2_cv fixtures (tests/golden/loop2d_*.npz, made by make_fixtures.py
--loop2d); the FP64 form reproduces them bit for bit, ADER and SSP-RK2,
uniform and non-uniform element sizes. The precision form (FP32 state) is
compared with the FP64 form by their errors against the exact solution (the
initial field translated by v t). The full configuration -- [-1, 1]^2
periodic (as [0, 2]^2 with the loop at (1, 1)), 512^2 elements, p = 4,
v = (2, 1), A_z = 1e-3 (0.3 - r), to t = 1 -- runs in both forms.
"""
import json
import os

import numpy as np
import pytest

from helpers import GOLDEN, field_loop_steps, same_bits

pytestmark = pytest.mark.gpu


def manifest_cases():
    with open(os.path.join(GOLDEN, "manifest.json")) as f:
        return json.load(f).get("loop2d_cases", {})


def config_from_overrides(ov, precision="fp64"):
    from spd_k_b200.induction import field_loop_config
    d = dict(o.split("=", 1) for o in ov)
    c = field_loop_config(N=int(d["mesh/nx1"]), p=int(d["mesh/p"]), precision=precision,
                          integrator=d.get("time/integrator", "ader"))
    c["N"] = [int(d["mesh/nx1"]), int(d["mesh/nx2"])]
    c["L"] = [float(d["mesh/x1len"]), float(d["mesh/x2len"])]
    c["cfl"] = float(d["time/cfl"])
    return c, float(d["time/tlim"]), float(d["output/dt"])


@pytest.mark.parametrize("case", sorted(manifest_cases()))
def test_matches_patched_reference(case):
    from spd_k_b200.induction import Induction2D
    entry = manifest_cases()[case]
    c, tlim, dt_out = config_from_overrides(entry["overrides"])
    s = Induction2D(c)
    steps = s.evolve(tlim, dt_out)
    assert steps == entry["steps"]
    want = np.load(os.path.join(GOLDEN, case + ".npz"))["B2_cv"]
    got = s.b2_cv()
    assert got.shape == want.shape
    assert same_bits(got, want), np.abs(got - want).max()
    s.close()


def loop_error(N, p, t_end, precision):
    """L1 of (Bx, By) sub-cell averages at t_end against the initial field
    translated by v t_end (a whole number of elements here), relative to the
    initial field's L1"""
    from spd_k_b200.induction import Induction2D, field_loop_config
    c = field_loop_config(N=N, p=p, precision=precision)
    s = Induction2D(c)
    b0 = s.b2_cv()
    steps = s.evolve(t_end, t_end)
    b = s.b2_cv()
    s.close()
    L = c["L"][0]
    shift = [int(round(c["velocity"][d] * t_end / (L / N))) % N for d in range(2)]
    exact = np.roll(b0, shift=(shift[1], shift[0]), axis=(1, 2))
    err = [float(np.abs(b[v] - exact[v]).sum() / np.abs(exact[v]).sum()) for v in range(2)]
    return err, steps


def test_fp32_matches_fp64_error():
    """64^2, p = 4, to t = 0.5 (the loop moves by (1, 0.5)): both forms'
    errors against the translated initial field agree to 1 %"""
    e64, n64 = loop_error(64, 4, 0.5, "fp64")
    e32, n32 = loop_error(64, 4, 0.5, "fp32")
    print(f"\nloop 64^2 p=4 t=0.5: fp64 {e64}  fp32 {e32}  ({n64} steps)")
    assert n64 == n32
    for a, b in zip(e64, e32):
        assert a < 0.05
        assert abs(b - a) <= 0.01 * a


def test_field_loop_512_to_t1():
    """the full configuration in both forms: errors against the initial field
    translated by (2, 1), the loop's peak |B|^2 kept, FP32 within 1 % of FP64"""
    res = {}
    for prec in ("fp64", "fp32"):
        res[prec] = loop_error(512, 4, 1.0, prec)
    print(f"\nloop 512^2 p=4 t=1: fp64 {res['fp64']}  fp32 {res['fp32']}")
    (e64, n64), (e32, n32) = res["fp64"], res["fp32"]
    assert n64 == n32
    for a, b in zip(e64, e32):
        assert a < 0.01
        assert abs(b - a) <= 0.01 * a


def against_plain_scheme(Nx, Ny, p, integrator, precision, steps=4):
    from spd_k_b200.induction import FIELD2_BX, FIELD2_BY, Induction2D, field_loop_config
    c = field_loop_config(N=Nx, p=p, precision=precision, integrator=integrator)
    c["N"], c["L"], c["velocity"], c["cfl"] = [Nx, Ny], [2.0, 2.0 * Ny / Nx], (1.3, -0.7), 0.4
    s = Induction2D(c)

    def fields():
        return (s.read(FIELD2_BX).reshape(Ny, Nx, p + 1, p + 2), s.read(FIELD2_BY).reshape(Ny, Nx, p + 2, p + 1))
    start, dt = fields(), s.dt()
    for _ in range(steps):
        s.step()
    got = fields()
    s.close()
    h = [c["L"][0] / Nx, c["L"][1] / Ny]
    want = field_loop_steps(*start, h, c["velocity"], p, integrator, dt, steps)
    # each step re-evaluates derivative sums of 2 (p + 2) terms: the round-off
    # of a value times their condition, at most 8 (p + 1)^2
    eps = 1.2e-7 if precision == "fp32" else 2.3e-16
    for a, b in zip(got, want):
        assert np.abs(a - b).max() <= steps * 8 * (p + 1) ** 2 * eps * np.abs(b).max()


@pytest.mark.parametrize("N,p,integrator", [(2, 2, "ader"), (5, 4, "ader"), (7, 3, "rk2"), (9, 5, "ader"), (11, 1, "rk3")])
def test_counts_that_no_tile_divides(N, p, integrator):
    """tiles hang over the domain's high edges: a few steps against the same
    scheme in plain FP64 numpy"""
    against_plain_scheme(N, N, p, integrator, "fp64")


# both sides of every switch between one-element, 2 x 2 and 4 x 4 tiles
SWITCHES = [(2, "fp64", [(21, 21), (22, 21), (47, 48), (50, 47)]), (3, "fp64", [(21, 21), (23, 20), (58, 59), (59, 60)]),
            (4, "fp64", [(21, 21), (22, 21), (59, 58), (59, 60)]), (4, "fp32", [(21, 21), (22, 21), (73, 72), (74, 73)]),
            (6, "fp64", [(21, 21), (22, 22)]), (7, "fp32", [(24, 24), (25, 24)]), (1, "fp32", [(3, 2), (33, 36), (36, 32)])]


@pytest.mark.parametrize("p,precision,size", [(p, f, n) for p, f, ns in SWITCHES for n in ns])
def test_tile_switches(p, precision, size):
    against_plain_scheme(*size, p, "ader" if size[0] % 2 else "rk3", precision, steps=3)
