"""Shared test helpers: run a configuration given as block/name=value
overrides through the oracle (CPU checker) or the GPU solver with the
reference's time loop, and compare states bit for bit."""
import hashlib
import json
import os

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
GOLDEN = os.path.join(HERE, "golden")


def manifest():
    with open(os.path.join(GOLDEN, "manifest.json")) as f:
        return json.load(f)


def fixture(name):
    return np.load(os.path.join(GOLDEN, name + ".npz"))["W_cv"]


def oracle_config(overrides):
    from oracle import oracle as O
    return O.config_from_params(O.apply_overrides({}, overrides))


def gpu_config(overrides):
    from spd_k_b200.api import apply_overrides, config_from_params
    return config_from_params(apply_overrides({}, overrides))


def oracle_active(o, name="W_cv"):
    """oracle array -> active region (5, Nz, Ny, Nx, nz, ny, nx)."""
    a = o.array(name)[0]
    a = a[:, 1:-1] if a.shape[1] > 1 else a
    return np.ascontiguousarray(a[:, :, 1:-1, 1:-1])


def oracle_run(overrides):
    """(W_cv of the last output, steps, oracle) through the reference loop."""
    from oracle import oracle as O
    c = oracle_config(overrides)
    o = O.Oracle(c)
    out = {}
    o.run(c["tlim"], c["output_dt"], on_output=lambda n, s: out.__setitem__(n, s.array("W_cv")))
    last = out[max(out)]
    a = last[0]
    a = a[:, 1:-1] if a.shape[1] > 1 else a
    return np.ascontiguousarray(a[:, :, 1:-1, 1:-1]), o.n_step, o, last


def reference_file_bytes(w_full):
    """Reference-format W_cv dump (6 slots; slot 5 is identically zero) from
    an oracle W_cv array of shape (1, 5, ...)."""
    full = np.zeros((1, 6) + w_full.shape[2:], dtype=np.float64)
    full[:, :5] = w_full
    return full.tobytes()


def sha256_bytes(b):
    return hashlib.sha256(b).hexdigest()


def gpu_run(overrides, device=0):
    """(W_cv at the last output in reference slot order, steps, solver)."""
    import spd_k_b200 as S
    c = gpu_config(overrides)
    g = S.HydroSolver(c, device=device)
    out = {}
    g.run(c["tlim"], c["output_dt"],
          on_output=lambda n, s: out.__setitem__(n, s.to_reference_slots(s.field_array(S.FIELD_W_CV))))
    return out[max(out)], g.n_step, g


def same_bits(a, b):
    """Equal as IEEE values, NaN matching NaN (signed zeros compare equal)."""
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return a.shape == b.shape and bool(np.all((a == b) | (np.isnan(a) & np.isnan(b))))


def rel_l1(a, b):
    """relative L1 difference per conserved/primitive slot"""
    return [float(np.abs(a[v] - b[v]).sum() / max(np.abs(a[v]).sum(), 1e-300)) for v in range(a.shape[0])]


def scheme_matrices(p, ader):
    """the scheme's matrices as spdk_build_matrices gives them (tests/test_host_abi.py checks their bits)"""
    import ctypes
    import spd_k_b200 as S
    n, nf, nt = p + 1, p + 2, p + 1 if ader else 1
    m = {"sp_to_fp": np.zeros((nf, n)), "dfp_to_sp": np.zeros((n, nf)), "sp_to_cv": np.zeros((n, n)),
         "cv_to_sp": np.zeros((n, n)), "invader": np.zeros((nt, nt)), "wt": np.zeros(nt)}
    L = S.load_library()
    L.spdk_build_matrices.argtypes = [ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 6
    assert L.spdk_build_matrices(p, int(ader), *(a.ctypes.data for a in m.values())) == 0
    return m


def field_loop_steps(Bx, By, h, v, p, integrator, dt, steps):
    """2D induction steps of the spectral-difference scheme in plain FP64 numpy
    (periodic): Bx [j][i][jj][ix], By [j][i][jy][ii]; E_z = v_x B_y - v_y B_x at
    the edge points, upwinded across x, then y interfaces; dB/dt = curl E"""
    ader = integrator == "ader"
    M = scheme_matrices(p, ader)
    S, D, wt = M["sp_to_fp"], M["dfp_to_sp"], M["wt"]
    nt = len(wt)

    def upwind(a, b, vel):
        return 0.5 * (a + b) if vel == 0 else (a if vel > 0 else b)

    def rate(B):
        E = v[0] * (B[1] @ S.T) - v[1] * (S @ B[0])
        q = upwind(np.roll(E[..., -1], 1, 1), E[..., 0], v[0])
        E[..., 0], E[..., -1] = q, np.roll(q, -1, 1)
        q = upwind(np.roll(E[:, :, -1], 1, 0), E[:, :, 0], v[1])
        E[:, :, 0], E[:, :, -1] = q, np.roll(q, -1, 0)
        return -(D @ E) / h[1], (E @ D.T) / h[0]

    B = (Bx, By)
    weights = [0.0] if ader else {1: [0.0], 2: [0.0, 0.5], 3: [0.0, 0.75, 1.0 / 3.0]}[int(integrator[2])]
    for _ in range(steps):
        B0 = B
        for a in weights:
            slices = [B] * nt
            for _ in range(nt - 1):
                r = [rate(q) for q in slices]
                slices = [tuple(B[i] - sum(r[l][i] * (M["invader"][t, l] * wt[l] * dt) for l in range(nt))
                                for i in range(2)) for t in range(nt)]
            r = [rate(q) for q in slices]
            B = tuple(B[i] - sum(r[l][i] * (wt[l] * dt) for l in range(nt)) for i in range(2))
            B = tuple(a * B0[i] + (1 - a) * B[i] for i in range(2)) if a else B
    return B
