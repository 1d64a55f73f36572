"""The benchmark's byte model against a count of the arrays each kernel of the
fallback names (no GPU)."""
from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("D,p,nt,esz", [(2, 3, 4, 8), (2, 3, 4, 4), (3, 2, 3, 8), (2, 1, 1, 4)])
def test_fallback_bytes_count_each_array_once(D, p, nt, esz):
    import bench
    E, n = 48, p + 1
    npt, V = n ** D, D + 2
    b = bench.algorithmic_bytes(SimpleNamespace(n_elements=E, nvar=V, n_points=npt, n_time_slices=nt, ndim=D, p=p),
                                True, esz)
    state, pair = E * V * npt * esz, E * npt * 16
    faces = D * E * V * n ** (D - 1) * (n + 1) * esz
    total = 0
    for t in range(nt):
        total += state + faces                                   # U_cv and the faces of slice t
        total += state + faces + 2 * pair if t < nt - 1 else 2 * state
    assert b["update"] * nt == pytest.approx(total, rel=1e-12)
    assert b["detect"] == 2 * pair + 2 * E * npt                 # candidates in; flags and cleared theta out
    assert "theta" not in b
