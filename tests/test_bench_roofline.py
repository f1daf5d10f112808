"""The bytes bench.py charges a pressure solve are those of the kernels that ran:
none where the vectors stay on chip, what does not fit where they are streamed."""
from types import SimpleNamespace

import pytest

from test_bench_replicas import _bench


def _solve(pf, tiles, **cfg):
    st = SimpleNamespace(iterations=100, refinements=2, solve_ms=1.0, n_cells=1000)
    return _bench().pcg_roofline(pf, pf.SolverConfig(**cfg), st, tiles, 6448.0)


@pytest.mark.parametrize("tiles,per", [(1, None), (888, None), (889, 64.0), (12 * 148, 64.0), (24 * 148, 96 - 16 * 29 / 24),
                                       (28 * 148, 96 - 16 * 24 / 28), (49 * 148, 96.0), (49 * 148 + 1, 139.0),
                                       (35937, 139.0)])
def test_plain_bytes_follow_the_path(pf, tiles, per):
    r = _solve(pf, tiles)
    if per is None:
        assert "frac" not in r and r["us_per_iteration"] == 10.0
    else:
        assert r["bytes_per_unknown"] == pytest.approx(100 * per)
        assert r["frac"] == pytest.approx(100 * per * 1000 / 1e-3 / 1e9 / 6448.0)


def test_mixed_and_learned_bytes(pf):
    mixed = dict(mode=pf.PF_SOLVER_MIXED, bf16_storage=1)
    assert "frac" not in _solve(pf, 1184, **mixed)
    assert _solve(pf, 1185, **mixed)["bytes_per_unknown"] == 65 * 100 + 165 * 2
    assert _solve(pf, 100, mode=pf.PF_SOLVER_LEARNED)["bytes_per_unknown"] == 133 * 100
