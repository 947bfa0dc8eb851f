"""The CSR solver's workspace size (no GPU needed): what the solver lays out fits, and a
restart beyond the system's rows asks for no more than the columns that are used."""
import pytest

CASES = [(1, 100), (2, 2), (600, 100), (13824, 100), (600, 1), (600, 100000), (100, 2000000),
         (3000, 3000), (3600, 3600), (5000, 100000), (20000, 9000), (200001, 300)]


def _bytes(n, method, restart):
    from tcad_b200 import _lib
    return _lib.load(require_gpu=False).tcad_csr_workspace_bytes(n, method, restart)


def _without_h(n, method, m):
    """Block inverses, vectors, partial sums of m + 1 columns, coefficients, slack."""
    return 8 * (9 * n + (8 * n if method == 0 else (m + 4) * n) + 4096 * 4 + 64 + 32
                + 4096 * (m + 1) + (m + 1) + n) + (1 << 20)


@pytest.mark.parametrize("n,restart", CASES)
def test_gmres_layout_fits(n, restart):
    m = min(restart, n)
    parts = [9 * n, 4096 * 4, 64, 32, (m + 1) * n, n, n, n, n, 592 * (m + 1), m * (m + 1)] \
        + [m + 1] * 5
    assert sum(-(-8 * p // 256) * 256 for p in parts) <= _bytes(n, 1, restart)


@pytest.mark.parametrize("n,restart", CASES)
def test_h_counts_only_where_it_is_larger_than_the_partials_leave(n, restart):
    m = min(restart, n)
    assert _bytes(n, 0, restart) == _without_h(n, 0, restart)
    extra = _bytes(n, 1, restart) - _without_h(n, 1, restart)
    assert extra == max(0, 8 * ((m + 1) * (m + 5) - 3504 * (restart + 1)))
    if m <= 3498:
        assert extra == 0
