"""Kernels compiled for one (n, d) answer for that (n, d) only.  No GPU needed."""
import pytest

# a shape each table has, and shapes whose d does not fit 4 bits beside it
TABLES = {0: (3, 1), 1: (3, 1), 2: (3, 1), 3: (3, 1), 4: (3, 2), 5: (3, 2), 6: (3, 6)}


@pytest.mark.parametrize("table", sorted(TABLES))
def test_tables_answer_only_for_their_own_shapes(table):
    from kronmult_gb300 import _lib

    lookup = _lib.lib().kronmult_diag_compiled_shape
    for n in range(0, 20):
        for d in range(0, 70):
            assert lookup(table, n, d) in (0, n * 100 + d), (n, d)
    n, d = TABLES[table]
    assert lookup(table, n, d) == n * 100 + d
    assert lookup(7, n, d) == -1
