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


@pytest.mark.parametrize("max_smem", [16 << 10, 48 << 10, 99 << 10, 163 << 10, 227 << 10])
def test_adjoint_blocks_have_the_shared_memory_of_their_threads(max_smem):
    """Also where a GPU has less shared memory than one CTA's groups would take."""
    import ctypes

    from kronmult_gb300 import _lib

    lib = _lib.lib()
    halved = 0
    for n in range(2, 9):
        for d in range(2, 9):
            for nb in (1, 200, 5000, 100000):
                s = (ctypes.c_longlong * 6)()
                if lib.kronmult_diag_adjoint_block_shape(n, d, nb, 152, max_smem, s) != 0:
                    continue
                fits, groups, threads, smem, group_threads, group_smem = s
                assert threads == groups * group_threads and smem == groups * group_smem
                assert fits == (smem <= max_smem) and (fits or groups == 1)
                whole = (ctypes.c_longlong * 6)()
                lib.kronmult_diag_adjoint_block_shape(n, d, nb, 152, 1 << 30, whole)
                halved += groups < whole[1]
    assert (halved > 0) == (max_smem < 213056)  # the largest CTA: d = 4, n = 8
