"""Which kernel a forward launches, on both sides of the limits of batch size where the FP32
register blocks give way to the other kernels."""
import pytest

from conftest import planned_kernel

pytestmark = pytest.mark.gpu
F64, F32, F32_F64OUT = 0, 1, 2


@pytest.mark.parametrize("d,n,dtype,nb,tuning,kernel", [
    (6, 2, F32, 1000, None, "fwd_pair_kernel"), (6, 2, F32, 60000, None, "fwd_block_kernel"),
    (2, 3, F32, 1000, None, "fwd_block_kernel"), (2, 3, F32, 5000, None, "fwd_smem_kernel"),
    (6, 4, F32, 2000, None, "fwd_tri4_kernel"), (6, 4, F32, 3000, None, "fwd_block_kernel"),
    (4, 8, F32, 1000, None, "fwd_pair8_kernel"), (4, 8, F32, 1200, None, "fwd_block_kernel"),
    (4, 8, F32_F64OUT, 3000, None, "fwd_pair8_kernel"), (4, 8, F32_F64OUT, 4500, None, "fwd_block_kernel"),
    (6, 4, F32_F64OUT, 3000, None, "fwd_tri4_kernel"), (3, 9, F32, 400, None, "fwd_block_kernel"),
    (4, 8, F32, 1200, {"team_size": 256}, "fwd_smem_kernel"), (6, 8, F32, 100, None, "fwd_block_kernel"),
    (4, 4, F32, 12000, None, "fwd_pair_kernel"), (4, 4, F32, 16000, None, "fwd_block_kernel"),
    (5, 4, F32_F64OUT, 6000, None, "fwd_pair_kernel"), (5, 4, F32_F64OUT, 12000, None, "fwd_block_kernel"),
    (3, 10, F64, 2000, None, "fwd_f64_kernel"), (9, 3, F64, 8, None, "fwd_global_kernel"),
])
def test_kernel(cuda, d, n, dtype, nb, tuning, kernel):
    assert kernel in planned_kernel(d, n, dtype, nb, tuning)
