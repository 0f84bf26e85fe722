"""Tensor-core forward, d = 4: batches of one to two waves of chunks, where a CTA walks several,
and of more, where each has one."""
import pytest
import torch

from test_tc_chunks_gpu import test_tail_of_a_large_batch as check_tail

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("chunks_per_sm", [7, 9, 18])
@pytest.mark.parametrize("compute", [1, 2, 3])
def test_chunks(cuda, compute, chunks_per_sm, off):
    """5, 6 and 8 CTAs per SM (split BF16, TF32, BF16); chunks of 8 entries, the last one ragged."""
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    check_tail(cuda, 4, sms * chunks_per_sm * 8 - 3, compute, 5, off)
