"""FP32 outputs of many entries: the FP32 forward adds them in short partial sums, not in one
chain of additions per team.

Tolerance: one rounding has a root-mean-square error of at most 2^-24 / sqrt(3) of the value, and
the partial values of a sum of m like terms have mean squares m / 2 of the whole's, so
    2^-24 / sqrt(3) * sqrt(roundings of an entry + 8 / 2 + (sums of at least 6 entries) / 2)
where the d modes of n additions count as d * n roundings of the whole."""
import math

import pytest
import torch

from conftest import planned_kernel

pytestmark = pytest.mark.gpu


def _error(cuda, d, n, outputs, fan, tuning):
    from kronmult_gb300 import DeviceBatch

    gen = torch.Generator(device=cuda)
    gen.manual_seed(17)
    N, nb = n ** d, outputs * fan
    factors = (torch.rand((outputs * d, n * n), generator=gen, device=cuda) * 2 - 1) / n ** 0.5
    x = torch.randn((nb, N), generator=gen, device=cuda)
    index = torch.arange(outputs, device=cuda).repeat_interleave(fan)
    db = DeviceBatch(d, n, n, factors, x, torch.zeros((outputs, N), device=cuda), index, index)
    db.forward(tuning=tuning)
    # an output's entries share their factors: K (x_1 + x_2 + ..), in 64 bits
    want = x.view(outputs, fan, N).sum(dim=1, dtype=torch.float64)
    mats = factors.double().view(outputs, d, n, n).transpose(-1, -2)  # [r, k]
    for i in range(d):
        want = torch.matmul(mats[:, i].unsqueeze(1), want.view(outputs, n ** i, n, -1)).reshape(outputs, N)
    return float((db.outputs.double() - want).norm() / want.norm())


@pytest.mark.parametrize("d,n,outputs", [(2, 3, 25), (4, 4, 4), (5, 3, 4), (3, 6, 10), (3, 8, 4), (3, 10, 4)])
def test_long_shares(cuda, d, n, outputs):
    """1000 entries per output, hundreds per team."""
    tuning = {"entries_per_team": 1000}
    assert "fwd_block_kernel" in planned_kernel(d, n, 1, outputs * 1000, tuning)
    tol = 2.0 ** -24 / math.sqrt(3) * math.sqrt(d * n + 8 / 2 + 1000 / 6 / 2)
    assert _error(cuda, d, n, outputs, 1000, tuning) <= tol


def test_long_shares_of_a_wave(cuda):
    """d = 6, n = 4: one team per SM with 256 entries of one output."""
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    assert "fwd_block_kernel" in planned_kernel(6, 4, 1, sms * 256, {"ctas_per_sm": 1})
    tol = 2.0 ** -24 / math.sqrt(3) * math.sqrt(24 + 8 / 2 + 256 / 6 / 2)
    assert _error(cuda, 6, 4, sms, 256, {"ctas_per_sm": 1}) <= tol
