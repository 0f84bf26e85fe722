"""The FP64 forward for short vectors: with one entry per output every value is, bit for bit,
that of the other FP64 kernels (forced by a tuning field), for one, two and four elements per
thread, a last CTA that is not full, odd strides and n^d from 2 to 2048; runs of entries with
one output are checked against the oracle (d n additions per value, fan more into the output,
each within 2^-53, with a factor 8 for the cancellation of random signs)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2), (5, 2), (11, 2), (2, 3), (4, 3), (6, 3), (3, 4), (5, 4), (2, 5), (4, 5), (3, 6), (4, 6), (2, 7), (3, 7),
          (2, 8), (3, 8), (1, 9), (3, 9), (1, 10), (2, 10), (3, 10)]


def _run(cuda, d, n, stride, nb, n_out, tuning=None):
    from kronmult_gb300 import DeviceBatch

    g = torch.Generator(device=cuda).manual_seed(n * 100 + d)
    f = (torch.rand((nb * d, stride * n), generator=g, device=cuda, dtype=torch.float64) * 2 - 1) / n ** 0.5
    x = torch.randn((nb, n ** d), generator=g, device=cuda, dtype=torch.float64)
    o = torch.zeros((n_out, n ** d), device=cuda, dtype=torch.float64)
    k = torch.arange(nb, device=cuda)
    b = DeviceBatch(d, n, stride, f, x, o, k, k * n_out // nb)
    torch.cuda.synchronize()
    b.forward(tuning=tuning)
    torch.cuda.synchronize()
    return o


@pytest.mark.parametrize("d,n", SHAPES)
def test_bitwise_per_entry(cuda, d, n):
    # one entry; a few; more than one, two and four elements per thread hold in one wave
    wave = 152 * 1024 // n ** d
    for nb in sorted({1, 7, wave // 2 + 3, 2 * wave + 5, 5 * wave + 1}):
        got = _run(cuda, d, n, n + nb % 2, nb, nb)
        want = _run(cuda, d, n, n + nb % 2, nb, nb, tuning={"prefetch": 1})
        assert torch.equal(got, want), nb


@pytest.mark.parametrize("d,n,nb,fan", [(3, 4, 1001, 7), (2, 9, 803, 3), (3, 10, 333, 111), (11, 2, 40, 8)])
def test_runs(cuda, d, n, nb, fan):
    from kronmult_gb300 import DeviceBatch
    from kronmult_gb300 import workloads as W

    b = W.make_batch(d, n, n + 1, nb // fan, fan, seed=d * n, factor_scale=1.0 / n ** 0.5)
    db = DeviceBatch.from_host(b, device=cuda)
    db.forward(sync=True)
    assert O.rel_l2(db.outputs.cpu().numpy(), O.forward(b)) <= 8 * (d * n + fan) * 2.0 ** -53
