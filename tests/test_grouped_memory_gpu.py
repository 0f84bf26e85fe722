"""Device memory of deterministic plans: sorted pointer tables, and partial sums of at most 96 MB
that the groups share."""
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_partial_sums_are_shared_and_bounded(cuda):
    from kronmult_gb300 import DeviceBatch
    from kronmult_gb300.grouped import GroupedPlan

    d, n, nb = 3, 10, 19000
    N = n ** d
    gen = torch.Generator(device=cuda)
    gen.manual_seed(5)
    factors = torch.rand((7 * d, n * n), generator=gen, device=cuda, dtype=torch.float64) - 0.5
    x = torch.randn((nb, N), generator=gen, device=cuda, dtype=torch.float64)
    sets = torch.arange(nb, device=cuda) % 7
    index = torch.arange(nb, device=cuda) // 3  # runs of 3, which units cut
    groups = [DeviceBatch(d, n, n, factors, x, torch.zeros(((nb + 2) // 3, N), dtype=torch.float64, device=cuda), sets,
                          index) for _ in range(3)]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    plan = GroupedPlan(groups, mode="deterministic")
    used = free - torch.cuda.mem_get_info()[0]
    tables = 3 * (2 * 32768 * 8 + nb * (d + 2) * 8)
    assert used <= (96 << 20) + tables + (16 << 20)  # the driver's granularity, streams and events
    plan.run()
    torch.cuda.synchronize()
    mats = factors.view(7, d, n, n).transpose(-1, -2)[sets]
    y = x
    for i in range(d):
        y = torch.matmul(mats[:, i].unsqueeze(1), y.view(nb, n ** i, n, -1)).reshape(nb, N)
    want = torch.zeros_like(groups[0].outputs).index_add_(0, index, y)
    for b in groups:
        assert O.rel_l2(b.outputs.cpu().numpy(), want.cpu().numpy()) <= 1e-13
        assert torch.equal(b.outputs, groups[0].outputs)
