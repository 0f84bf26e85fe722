"""FP64 deterministic groups, whose sums form in L2: bitwise the same on every run and for every
plan of one unit size, for runs that are whole segments, cross one unit edge or span many units,
native and emulated arithmetic; and the oracle's sums (d n additions per value, one per entry of
the output, each within 2^-53, with a factor 8 for the cancellation of random signs; emulated
arithmetic 1e-13)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arithmetic", ["native", "emulated"])
@pytest.mark.parametrize("d,n,n_out,fan,unit", [(2, 8, 300, 7, 0), (3, 3, 5, 401, 8), (4, 4, 2, 60, 1), (1, 5, 900, 1, 3),
                                                (3, 7, 40, 9, 64)])
def test_same_bits_on_every_run(cuda, d, n, n_out, fan, unit, arithmetic):
    from kronmult_gb300 import DeviceBatch
    from kronmult_gb300 import workloads as W
    from kronmult_gb300.grouped import GroupedPlan

    b = W.make_batch(d, n, n, n_out, fan, seed=d * n + fan, out_init="normal", factor_scale=1.0 / n ** 0.5)
    b.out_index[:] = b.out_index[np.random.Generator(np.random.PCG64(5)).permutation(b.nb)]
    first = None
    for _ in range(2):
        db = DeviceBatch.from_host(b, device=cuda)
        plan = GroupedPlan([db], mode="deterministic", arithmetic=arithmetic, tunings=[{"entries_per_team": unit}])
        for _ in range(10):
            db.outputs.copy_(torch.from_numpy(b.out_init))
            torch.cuda.synchronize()
            plan.run()
            torch.cuda.synchronize()
            got = db.outputs.cpu().numpy().copy()
            first = got if first is None else first
            assert np.array_equal(got, first)
        plan.close()
    tol = 8 * (d * n + fan) * 2.0 ** -53 if arithmetic == "native" else 1e-13
    assert O.rel_l2(first, O.forward(b)) <= tol


@pytest.mark.parametrize("d,n,nb,fan", [(1, 2, 3001, 5), (2, 3, 4000, 1), (6, 2, 2500, 300), (3, 5, 1203, 17), (7, 2, 900, 4),
                                        (2, 10, 777, 9), (3, 6, 30001, 11), (3, 9, 31000, 13), (3, 5, 300001, 23)])
def test_short_vector_units(cuda, d, n, nb, fan):
    """Units of one step and of several (the last three), threads owning a position over all
    entries (n^d >= 128) or over one run: the same bits on every run, and the sum of the
    per-entry results to rounding (one addition per entry, each within 2^-53, factor 8)."""
    from kronmult_gb300 import DeviceBatch
    from kronmult_gb300.grouped import GroupedPlan

    g = torch.Generator(device=cuda).manual_seed(nb)
    N, n_out = n ** d, (nb + fan - 1) // fan
    f = (torch.rand((nb * d, n * n), generator=g, device=cuda, dtype=torch.float64) * 2 - 1) / n ** 0.5
    x = torch.randn((nb, N), generator=g, device=cuda, dtype=torch.float64)
    k = torch.arange(nb, device=cuda)
    out = (k // fan)[torch.randperm(nb, generator=g, device=cuda)]
    one = torch.zeros((nb, N), device=cuda, dtype=torch.float64)
    b1 = DeviceBatch(d, n, n, f, x, one, k, k)
    o = torch.empty((n_out, N), device=cuda, dtype=torch.float64)
    b = DeviceBatch(d, n, n, f, x, o, k, out)
    torch.cuda.synchronize()
    b1.forward()
    want = torch.zeros((n_out, N), device=cuda, dtype=torch.float64).index_add_(0, out, one)
    plan, first = GroupedPlan([b], mode="deterministic"), None
    for _ in range(4):
        o.zero_()
        torch.cuda.synchronize()
        plan.run()
        torch.cuda.synchronize()
        first = o.clone() if first is None else first
        assert torch.equal(o, first)
    plan.close()
    err = ((first - want).norm() / want.norm()).item()
    assert err <= 8 * fan * 2.0 ** -53, err
