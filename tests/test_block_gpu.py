"""The FP32 register-block forward (n = 2..10): every output value is the k-ascending FMA
chain of the one-mode-per-step kernels, so with one entry per output the two agree bit for
bit; ragged runs of entries, odd strides, inputs off 16-byte boundaries and few or many
entries per team change only which FP32 sums are formed (FP32 outputs) or nothing (FP64
outputs, whose FP32 run sums are cut at fixed entries)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# a single pass, one pass and a remainder, two and three passes; teams of 1 to 343 threads
SHAPES = [(1, 2), (6, 2), (12, 2), (2, 3), (3, 3), (5, 3), (6, 3), (8, 3), (1, 4), (3, 4), (5, 4), (6, 4), (7, 4),
          (1, 5), (3, 5), (4, 5), (5, 5), (3, 6), (4, 6), (5, 6), (2, 7), (3, 7), (4, 7), (2, 8), (3, 8), (4, 8),
          (1, 9), (2, 9), (3, 9), (4, 9), (2, 10), (3, 10), (4, 10)]


def _batch(d, n, n_out, fan, stride, seed):
    from kronmult_gb300 import workloads as W

    return W.make_batch(d, n, stride, n_out, fan, seed=seed, factor_scale=1.0 / n ** 0.5)


def _run(b, cuda, out_dtype=torch.float32, tuning=None):
    from kronmult_gb300 import DeviceBatch

    db = DeviceBatch.from_host(b, device=cuda, dtype=torch.float32, out_dtype=out_dtype)
    db.forward(tuning=tuning)
    torch.cuda.synchronize()
    return db.outputs.cpu().numpy()


def _entries(d, n):
    return max(3, min(2600, 4_000_000 // n ** d))


@pytest.mark.parametrize("d,n", SHAPES)
def test_one_entry_per_output_bitwise(cuda, d, n):
    """Small and (where the shape has one) large batches against the forced
    one-mode-per-step kernel; n = 9, 10 have none and are held to FP32 rounding."""
    for count in (5, _entries(d, n)):
        b = _batch(d, n, count, 1, n + 1, seed=7000 + 100 * d + n)
        got = _run(b, cuda)
        if n <= 8 and n ** d <= 8192:
            assert np.array_equal(got, _run(b, cuda, tuning={"team_size": 256}))
        else:
            assert O.rel_l2(got, O.forward(b, dtype=np.float32)) <= 1e-6


@pytest.mark.parametrize("d,n", [(2, 3), (3, 4), (3, 5), (4, 5), (3, 6), (4, 7), (3, 8), (4, 8), (2, 9), (3, 10)])
def test_ragged_runs(cuda, d, n):
    """Runs of 1..19 entries per output, more entries than one wave of teams, into FP32 and
    FP64 outputs: the oracle's FP32 sweep up to the rounding of FP32 sums (a run of at most
    19 terms: 19 x 2^-24 = 1.2e-6 of their magnitudes)."""
    rng = np.random.Generator(np.random.PCG64(71))
    fan = rng.integers(1, 20, size=max(4, _entries(d, n) // 10))
    b = _batch(d, n, len(fan), fan, n, seed=7100 + 100 * d + n)
    want = O.forward(b, dtype=np.float32)
    for out_dtype in (torch.float32, torch.float64):
        for tuning in (None, {"entries_per_team": 5}, {"prefetch": 1}, {"ctas_per_sm": 1}):
            assert O.rel_l2(_run(b, cuda, out_dtype, tuning), want) <= 1.2e-6


@pytest.mark.parametrize("d,n", [(3, 4), (4, 5), (2, 6), (3, 6), (3, 8), (4, 10)])
def test_unaligned_inputs(cuda, d, n):
    """Inputs that start 4 bytes past a 16-byte boundary give the bits of aligned ones."""
    from kronmult_gb300 import DeviceBatch, _lib

    b = _batch(d, n, 40, 1, n + 2, seed=7200 + 100 * d + n)
    want = _run(b, cuda)
    db = DeviceBatch.from_host(b, device=cuda, dtype=torch.float32)
    pitch = b.N + (5 - b.N % 4)  # rows 1 float off a multiple of 4
    shifted = torch.zeros((b.nb, pitch), dtype=torch.float32, device=cuda)
    shifted[:, 1:b.N + 1] = db.inputs
    k = torch.arange(b.nb, device=cuda, dtype=torch.int64)
    in_ptrs = (shifted.data_ptr() + 4 + k * (pitch * 4)).contiguous()
    torch.cuda.synchronize()
    assert _lib.lib().kronmult_batched_f32(b.d, b.n, db.mat_ptrs.data_ptr(), b.stride, in_ptrs.data_ptr(),
                                           db.out_ptrs.data_ptr(), None, b.nb) == 0
    assert np.array_equal(db.outputs.cpu().numpy(), want)


@pytest.mark.parametrize("d,n,out_dtype", [(6, 4, torch.float32), (4, 8, torch.float32), (4, 8, torch.float64),
                                           (5, 3, torch.float64)])
def test_several_waves(cuda, d, n, out_dtype):
    """Large vectors in more than one wave of CTAs, ragged runs, a count that no share divides: the
    tolerance of test_ragged_runs."""
    from kronmult_gb300 import DeviceBatch
    from conftest import planned_kernel

    gen = torch.Generator(device=cuda)
    gen.manual_seed(31)
    N, nb = n ** d, {(6, 4): 19013, (4, 8): 36013, (5, 3): 95013}[d, n]
    fan = torch.randint(1, 20, (nb,), generator=gen, device=cuda)
    fan = fan[: int((fan.cumsum(0) < nb).sum()) + 1]
    fan[-1] -= int(fan.sum()) - nb
    outputs = fan.numel()
    index = torch.arange(outputs, device=cuda).repeat_interleave(fan)
    factors = (torch.rand((outputs * d, n * n), generator=gen, device=cuda) * 2 - 1) / n ** 0.5
    x = torch.randn((nb, N), generator=gen, device=cuda)
    assert "fwd_block_kernel" in planned_kernel(d, n, 1 if out_dtype == torch.float32 else 2, nb)
    db = DeviceBatch(d, n, n, factors, x, torch.zeros((outputs, N), dtype=out_dtype, device=cuda), index, index)
    db.forward()
    # an output's entries share their factors: K (x_1 + x_2 + ..), in 64 bits
    want = torch.zeros((outputs, N), dtype=torch.float64, device=cuda).index_add_(0, index, x.double())
    mats = factors.double().view(outputs, d, n, n).transpose(-1, -2)
    for i in range(d):
        want = torch.matmul(mats[:, i].unsqueeze(1), want.view(outputs, n ** i, n, -1)).reshape(outputs, N)
    assert float((db.outputs.double() - want).norm() / want.norm()) <= 1.2e-6
