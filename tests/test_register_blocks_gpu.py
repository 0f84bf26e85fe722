"""The FP32 register blocks at batch sizes that they serve: the same bits as the one-mode-per-step
kernels, infinities, NaN and subnormals included, and kernels that allocate tensor memory on two
streams at once."""
import pytest
import torch

from conftest import planned_kernel

pytestmark = pytest.mark.gpu
F32, F32_F64OUT = 1, 2
# (d, n): entries from which FP32 outputs are the register blocks', beyond any band of batch sizes
ENTRIES = {(1, 2): 400003, (2, 2): 120007, (6, 2): 26003, (12, 2): 20003, (2, 3): 20011, (3, 3): 20011, (5, 3): 3001,
           (8, 3): 301, (1, 4): 120011, (3, 4): 5003, (4, 4): 5003, (5, 4): 3001, (6, 4): 9203, (7, 4): 301,
           (1, 5): 200003, (3, 5): 25013, (4, 5): 5003, (3, 6): 9001, (4, 6): 2003, (2, 7): 50021, (3, 7): 4507,
           (4, 7): 1201, (2, 8): 9001, (3, 8): 5003, (4, 8): 5003}


def _batch(cuda, d, n, nb, out_dtype, spoil=None):
    from kronmult_gb300 import DeviceBatch

    gen = torch.Generator(device=cuda)
    gen.manual_seed(100 * d + n)
    f = (torch.rand((nb * d, (n + 1) * n), generator=gen, device=cuda) * 2 - 1) / n ** 0.5
    x = torch.randn((nb, n ** d), generator=gen, device=cuda)
    if spoil is not None:
        spoil(x)
    k = torch.arange(nb, device=cuda)
    return DeviceBatch(d, n, n + 1, f, x, torch.zeros((nb, n ** d), dtype=out_dtype, device=cuda), k, k)


def _same(a, b):
    return torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(0.0), b.nan_to_num(0.0))


def _both(b, dtype, tuning={"team_size": 256}):
    assert "fwd_block_kernel" in planned_kernel(b.d, b.n, dtype, b.nb)
    assert "fwd_block_kernel" not in planned_kernel(b.d, b.n, dtype, b.nb, tuning)
    b.forward()
    got = b.outputs.clone()
    b.outputs.zero_()
    b.forward(tuning=tuning)
    torch.cuda.synchronize()
    return got, b.outputs


@pytest.mark.parametrize("d,n", sorted(ENTRIES))
def test_one_entry_per_output_bitwise(cuda, d, n):
    got, want = _both(_batch(cuda, d, n, ENTRIES[d, n], torch.float32), F32)
    assert torch.equal(got, want)


def _specials(x):
    """Rows of one infinity, one NaN, the largest and subnormal values; others as they were."""
    x[1::7, 0] = float("inf")
    x[2::7, -1] = float("nan")
    x[3::7] = torch.finfo(torch.float32).max
    x[4::7] *= 1e-42
    x[5::7] = torch.finfo(torch.float32).min


@pytest.mark.parametrize("out_dtype,dtype", [(torch.float32, F32), (torch.float64, F32_F64OUT)])
@pytest.mark.parametrize("d,n,nb", [(4, 4, 5003), (4, 5, 5003), (3, 6, 26003), (3, 8, 19001), (4, 8, 9601)])
def test_specials(cuda, d, n, nb, out_dtype, dtype):
    b = _batch(cuda, d, n, nb, out_dtype, _specials)
    got, want = _both(b, dtype)
    assert _same(got, want)
    assert torch.isfinite(got[0::7]).all() and not torch.isfinite(got[1::7]).all()
    if out_dtype == torch.float64:  # (single-precision additions in memory flush subnormals to zero)
        assert 0 < float(got[4::7].abs().max()) < 1e-37


def test_specials_stay_with_their_factor_set(cuda):
    """FP32 adjoint: an entry with a NaN spoils the gradients of its own set alone."""
    from kronmult_gb300 import DeviceBatch, adjoint

    for d, n in ((2, 3), (3, 6), (4, 8)):
        gen = torch.Generator(device=cuda)
        gen.manual_seed(d)
        sets, fan, N = 300, 5, n ** d
        f = (torch.rand((sets * d, n * n), generator=gen, device=cuda) * 2 - 1) / n ** 0.5
        x = torch.randn((sets * fan, N), generator=gen, device=cuda)
        g = torch.randn((sets, N), generator=gen, device=cuda)
        index = torch.arange(sets, device=cuda).repeat_interleave(fan)
        grads = []
        for spoiled in (False, True):
            if spoiled:
                x[7 * fan + 2, 1] = float("nan")
                x[100 * fan, 0] = float("inf")
            b = DeviceBatch(d, n, n, f, x, torch.zeros((sets, N), device=cuda), index, index)
            gf = torch.zeros_like(f)
            adjoint(b, g, None, gf)
            torch.cuda.synchronize()
            grads.append(gf.view(sets, -1))
        bad = torch.zeros(sets, dtype=torch.bool, device=cuda)
        bad[7] = bad[100] = True
        assert not torch.isfinite(grads[1][7]).any() or not torch.isfinite(grads[1][7]).all()
        assert not torch.isfinite(grads[1][100]).all()
        clean, want = grads[1][~bad], grads[0][~bad]
        assert torch.isfinite(clean).all()
        # the order of additions in memory differs from run to run: single-precision rounding
        assert float((clean - want).norm() / want.norm()) <= 1e-6


def test_two_streams(cuda):
    """Tensor-core, register-block and adjoint kernels, all of which allocate tensor memory, side by
    side: with one entry per output the results are the bits of runs one after another."""
    from kronmult_gb300 import adjoint, forward_f32_f64out

    tc = _batch(cuda, 4, 8, 6007, torch.float64)
    blk = _batch(cuda, 4, 5, 20011, torch.float32)
    wide = _batch(cuda, 6, 4, 6007, torch.float32)
    gout = torch.randn_like(blk.outputs)
    gin, gfa = torch.zeros_like(blk.inputs), torch.zeros_like(blk.factors)

    def clear():
        for t in (tc.outputs, blk.outputs, wide.outputs, gin, gfa):
            t.zero_()
        torch.cuda.synchronize()

    def results():
        torch.cuda.synchronize()
        return [t.clone() for t in (tc.outputs, blk.outputs, wide.outputs, gin, gfa)]

    clear()
    forward_f32_f64out(tc, compute=1)
    blk.forward()
    wide.forward()
    adjoint(blk, gout, gin, gfa)
    want = results()
    streams = [torch.cuda.Stream() for _ in range(3)]
    for _ in range(5):
        clear()
        forward_f32_f64out(tc, compute=1, stream=streams[0])
        blk.forward(stream=streams[1])
        wide.forward(stream=streams[2])
        adjoint(blk, gout, gin, gfa, stream=streams[0])
        for a, b in zip(results(), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("d,nb", [(3, 9001), (4, 12007)])
def test_pairs_bitwise(cuda, d, nb):
    """n = 4 in a band of batch sizes that the register blocks leave to the bi-fibre kernel."""
    b = _batch(cuda, d, 4, nb, torch.float32)
    assert "fwd_pair_kernel" in planned_kernel(d, 4, F32, nb)
    b.forward()
    got = b.outputs.clone()
    b.outputs.zero_()
    b.forward(tuning={"team_size": 256})
    torch.cuda.synchronize()
    assert torch.equal(got, b.outputs)
