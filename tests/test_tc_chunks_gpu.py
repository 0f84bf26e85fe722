"""Tensor-core forward over more chunks than CTAs: every entry's result and every run sum is
the one of a small batch holding the same entries (chunks of 8 start at the same entries), bit
for bit, for bulk copies and for inputs off 16-byte boundaries."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("fan", [1, 5])
@pytest.mark.parametrize("compute", [1, 2, 3])
@pytest.mark.parametrize("d,nb", [(1, 20555), (2, 20555), (3, 20555), (4, 7965)])
def test_tail_of_a_large_batch(cuda, d, nb, compute, fan, off):
    from kronmult_gb300 import DeviceBatch, forward_f32_f64out

    N = 8 ** d
    g = torch.Generator(device=cuda).manual_seed(d * 10 + fan)
    x = torch.randn((nb, N), generator=g, device=cuda)
    f = torch.randn((nb * d, 64), generator=g, device=cuda) / 8
    # more chunks than fit at once (16 CTAs per SM for d < 4, 8 for d = 4), the last one ragged
    k = torch.arange(nb, device=cuda)
    buf = torch.zeros(nb * N + off, device=cuda)
    buf[off:] = x.reshape(-1)

    def outputs(first, stream_in):
        sel = slice(first, nb)
        n_out = (nb - first + fan - 1) // fan
        o = torch.zeros((n_out, N), device=cuda, dtype=torch.float64)
        b = DeviceBatch(d, 8, 8, f, x[sel].contiguous(), o, k[sel].contiguous(), (k[sel] - first) // fan)
        if stream_in:
            b.in_ptrs = (buf.data_ptr() + 4 * (off + N * k[sel])).contiguous()
        forward_f32_f64out(b, compute=compute)
        torch.cuda.synchronize()
        return o

    first = nb // 40 * 40 - 40  # a multiple of the chunk length and of the fan-in
    big, small = outputs(0, True), outputs(first, False)
    assert torch.equal(big[first // fan:], small)
    assert torch.isfinite(big).all()
