"""The FP64 adjoint with n and d at compile time against the element kernels (forced by a tuning
field): input gradients bit for bit, factor gradients to the rounding of their sums (n^(d-1)
products and the entries of a factor, each within 2^-53, with a factor 8 for the cancellation of
random signs); one, two and four elements per thread, a last CTA that is not full, either
gradient alone, odd strides and factor sets shared by entries."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2), (5, 2), (8, 2), (2, 3), (6, 3), (7, 3), (3, 4), (6, 4), (2, 5), (5, 5), (3, 6), (2, 7), (4, 7), (3, 8), (4, 8),
          (2, 9), (3, 10)]


def _run(cuda, d, n, nb, share, want, tuning=None):
    from kronmult_gb300 import DeviceBatch, adjoint

    g = torch.Generator(device=cuda).manual_seed(n * 100 + d)
    sets, st = (nb + share - 1) // share, n + nb % 2
    f = (torch.rand((sets * d, st * n), generator=g, device=cuda, dtype=torch.float64) * 2 - 1) / n ** 0.5
    x = torch.randn((nb, n ** d), generator=g, device=cuda, dtype=torch.float64)
    o = torch.zeros((nb, n ** d), device=cuda, dtype=torch.float64)
    go = torch.randn((nb, n ** d), generator=g, device=cuda, dtype=torch.float64)
    k = torch.arange(nb, device=cuda)
    b = DeviceBatch(d, n, st, f, x, o, k // share, k)
    gi = torch.zeros_like(x) if "i" in want else None
    gf = torch.zeros_like(f) if "f" in want else None
    torch.cuda.synchronize()
    adjoint(b, go, gi, gf, tuning=tuning)
    torch.cuda.synchronize()
    return gi, gf


@pytest.mark.parametrize("d,n", SHAPES)
def test_against_element_kernels(cuda, d, n):
    wave = 152 * 1024 // n ** d
    for nb in sorted({1, 7, wave // 2 + 3, 2 * wave + 5, 5 * wave + 1}):
        for want in ("if", "i", "f") if nb == 7 else ("if",):
            gi, gf = _run(cuda, d, n, nb, 3, want)
            wi, wf = _run(cuda, d, n, nb, 3, want, tuning={"ctas_per_sm": 1})
            if "i" in want:
                assert torch.equal(gi, wi), (nb, want)
            if "f" in want:
                err = ((gf - wf).norm() / wf.norm()).item()
                assert err <= 8 * (n ** (d - 1) + 3) ** 0.5 * 2.0 ** -53, (nb, want, err)
