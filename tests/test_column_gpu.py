"""FP32 vectors beyond shared memory through the two register-block passes, every n at its
smallest and largest d, partial pass-2 tiles (C = n^d1 not a multiple of 32), runs of entries
that end inside a warp's share, workspaces and inputs off 16-byte boundaries.  Tolerance: the
d n additions of a value's chain and the fan additions into the output, each within 2^-24."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [(14, 2), (18, 2), (9, 3), (11, 3), (8, 4), (9, 4), (6, 5), (7, 5), (6, 6), (7, 6), (6, 7), (5, 8), (6, 8)]


def _check(cuda, b, out_dtype, off=0):
    from kronmult_gb300 import DeviceBatch

    db = DeviceBatch.from_host(b, device=cuda, dtype=torch.float32, out_dtype=out_dtype, with_workspace=True)
    moved = []  # the same vectors, off floats into larger buffers
    if off:
        N = b.n ** b.d
        for src, table in ((db.inputs, "in_ptrs"), (db.workspace, "ws_ptrs")):
            buf = torch.empty(b.nb * N + off, device=cuda, dtype=torch.float32)
            buf[off:] = src.reshape(-1)
            moved.append(buf)
            k = torch.arange(b.nb, device=cuda, dtype=torch.int64)
            setattr(db, table, (buf.data_ptr() + 4 * (off + k * N)).contiguous())
    x0 = [m.clone() for m in moved[:1]] or [db.inputs.clone()]
    db.forward(sync=True)
    fan = b.nb // b.out_init.shape[0]
    assert O.rel_l2(db.outputs.double().cpu().numpy(), O.forward(b)) <= (b.d * b.n + fan) * 2.0 ** -24
    assert torch.equal((moved or [db.inputs])[0], x0[0])


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("d,n", SHAPES)
def test_shapes(cuda, d, n, out_dtype):
    from kronmult_gb300 import workloads as W

    b = W.make_batch(d, n, n + 1, 2, 3, seed=40 * d + n, factor_scale=1.0 / n ** 0.5)
    _check(cuda, b, out_dtype, off=1 if n % 2 else 0)


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("d,n,n_out,fan,off", [(5, 8, 3, 67, 0), (5, 8, 201, 1, 2), (6, 6, 1, 90, 1), (9, 3, 5, 31, 3)])
def test_runs(cuda, d, n, n_out, fan, off, out_dtype):
    """Many entries per output, one per output, and every copy off its 16 bytes."""
    from kronmult_gb300 import workloads as W

    b = W.make_batch(d, n, n, n_out, fan, seed=d + n + fan, factor_scale=1.0 / n ** 0.5)
    _check(cuda, b, out_dtype, off)
