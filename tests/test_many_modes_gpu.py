"""Vectors of 17 and more modes: n = 1 and n = 2, FP64, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(17, 1), (27, 1), (17, 2), (18, 2)])
def test_forward(cuda, d, n):
    from kronmult_gb300 import DeviceBatch, workloads as W

    b = W.make_batch(d, n, n + 1, 2, 3, seed=9000 + d, factor_scale=1.0 / n ** 0.5)
    db = DeviceBatch.from_host(b, device=cuda, with_workspace=True)
    db.forward()
    torch.cuda.synchronize()
    assert O.rel_l2(db.outputs.cpu().numpy(), O.forward(b)) <= 1e-13


@pytest.mark.parametrize("d,n", [(17, 2), (23, 2), (17, 3)])
def test_adjoint_not_supported(cuda, d, n):
    """Vectors beyond shared memory have no adjoint: refused before any access."""
    from kronmult_gb300 import _lib

    p = torch.zeros(64, dtype=torch.int64, device=cuda).data_ptr()
    status = _lib.lib().kronmult_batched_adjoint_f64_async(d, n, p, n, p, p, p, p, n, 1, None, None)
    assert "not supported" in _lib.error_string(status)
