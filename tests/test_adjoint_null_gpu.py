"""Null entries in the table of factor-gradient pointers: those factors get no gradient, the
others and the input gradients are what they are without null entries."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float64, 1e-13)])
@pytest.mark.parametrize("d,n", [(2, 3), (3, 4), (3, 6), (4, 6), (4, 8)])
def test_null_factor_gradients(cuda, d, n, dtype, tol):
    from kronmult_gb300 import DeviceBatch, _lib, workloads as W

    fan = [3, 1, 9, 4, 2, 6, 1]
    b = W.make_batch(d, n, n, len(fan), fan, seed=9100 + 10 * d + n, shared_factors=True, factor_scale=1.0 / n ** 0.5)
    g = np.random.Generator(np.random.PCG64(9)).standard_normal((b.n_out, b.N))
    db = DeviceBatch.from_host(b, device=cuda, dtype=dtype)
    gout = torch.from_numpy(g).to(cuda, dtype)
    gin, gfa = torch.zeros_like(db.inputs), torch.zeros_like(db.factors)
    es = gout.element_size()
    gout_ptrs = gout.data_ptr() + db.out_index * (b.N * es)
    gin_ptrs = gin.data_ptr() + torch.arange(b.nb, device=cuda) * (b.N * es)
    row = db.fac_index[:, None] * d + torch.arange(d, device=cuda)[None, :]
    wanted = (row % 3 != 1) & (db.fac_index[:, None] != 2)  # some factors of a set, all of another
    gmat_ptrs = torch.where(wanted, gfa.data_ptr() + row * (gfa.shape[1] * es), 0).reshape(-1).contiguous()
    name = "kronmult_batched_adjoint_f32_async" if dtype == torch.float32 else "kronmult_batched_adjoint_f64_async"
    torch.cuda.synchronize()
    assert getattr(_lib.lib(), name)(d, n, db.mat_ptrs.data_ptr(), b.stride, db.in_ptrs.data_ptr(),
                                     gout_ptrs.data_ptr(), gin_ptrs.data_ptr(), gmat_ptrs.data_ptr(), b.stride, b.nb,
                                     None, None) == 0
    torch.cuda.synchronize()
    f = gfa.cpu().numpy()
    got = np.stack([f[:, r + b.stride * np.arange(n)] for r in range(n)], axis=1)
    want = np.asarray(O.grad_factors(b, g)).reshape(got.shape).copy()
    rows = np.arange(len(fan) * d)
    want[(rows % 3 == 1) | (rows // d == 2)] = 0.0
    assert O.rel_l2(got.reshape(-1), want.reshape(-1)) <= tol
    assert not got[(rows % 3 == 1) | (rows // d == 2)].any()
    assert O.rel_l2(gin.cpu().numpy(), O.forward(O.transposed_batch(b, g))) <= tol
