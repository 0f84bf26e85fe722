"""The FP32 register-block adjoint (n = 2..8): both gradients against the FP64 formulas.
The tolerance is the FP32 contract of the package (1e-5 relative L2); the sweeps' own
rounding is a few 1e-7."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-5

# one and several passes, a remainder axis, teams of 1 to 125 threads, entries sharing 8 warps
SHAPES = [(2, 2), (4, 2), (5, 2), (8, 2), (2, 3), (4, 3), (6, 3), (2, 4), (3, 4), (5, 4), (2, 5), (3, 5), (5, 5),
          (2, 6), (3, 6), (4, 6), (3, 7), (4, 7), (2, 8), (3, 8), (4, 8)]


def _batch(d, n, fan, seed, stride=None):
    from kronmult_gb300 import workloads as W

    return W.make_batch(d, n, stride or n + 1, len(fan), fan, seed=seed, shared_factors=True,
                        factor_scale=1.0 / n ** 0.5)


def _run(b, g, cuda, want_gin=True, want_gA=True):
    from kronmult_gb300 import DeviceBatch, adjoint

    db = DeviceBatch.from_host(b, device=cuda, dtype=torch.float32)
    gin = torch.full_like(db.inputs, 0.5) if want_gin else None  # accumulated into
    gfa = torch.zeros_like(db.factors) if want_gA else None
    adjoint(db, torch.from_numpy(g).to(cuda, torch.float32), gin, gfa)
    torch.cuda.synchronize()
    mats = None
    if want_gA:
        f = gfa.cpu().numpy()
        mats = np.stack([f[:, r + b.stride * np.arange(b.n)] for r in range(b.n)], axis=1)
        pad = np.ones(f.shape[1], dtype=bool)
        pad[(np.arange(b.n)[:, None] + b.stride * np.arange(b.n)).ravel()] = False
        assert not f[:, pad].any()  # the blocks' padding is left alone
    return gin.cpu().numpy() - 0.5 if want_gin else None, mats


def _check(b, cuda, seed, **want):
    g = np.random.Generator(np.random.PCG64(seed)).standard_normal((b.n_out, b.N))
    gin, gA = _run(b, g, cuda, **want)
    if gin is not None:
        assert O.rel_l2(gin, O.forward(O.transposed_batch(b, g))) <= TOL
    if gA is not None:
        assert O.rel_l2(gA.reshape(-1), np.asarray(O.grad_factors(b, g)).reshape(-1)) <= TOL


@pytest.mark.parametrize("d,n", SHAPES)
def test_shapes(cuda, d, n):
    """A few entries (one per team) and runs of 1..9 entries."""
    _check(_batch(d, n, [1, 3], 8000 + 10 * d + n), cuda, 1)
    _check(_batch(d, n, [2, 9, 1, 4, 7, 1, 5], 8100 + 10 * d + n), cuda, 2)


@pytest.mark.parametrize("d,n", [(2, 3), (3, 4), (3, 6), (4, 5)])
def test_many_entries_per_team(cuda, d, n):
    """More entries than one wave of teams: partials carried from entry to entry, runs that
    start and end inside a team's share."""
    rng = np.random.Generator(np.random.PCG64(3))
    count = {(2, 3): 9000, (3, 4): 5000, (3, 6): 2500, (4, 5): 1200}[(d, n)]
    _check(_batch(d, n, rng.integers(1, 20, size=count // 2), 8200 + 10 * d + n, stride=n), cuda, 4)


@pytest.mark.parametrize("want", [{"want_gA": False}, {"want_gin": False}])
@pytest.mark.parametrize("d,n", [(3, 5), (4, 4), (4, 6)])
def test_one_gradient(cuda, d, n, want):
    _check(_batch(d, n, [3, 8, 1, 6], 8300 + 10 * d + n), cuda, 5, **want)
