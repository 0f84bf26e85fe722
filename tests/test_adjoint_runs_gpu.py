"""FP32 factor gradients summed over many entries: in parts of at most 32 entries per team, and
over the teams of a warp before they go to memory.

Tolerance: one rounding has a root-mean-square error of at most 2^-24 / sqrt(3) of the value, and
the partial values of a sum of m like terms have mean squares m / 2 of the whole's.  A
gradient element is 3 d - 1 mode products of n additions and a contraction over n^(d-1) (in parts),
then sums over chains of at most 32 entries, teams (a tree) and parts in memory of at least 8
entries."""
import math

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _batch(d, n, fan, seed):
    from kronmult_gb300 import workloads as W

    return W.make_batch(d, n, n, len(fan), fan, seed=seed, shared_factors=True, factor_scale=1.0 / n ** 0.5)


def _factor_gradients(cuda, b, g):
    from kronmult_gb300 import DeviceBatch, adjoint

    db = DeviceBatch.from_host(b, device=cuda, dtype=torch.float32)
    gfa = torch.zeros_like(db.factors)
    adjoint(db, torch.from_numpy(g).to(cuda, torch.float32), None, gfa)
    f = gfa.cpu().numpy()
    return np.stack([f[:, r + b.stride * np.arange(b.n)] for r in range(b.n)], axis=1)


@pytest.mark.parametrize("d,n,sets", [(2, 2, 30), (2, 3, 30), (3, 4, 15)])
def test_long_runs(cuda, d, n, sets):
    """2000 entries per factor set, a set per several warps of teams."""
    b = _batch(d, n, [2000] * sets, 8400 + 10 * d + n)
    g = np.random.Generator(np.random.PCG64(3)).standard_normal((b.n_out, b.N))
    want = np.asarray(O.grad_factors(b, g)).reshape(-1)
    tol = 2.0 ** -24 / math.sqrt(3) * math.sqrt((3 * d - 1) * n + n ** (d - 1) / 2 + 32 / 2 + 2000 / 8 / 2)
    assert O.rel_l2(_factor_gradients(cuda, b, g).reshape(-1), want) <= tol


@pytest.mark.parametrize("d,n", [(2, 2), (3, 2), (2, 3), (3, 3), (2, 4), (3, 4)])
def test_ragged_runs_over_teams(cuda, d, n):
    """Runs of 1 to 40 entries that begin and end inside a warp's teams, one entry per team and more."""
    rng = np.random.Generator(np.random.PCG64(5))
    for count in (40, 900, 6000):
        b = _batch(d, n, rng.integers(1, 41, size=count), 8500 + 10 * d + n)
        g = rng.standard_normal((b.n_out, b.N))
        want = np.asarray(O.grad_factors(b, g)).reshape(-1)
        tol = 2.0 ** -24 / math.sqrt(3) * math.sqrt((3 * d - 1) * n + n ** (d - 1) / 2 + 32 / 2 + 40 / 2)
        assert O.rel_l2(_factor_gradients(cuda, b, g).reshape(-1), want) <= tol


@pytest.mark.parametrize("d,n,count", [(4, 6, 2411), (4, 7, 1613)])
def test_entries_sharing_eight_warps(cuda, d, n, count):
    """7 and 5 entries per CTA of 8 warps, several per team, runs that end at different entries."""
    rng = np.random.Generator(np.random.PCG64(6))
    fan = rng.integers(1, 20, size=count)
    fan = fan[: int((np.cumsum(fan) < count).sum()) + 1]
    fan[-1] -= fan.sum() - count
    b = _batch(d, n, fan, 8600 + 10 * d + n)
    g = rng.standard_normal((b.n_out, b.N))
    want = np.asarray(O.grad_factors(b, g)).reshape(-1)
    assert O.rel_l2(_factor_gradients(cuda, b, g).reshape(-1), want) <= 1e-5
