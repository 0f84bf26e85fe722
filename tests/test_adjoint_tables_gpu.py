"""The adjoint's pointer tables: made anew when what they point to changes, on the stream that
reads them, and left alone by captured graphs."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu
D, N = 2, 3


def _setup(cuda, seed=1):
    from kronmult_gb300 import DeviceBatch, workloads as W

    b = W.make_batch(D, N, N, 6, [3, 1, 4, 2, 5, 1], seed=seed, shared_factors=True)
    g = np.random.Generator(np.random.PCG64(seed)).standard_normal((b.n_out, b.N))
    db = DeviceBatch.from_host(b, device=cuda)
    gout = torch.from_numpy(g).to(cuda)
    return b, g, db, gout, torch.zeros_like(db.inputs), torch.zeros_like(db.factors)


def _check(b, g, gin, gfa):
    f = gfa.cpu().numpy()
    mats = np.stack([f[:, r + b.stride * np.arange(b.n)] for r in range(b.n)], axis=1)
    assert O.rel_l2(gin.cpu().numpy(), O.forward(O.transposed_batch(b, g))) <= 1e-13
    assert O.rel_l2(mats.reshape(-1), np.asarray(O.grad_factors(b, g)).reshape(-1)) <= 1e-13


@pytest.mark.parametrize("in_place", [False, True])
def test_changed_indices(cuda, in_place):
    """Another order of the entries between two calls with the same gradient tensors."""
    from kronmult_gb300 import adjoint

    b, g, db, gout, gin, gfa = _setup(cuda)
    adjoint(db, gout, gin, gfa)
    _check(b, g, gin, gfa)
    perm = np.random.Generator(np.random.PCG64(3)).permutation(b.nb)
    b.out_index, b.fac_index = b.out_index[perm].copy(), b.fac_index[perm].copy()
    if in_place:
        db.out_index.copy_(torch.from_numpy(b.out_index))
        db.fac_index.copy_(torch.from_numpy(b.fac_index))
    else:
        db.out_index, db.fac_index = torch.from_numpy(b.out_index).to(cuda), torch.from_numpy(b.fac_index).to(cuda)
    db.build_pointers()
    gin.zero_()
    gfa.zero_()
    adjoint(db, gout, gin, gfa)
    _check(b, g, gin, gfa)


def test_arguments_checked_on_every_call(cuda):
    """Tensors of another shape or type at the address of earlier ones are refused."""
    from kronmult_gb300 import adjoint

    b, g, db, gout, gin, gfa = _setup(cuda)
    adjoint(db, gout, gin, gfa)
    with pytest.raises(ValueError):
        adjoint(db, gout, gin[:-1], gfa)
    with pytest.raises(ValueError):
        adjoint(db, gout, gin, gfa[:-1])
    with pytest.raises(ValueError):
        adjoint(db, gout, gin.view(torch.int64), gfa)
    with pytest.raises(ValueError):
        adjoint(db, gout.view(torch.int64), gin, gfa)


@pytest.mark.parametrize("as_int", [False, True])
def test_other_stream_does_not_wait_for_the_current_one(cuda, as_int):
    """The tables of a call on another stream are ready there whatever the current stream does;
    a gradient that has to be copied first is copied there too."""
    from kronmult_gb300 import adjoint

    b, g, db, gout, gin, gfa = _setup(cuda)
    wide = torch.zeros((gout.shape[0], gout.shape[1] + 1), dtype=gout.dtype, device=cuda)
    wide[:, 1:] = gout
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    for grad in (gout, wide[:, 1:]):
        torch.cuda._sleep(100_000_000)  # the current stream is busy
        adjoint(db, grad, gin, gfa, stream=s.cuda_stream if as_int else s)
        s.synchronize()
        _check(b, g, gin, gfa)
        torch.cuda.synchronize()
        gin.zero_()
        gfa.zero_()
        torch.cuda.synchronize()


def test_captured_calls(cuda):
    """A graph captured with warm tables survives calls with other gradients; one captured without
    leaves no tables behind that only its replay fills."""
    from kronmult_gb300 import adjoint

    b, g, db, gout, gin, gfa = _setup(cuda)
    gin2, gfa2 = torch.zeros_like(gin), torch.zeros_like(gfa)
    adjoint(db, gout, gin, gfa)
    torch.cuda.synchronize()
    warm, cold = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(warm):
        adjoint(db, gout, gin, gfa)
    with torch.cuda.graph(cold):
        adjoint(db, gout, gin2, gfa2)
    adjoint(db, gout, gin2, gfa2)  # before the graph has run
    _check(b, g, gin2, gfa2)
    junk = [torch.full((64,), 7, dtype=torch.int64, device=cuda) for _ in range(64)]
    for graph, a, f in ((warm, gin, gfa), (cold, gin2, gfa2), (warm, gin, gfa)):
        a.zero_()
        f.zero_()
        graph.replay()
        _check(b, g, a, f)
    assert len(junk) == 64
