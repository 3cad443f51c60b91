"""Order of the substitution pipelines' progress counter: it advances one block at
a time, whatever block is done first, and names no block whose rows are not there."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tickets", [1, 2, 3, 16])
def test_counter_advances_in_block_order(cuda_dev, tickets):
    from charmlu_b200 import _lib
    scratch = torch.zeros(32, dtype=torch.int32, device="cuda")
    out = np.full(4, -1, dtype=np.int32)
    rc = _lib.load().lub_test_publish_progress(tickets, ctypes.c_void_p(scratch.data_ptr()),
                                               ctypes.c_void_p(out.ctypes.data),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    assert out.tolist() == [tickets, 0, 0, 0]


@pytest.mark.parametrize("nrhs", [1, 7, 16])
def test_repeated_solves_give_the_same_bits(cuda_dev, nrhs):
    """Many blocks, so that most rows are read by way of the counter; every sum
    has one order, so a row read too early shows in the bits."""
    import charmlu_b200 as lu
    n = 6016
    A = lu.generate_uniform(n, n, seed=5)
    A.diagonal().add_(float(n) ** 0.5)
    B = lu.generate_uniform(n, nrhs, seed=6)
    s = lu.LUSolver(lu.LUConfig(n, 128))
    F = A.clone()
    piv = s.factor(F)
    assert s.status() == 0
    for trans in (False, True):
        first = None
        for _ in range(15):
            X = B.clone()
            s.solve(F, piv, X, trans=trans)
            assert s.status() == 0
            if first is None:
                first = X
            assert torch.equal(X, first)
        # backward stable: residual within n roundings of the terms' size
        R = (A.T if trans else A) @ first - B
        scale = A.abs().sum(1).max() * first.abs().max() + B.abs().max()
        assert R.abs().max() < 16 * n * 2.0 ** -52 * scale
    s.close()


@pytest.mark.parametrize("upper", [0, 1])
def test_substitutions_of_changing_size_share_one_ring(cuda_dev, upper):
    """Orders of 1 to 6 blocks in turn through one handle: the ring of packets
    starts cleared as far as a call reads it, whatever the call before left."""
    from charmlu_b200.blocks import CudaBlocks
    bl = CudaBlocks(384, 64)
    gen = torch.Generator(device="cuda").manual_seed(upper)
    for it in range(4):
        for w in [384, 64, 320, 65, 256, 128, 257, 129, 1, 192, 384, 193, 2]:
            T = torch.zeros(w, w + (w & 1), dtype=torch.float64, device="cuda")[:, :w]
            T.copy_((torch.rand(w, w, dtype=torch.float64, device="cuda", generator=gen) - 0.5) * 0.1)
            T.diagonal().fill_(1.0)
            x = torch.rand(w, dtype=torch.float64, device="cuda", generator=gen)
            ref = torch.linalg.solve_triangular(T, x.view(-1, 1), upper=bool(upper), unitriangular=not upper).view(-1)
            bl.trsv_block(T, upper, x)
            # |T| <= 1 off a unit diagonal of small rows: both are within w roundings of the size
            assert (x - ref).abs().max() <= 1e-12 * ref.abs().max(), (it, w)
    bl.close()
