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
