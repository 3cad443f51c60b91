"""The look-ahead schedule hands over to the sequential one when few rows are
left (LU_B200_LA_MIN): look-ahead to the end, a hand-over in the middle, at the
last panel, and none at all give the same factorisation."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n,b", [(701, 64), (1024, 128), (130, 64)])
def test_fp64_hand_over(cuda_dev, monkeypatch, n, b, graph):
    import charmlu_b200 as lu
    import scipy.linalg
    A0 = np.random.default_rng(n).uniform(-0.5, 0.5, (n, n))
    ref, piv = scipy.linalg.lu_factor(A0)
    for least in ("0", "1", str(n // 2), str(n)):
        monkeypatch.setenv("LU_B200_LA_MIN", least)
        buf = torch.zeros(n, n + (n & 1), dtype=torch.float64, device="cuda")
        A = buf[:, :n]
        A.copy_(torch.from_numpy(A0))
        s = lu.LUSolver(lu.LUConfig(n, b, lookahead=True, use_graph=graph))
        ipiv = s.factor(A)
        assert s.status() == 0
        assert ipiv.cpu().numpy().tolist() == piv.tolist()
        # two elimination orders: 1e-12 of the largest entry, as for the other parity tests of this size
        assert np.abs(A.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("prec", ["FP16X3", "FP16S"])
@pytest.mark.parametrize("n,b", [(1100, 128), (777, 64)])
def test_mixed_hand_over(cuda_dev, monkeypatch, n, b, prec):
    import charmlu_b200 as lu
    rng = np.random.default_rng(n)
    A0 = rng.uniform(-0.5, 0.5, (n, n)) + np.eye(n) * np.sqrt(n)  # well conditioned: any factors refine
    r = rng.uniform(-0.5, 0.5, n)
    ref = np.linalg.solve(A0, r)
    A = torch.zeros(n, n + (n & 1), dtype=torch.float64, device="cuda")[:, :n]
    A.copy_(torch.from_numpy(A0))
    for least in ("0", "1", str(n // 2), str(n)):
        monkeypatch.setenv("LU_B200_LA_MIN", least)
        s = lu.LUSolver(lu.LUConfig(n, b, precision=getattr(lu, "LU_PREC_" + prec), lookahead=True, use_graph=True,
                                    ir_target=1e-3))
        for _ in range(2):  # captured, then replayed
            x, info = s.refine_solve(A, torch.from_numpy(r).cuda())
            assert info["status"] == 0 and info["r_hpl"] < 1e-3
            # ||dx|| <= kappa n eps r_hpl (...) with kappa < 10 here
            assert np.abs(x.cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max()
