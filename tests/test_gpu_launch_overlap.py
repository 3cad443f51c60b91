"""Kernels whose launch overlaps the end of the one ahead: factorisations issued
back to back, each on freshly copied data, must equal the same factorisation
replayed from a captured graph, whose kernels keep full dependencies, in every
bit (the arithmetic is the same, so the tolerance is zero)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _padded(n):
    return torch.zeros(n, n + (n & 1), dtype=torch.float64, device="cuda")[:, :n]


@pytest.mark.parametrize("n,b,lookahead", [(33, 32, False), (256, 64, False), (701, 64, True), (1500, 192, False),
                                           (2048, 128, True), (7000, 192, True)])
def test_fp64_back_to_back(cuda_dev, n, b, lookahead):
    import charmlu_b200 as lu
    g = torch.Generator(device="cuda").manual_seed(n)
    src = [torch.rand(n, n, dtype=torch.float64, device="cuda", generator=g) - 0.5 for _ in range(2)]
    want = []
    s = lu.LUSolver(lu.LUConfig(n, b, lookahead=lookahead, use_graph=True))
    for A0 in src:
        A = _padded(n)
        A.copy_(A0)
        ipiv = s.factor(A)
        want.append((A.clone(), ipiv.clone()))
    s.close()
    s = lu.LUSolver(lu.LUConfig(n, b, lookahead=lookahead, use_graph=False))
    A = _padded(n)
    got = []
    for i in range(6):
        A.copy_(src[i % 2])
        ipiv = s.factor(A)
        got.append((A.clone(), ipiv.clone()))
    s.check("factor")
    s.close()
    for i, (A, ipiv) in enumerate(got):
        assert torch.equal(ipiv, want[i % 2][1])
        assert torch.equal(A, want[i % 2][0])


@pytest.mark.parametrize("n,lookahead", [(128, False), (1000, False), (3000, True)])
def test_mixed_back_to_back(cuda_dev, n, lookahead):
    import charmlu_b200 as lu
    g = torch.Generator(device="cuda").manual_seed(n)
    src = [torch.rand(n, n, dtype=torch.float64, device="cuda", generator=g) - 0.5 for _ in range(2)]
    rhs = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    out = {}
    for graph in (True, False):
        s = lu.LUSolver(lu.LUConfig(n, 128, precision=lu.LU_PREC_FP16X3, lookahead=lookahead, use_graph=graph))
        A = _padded(n)
        for i in range(4):
            A.copy_(src[i % 2])
            s.refine_factor(A)
            X, info = s.refine_apply(A, rhs.clone())
            assert info["status"] == lu.LU_OK
            out[graph, i] = X.clone()
        s.close()
    for i in range(4):
        assert torch.equal(out[False, i], out[True, i])
