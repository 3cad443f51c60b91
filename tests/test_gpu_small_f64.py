"""The small-tile FP64 product and the one-launch triangular solve give the bits
of the forms they stand in for: the 128 x 128 tiles, and the recursion over
halves (solve, product, solve)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mat(rng, r, c):
    buf = torch.zeros(r, c + (c & 1) + 2, dtype=torch.float64, device="cuda")
    buf[:, :c] = torch.from_numpy(rng.uniform(-0.5, 0.5, (r, c)))
    return buf[:, :c]


@pytest.mark.parametrize("K", [1, 15, 16, 31, 32, 33, 100])
@pytest.mark.parametrize("N", [1, 17, 32, 63, 64])
def test_small_tiles_give_the_bits_of_large_ones(cuda_dev, N, K):
    from charmlu_b200.blocks import CudaBlocks
    M, wide = 8191, 768  # 64 x 6 tiles of 128: the large kernel
    rng = np.random.default_rng(N * 1000 + K)
    bl = CudaBlocks(M, 64)
    A, B, C = _mat(rng, M, K), _mat(rng, K, wide), _mat(rng, M, wide)
    D = _mat(rng, M, wide)
    D.copy_(C)
    pad = torch.full((M, ((N + 1) // 2) * 2 + 2), 7.0, dtype=torch.float64, device="cuda")
    S = pad[:, :N]
    S.copy_(C[:, :N])
    bl.gemm_update(A, B, D)
    bl.gemm_update(A, B[:, :N], S)
    assert torch.equal(S, D[:, :N])
    assert (pad[:, N:] == 7.0).all()  # nothing right of C is written
    # and the rows of a short product
    T = _mat(rng, 70, wide)
    T.copy_(C[:70])
    bl.gemm_update(A[:70], B, T)
    assert torch.equal(T, D[:70])


@pytest.mark.parametrize("ncols", [1, 15, 33, 2368, 2369])
@pytest.mark.parametrize("w", [33, 48, 64, 100, 128, 191, 192, 256])
def test_one_launch_solve_gives_the_recursions_bits(cuda_dev, w, ncols):
    from charmlu_b200.blocks import CudaBlocks
    rng = np.random.default_rng(w * 10000 + ncols)
    bl = CudaBlocks(256, 64)
    L = _mat(rng, w, w)
    B = _mat(rng, w, ncols)
    ref = _mat(rng, w, ncols)
    ref.copy_(B)

    def solve(l0, h):
        if h <= 32:
            bl.trsm_lower_unit(L[l0:l0 + h, l0:l0 + h], ref[l0:l0 + h])
            return
        h1 = max(h // 2 & ~15 if h // 2 >= 16 else h // 2 & ~1, 2)
        solve(l0, h1)
        bl.gemm_update(L[l0 + h1:l0 + h, l0:l0 + h1], ref[l0:l0 + h1], ref[l0 + h1:l0 + h])
        solve(l0 + h1, h - h1)

    solve(0, w)
    out = _mat(rng, w, ncols + 1)[:, :ncols]
    out.copy_(B)
    bl.trsm_lower_unit(L, out)
    assert torch.equal(out, ref)


@pytest.mark.parametrize("M,N,K", [(1280, 1280, 130), (1536, 1408, 64), (1536, 1536, 257), (1792, 1800, 255),
                                   (2048, 2048, 192), (2048, 2048, 300), (2177, 2175, 96), (2304, 2304, 40),
                                   (3328, 3328, 33), (3328, 3328, 1030)])
def test_every_choice_of_tiles_gives_the_same_bits(cuda_dev, M, N, K):
    """Products on both sides of the lines between small and large tiles, and with
    and without the late start of an SM's second CTA, against slices of 64 columns."""
    from charmlu_b200.blocks import CudaBlocks
    bl = CudaBlocks(4096, 64)
    gen = torch.Generator(device="cuda").manual_seed(M + K)

    def mat(r, c):
        return torch.rand(r, c + (c & 1), dtype=torch.float64, device="cuda", generator=gen)[:, :c].sub_(0.5)

    A, B, C = mat(M, K), mat(K, N), mat(M, N)
    D = torch.empty(M, N + (N & 1), dtype=torch.float64, device="cuda")[:, :N]
    D.copy_(C)
    bl.gemm_update(A, B, C)
    for c in range(0, N, 64):
        bl.gemm_update(A, B[:, c:c + 64], D[:, c:c + 64])
    assert torch.equal(C, D)
    bl.close()
