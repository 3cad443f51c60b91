"""The panel leaf (getf2 on register-resident rows) at the edges of its row
ranges: one CTA, a cluster, a cooperative grid, 1 to 6 rows per thread, widths
that do not fill the 16- or 32-column instance.

P A = L U is held to the rounding bound of elimination with one fma per
update, |P A - L U| <= gamma_w |L||U| with gamma_w = w u / (1 - w u) (Higham,
Accuracy and Stability, theorem 9.3); the products are formed in FP64 (FP32
leaf) or extended precision (FP64 leaf), and one more unit covers storing A.
Pivots are checked by |l| <= 1, and on exact integer data against the
lowest-row rule."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _leaf32(A, ncols, lc0, max_ctas, alone):
    from charmlu_b200 import _lib
    f = _lib.load().lub_test_getf2_leaf
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_void_p, ctypes.c_int64] + [ctypes.c_int] * 4 + [ctypes.c_void_p] + [ctypes.c_int] * 2 + \
        [ctypes.c_void_p]
    ipiv = torch.empty(ncols, dtype=torch.int32, device="cuda")
    rc = f(A.data_ptr(), A.stride(0), A.shape[0], ncols, A.shape[1], lc0, ipiv.data_ptr(), max_ctas, alone,
           torch.cuda.current_stream().cuda_stream)
    return rc, ipiv.cpu().numpy()


def _leaf64(A, ncols, lookahead):
    from charmlu_b200.blocks import CudaBlocks
    bl = CudaBlocks(max(A.shape[0], 2), 32, lookahead=lookahead)
    ipiv = torch.empty(ncols, dtype=torch.int32, device="cuda")
    bl.clear_status()
    bl.panel_factor(A[:, :ncols], ipiv, 0)
    return bl.status(), ipiv.cpu().numpy()


def _perm(M, ipiv):
    r = np.arange(M)
    for j, p in enumerate(ipiv):
        r[[j, p]] = r[[p, j]]
    return r


def _check(A0, LU, ipiv, ncols, wide, u):
    M = A0.shape[0]
    k = min(M, ncols)
    r = _perm(M, ipiv[:k])
    L = np.tril(LU[:, :k], -1).astype(wide)
    L[np.arange(k), np.arange(k)] = 1
    U = np.triu(LU[:k, :ncols]).astype(wide)
    assert np.abs(L).max() <= 1
    gamma = (ncols + 1) * u / (1 - (ncols + 1) * u)
    bound = gamma * (np.abs(L) @ np.abs(U)) + u * np.abs(A0[r, :ncols])
    assert (np.abs(A0[r, :ncols].astype(wide) - L @ U) <= bound).all()


GRIDS = [(148, 1), (148, 0), (3, 0)]  # max CTAs, alone on the GPU


@pytest.mark.parametrize("ncols", [1, 7, 16, 17, 32])
@pytest.mark.parametrize("M", [32, 255, 257, 512, 513, 1025, 2049, 4097, 24576, 24577])
def test_fp32_leaf(cuda_dev, M, ncols):
    rng = np.random.default_rng(M * 100 + ncols)
    pw, lc0 = ncols + 41, 20
    A0 = rng.uniform(-0.5, 0.5, (M, pw)).astype(np.float32)
    for max_ctas, alone in GRIDS:
        A = torch.from_numpy(A0).cuda()
        rc, ipiv = _leaf32(A, ncols, lc0, max_ctas, alone)
        assert rc == 0
        out = A.cpu().numpy()
        leaf = slice(lc0, lc0 + ncols)
        _check(A0[:, leaf], out[:, leaf], ipiv, ncols, np.float64, 2.0 ** -24)
        # the enclosing panel's other columns carry the same interchanges
        r = _perm(M, ipiv)
        others = np.r_[0:lc0, lc0 + ncols:pw]
        np.testing.assert_array_equal(out[:, others], A0[r][:, others])


@pytest.mark.parametrize("ncols", [2, 15, 16, 31, 32])
@pytest.mark.parametrize("M", [32, 256, 511, 513, 2049, 8191, 12288, 12289, 24577, 37889])
def test_fp64_leaf(cuda_dev, M, ncols):
    rng = np.random.default_rng(M * 100 + ncols)
    A0 = rng.uniform(-0.5, 0.5, (M, ncols + (ncols & 1)))
    for la in (False, True):
        A = torch.from_numpy(A0).cuda()
        st, ipiv = _leaf64(A, ncols, la)
        assert st == 0
        _check(A0[:, :ncols], A.cpu().numpy()[:, :ncols], ipiv, ncols, np.longdouble, 2.0 ** -53)


@pytest.mark.parametrize("M", [40, 300, 700, 5000])
def test_ties_zero_and_nonfinite_columns(cuda_dev, M):
    # +-1 columns that stay integers: every pivot search is a tie, the lowest row wins
    rng = np.random.default_rng(M)
    A0 = np.zeros((M, 8))
    A0[:, 0] = rng.choice([-1.0, 1.0], M)
    A0[:, 1] = rng.choice([-1.0, 1.0], M)
    A0[:, 3] = rng.choice([-1.0, 1.0], M)  # column 2 is zero
    A0[:, 4:] = rng.choice([-1.0, 1.0], (M, 4))
    A0[M - 3, 7] = np.nan
    ref, want = A0.copy(), []
    first_bad = 0
    for j in range(8):
        c = np.abs(ref[j:, j])
        c[np.isnan(c)] = 0
        p = j + int(np.argmax(c)) if c.max() > 0 else j
        want.append(p)
        ref[[j, p]] = ref[[p, j]]
        if c.max() > 0:
            ref[j + 1:, j] /= ref[j, j]
            ref[j + 1:, j + 1:] -= np.outer(ref[j + 1:, j], ref[j, j + 1:])
        elif not first_bad:
            first_bad = j + 1
    for la in (False, True):
        A = torch.from_numpy(A0).cuda()
        st, ipiv = _leaf64(A, 8, la)
        assert st == first_bad
        assert ipiv.tolist() == want
        np.testing.assert_allclose(A.cpu().numpy(), ref, rtol=0, atol=64 * 2.0 ** -53)
    for max_ctas, alone in GRIDS:
        A = torch.from_numpy(A0.astype(np.float32)).cuda()
        rc, ipiv = _leaf32(A, 8, 0, max_ctas, alone)
        assert rc == first_bad
        assert ipiv.tolist() == want
        np.testing.assert_allclose(A.cpu().numpy(), ref, rtol=0, atol=64 * 2.0 ** -24)


@pytest.mark.parametrize("M", [227328, 227329, 240000, 245761])
def test_panels_taller_than_sixteen_columns_allow(cuda_dev, M):
    """FP64 panels around 148 CTAs x 6 rows per thread, above which leaves are 8
    columns wide with 12 rows per thread."""
    w = 16
    A0 = torch.rand(M, w, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(M)) - 0.5
    A = A0.clone()
    rc, piv = _leaf64(A, w, True)
    assert rc == 0
    order = np.arange(M)
    for j, p in enumerate(piv):
        assert j <= p < M
        order[[j, p]] = order[[p, j]]
    PA = A0[torch.from_numpy(order).cuda()]
    L = torch.tril(A, -1)
    L.diagonal().fill_(1.0)
    U = torch.triu(A[:w])
    assert L.abs().max() <= 1
    # w roundings by elimination, as many again in the FP64 products here
    u = 2.0 ** -53
    bound = 2 * (w + 1) * u / (1 - 2 * (w + 1) * u) * (L.abs() @ U.abs()) + u
    assert ((PA - L @ U).abs() <= bound).all()
