"""Batched uneven factor + solve in one persistent launch (no reference
counterpart).  Each system is checked against the per-system contract the
single-matrix path meets: scaled residual r_hpl < 16, and the solution
against an FP64 LAPACK solve."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LU_PREC_FP64, LU_PREC_FP32 = 0, 4


def _systems(count, lo, hi, seed):
    rng = np.random.default_rng(seed)
    n = np.exp(rng.uniform(np.log(lo), np.log(hi + 1), count)).astype(np.int32)
    n = np.clip(n, lo, hi)
    a_off = np.concatenate([[0], np.cumsum(n.astype(np.int64) ** 2)[:-1]]).astype(np.int64)
    b_off = np.concatenate([[0], np.cumsum(n.astype(np.int64))[:-1]]).astype(np.int64)
    return n, a_off, b_off


def _run(n, a_off, b_off, precision, seed=42):
    import charmlu_b200 as lu
    from charmlu_b200 import _lib
    L = _lib.load()
    count = len(n)
    tot_a = int(a_off[-1] + int(n[-1]) ** 2)
    tot_b = int(b_off[-1] + int(n[-1]))
    A = lu.generate_uniform(1, tot_a, seed=seed, stream_id=10).view(-1)
    b = lu.generate_uniform(1, tot_b, seed=seed, stream_id=11).view(-1)
    A0, b0 = A.clone(), b.clone()
    dn = torch.from_numpy(n).cuda()
    da = torch.from_numpy(a_off).cuda()
    dbo = torch.from_numpy(b_off).cuda()
    info = torch.full((count,), -99, dtype=torch.int32, device="cuda")
    wb = L.lu_batched_work_bytes(count, ctypes.c_void_p(n.ctypes.data), precision)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    rc = L.lu_batched_factor_solve(count, ctypes.c_void_p(dn.data_ptr()), ctypes.c_void_p(da.data_ptr()),
                                   ctypes.c_void_p(dbo.data_ptr()), ctypes.c_void_p(A.data_ptr()),
                                   ctypes.c_void_p(b.data_ptr()), ctypes.c_void_p(info.data_ptr()), precision,
                                   ctypes.c_void_p(work.data_ptr()), wb,
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0
    if precision == LU_PREC_FP32:
        # every system lands in exactly one bin of the refinement-step histogram
        hist = np.zeros(12, dtype=np.int32)
        assert L.lu_batched_refine_histogram(ctypes.c_void_p(work.data_ptr()), ctypes.c_void_p(hist.ctypes.data),
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        assert hist.sum() == count and hist[11] == int((info.cpu().numpy() != 0).sum()), hist
    return A0.cpu().numpy(), b0.cpu().numpy(), b.cpu().numpy(), info.cpu().numpy(), A


def _check(n, a_off, b_off, A0, b0, x, info, fe_tol):
    eps = np.finfo(np.float64).eps
    assert np.all(info == 0), info[info != 0][:10]
    worst = 0.0
    for i in range(len(n)):
        k = int(n[i])
        Ai = A0[a_off[i]:a_off[i] + k * k].reshape(k, k)
        bi = b0[b_off[i]:b_off[i] + k]
        xi = x[b_off[i]:b_off[i] + k]
        r = np.abs(bi - Ai @ xi).max()
        r_hpl = r / ((np.abs(Ai).sum(1).max() * np.abs(xi).max() + np.abs(bi).max()) * k * eps)
        worst = max(worst, r_hpl)
        assert r_hpl < 16, (i, k, r_hpl)
        xr = np.linalg.solve(Ai, bi)
        assert np.abs(xi - xr).max() / np.abs(xr).max() < fe_tol, (i, k)
    return worst


@pytest.mark.parametrize("lo,hi,count", [(1, 40, 300), (32, 1024, 160), (150, 300, 64)])
def test_batched_fp64(cuda_dev, lo, hi, count):
    n, a_off, b_off = _systems(count, lo, hi, seed=lo * 7 + hi)
    A0, b0, x, info, _ = _run(n, a_off, b_off, LU_PREC_FP64)
    _check(n, a_off, b_off, A0, b0, x, info, fe_tol=1e-9)


@pytest.mark.parametrize("lo,hi,count", [(32, 1024, 160), (1, 40, 100)])
def test_batched_fp32_one_refinement(cuda_dev, lo, hi, count):
    n, a_off, b_off = _systems(count, lo, hi, seed=lo * 11 + hi)
    A0, b0, x, info, A_after = _run(n, a_off, b_off, LU_PREC_FP32)
    # the FP64 matrices are left untouched in FP32 mode
    assert np.array_equal(A_after.cpu().numpy(), A0)
    _check(n, a_off, b_off, A0, b0, x, info, fe_tol=1e-7)


def test_batched_matches_single_matrix_path(cuda_dev):
    """Same pivots and factors as lu_factor on each system (FP64)."""
    import charmlu_b200 as lu
    n, a_off, b_off = _systems(24, 16, 200, seed=5)
    A0, b0, x, info, A_fact = _run(n, a_off, b_off, LU_PREC_FP64)
    Af = A_fact.cpu().numpy()
    for i in range(len(n)):
        k = int(n[i])
        Ai = A0[a_off[i]:a_off[i] + k * k].reshape(k, k)
        buf = torch.zeros(k, k + (k & 1), dtype=torch.float64, device="cuda")
        Ad = buf[:, :k]
        Ad.copy_(torch.from_numpy(Ai))
        s = lu.LUSolver(lu.LUConfig(k, 16))
        s.factor(Ad)
        assert s.status() == 0
        ref = Ad.cpu().numpy()
        got = Af[a_off[i]:a_off[i] + k * k].reshape(k, k)
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max(), i


def test_batched_rejects_bad_order(cuda_dev):
    n = np.array([10, 5000, 7], dtype=np.int32)
    a_off = np.array([0, 100, 100 + 5000 * 5000], dtype=np.int64)
    b_off = np.array([0, 10, 5010], dtype=np.int64)
    from charmlu_b200 import _lib
    L = _lib.load()
    # the prep kernel marks every system LU_ERR_ARG and the solve kernel does nothing
    count = 3
    dn = torch.from_numpy(n).cuda()
    da = torch.from_numpy(a_off).cuda()
    dbo = torch.from_numpy(b_off).cuda()
    A = torch.zeros(16, dtype=torch.float64, device="cuda")
    b = torch.zeros(16, dtype=torch.float64, device="cuda")
    info = torch.zeros(count, dtype=torch.int32, device="cuda")
    work = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    rc = L.lu_batched_factor_solve(count, ctypes.c_void_p(dn.data_ptr()), ctypes.c_void_p(da.data_ptr()),
                                   ctypes.c_void_p(dbo.data_ptr()), ctypes.c_void_p(A.data_ptr()),
                                   ctypes.c_void_p(b.data_ptr()), ctypes.c_void_p(info.data_ptr()), 0,
                                   ctypes.c_void_p(work.data_ptr()), 1 << 20,
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0
    assert np.all(info.cpu().numpy() == -1)


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_batched_edges_of_blocks_and_tiles(cuda_dev, prec):
    """Orders at the edges of the kernel's shapes: panel widths, the shared-memory
    threshold, outer blocks of 64 / 128, 64- and 128-wide tiles, 512 and 1024
    panel rows.  FP64 factors against the bound |P A - L U| <= gamma_n |L||U|
    (elimination, each update one fma or a sum of products subtracted once: at
    most n roundings per element, Higham theorem 9.3), solutions by r_hpl < 16."""
    import scipy.linalg
    from charmlu_b200 import LU_PREC_FP32, LU_PREC_FP64
    from charmlu_b200.batched import BatchedSystems
    ns = [1, 2, 3, 15, 16, 17, 31, 33, 63, 64, 65, 95, 97, 127, 128, 129, 159, 160, 161, 191, 193, 255, 257, 320, 383,
          385, 511, 512, 513, 577, 650, 652, 769, 1023, 1025]
    rng = np.random.default_rng(11)
    mats = [rng.uniform(-0.5, 0.5, (n, n)) for n in ns]
    rhs = [rng.uniform(-0.5, 0.5, n) for n in ns]
    bs = BatchedSystems(ns)
    A = torch.from_numpy(np.concatenate([m.ravel() for m in mats])).cuda()
    b = torch.from_numpy(np.concatenate(rhs)).cuda()
    info = bs.factor_solve(A, b, LU_PREC_FP64 if prec == "fp64" else LU_PREC_FP32).cpu().numpy()
    assert (info == 0).all()
    x, F = b.cpu().numpy(), A.cpu().numpy()
    u = 2.0 ** -53
    for i, n in enumerate(ns):
        xi = x[bs.b_off[i]:bs.b_off[i] + n]
        r = np.abs(rhs[i] - mats[i] @ xi).max()
        assert r < 16 * n * 2 * u * (np.abs(mats[i]).sum(1).max() * np.abs(xi).max() + np.abs(rhs[i]).max()), n
        if prec == "fp64":
            LU = F[bs.a_off[i]:bs.a_off[i] + n * n].reshape(n, n)
            L = np.tril(LU, -1) + np.eye(n)
            U = np.triu(LU)
            assert np.abs(L).max() <= 1, n
            _, piv = scipy.linalg.lu_factor(mats[i])
            P = np.arange(n)
            for j, p in enumerate(piv):
                P[[j, p]] = P[[p, j]]
            # the products below round too (in FP64): n more roundings
            bound = 2 * (n + 1) * u / (1 - 2 * (n + 1) * u) * (np.abs(L) @ np.abs(U)) + u
            assert (np.abs(mats[i][P] - L @ U) <= bound).all(), n
        else:
            np.testing.assert_array_equal(F[bs.a_off[i]:bs.a_off[i] + n * n], mats[i].ravel())


def test_batched_singular_and_ties(cuda_dev):
    """A zero column is reported at its place; all-equal candidates take the lowest row."""
    from charmlu_b200 import LU_PREC_FP64
    from charmlu_b200.batched import BatchedSystems
    ns = [20, 70, 200, 300]
    rng = np.random.default_rng(3)
    mats = []
    for n in ns:
        m = rng.uniform(-0.5, 0.5, (n, n))
        m[:, n // 2] = 0
        mats.append(m)
    eye = [np.eye(n) for n in ns]  # every step has one candidate; no interchange, x = b
    bs = BatchedSystems(ns + ns)
    A = torch.from_numpy(np.concatenate([m.ravel() for m in mats + eye])).cuda()
    rhs = np.concatenate([rng.uniform(-0.5, 0.5, n) for n in ns + ns])
    b = torch.from_numpy(rhs).cuda()
    info = bs.factor_solve(A, b, LU_PREC_FP64).cpu().numpy()
    assert info.tolist() == [n // 2 + 1 for n in ns] + [0] * 4
    o = int(bs.b_off[4])
    np.testing.assert_array_equal(b.cpu().numpy()[o:], rhs[o:])


@pytest.mark.parametrize("prec", [LU_PREC_FP64, LU_PREC_FP32])
@pytest.mark.parametrize("orders", [[1335, 1336, 1400, 1427], [1385, 1386, 1428, 1536], [1537, 2047, 2048]])
def test_batched_orders_above_1025(cuda_dev, prec, orders):
    """Orders around those at which the panel width halves (FP64 1386, FP32 1428),
    at which fewer rows of L are staged (FP32 1336 .. 1427), and the largest;
    several panels of 512 rows per thread.  The contract of every system."""
    n = np.array(orders, dtype=np.int32)
    a_off = np.concatenate([[0], np.cumsum(n.astype(np.int64) ** 2)[:-1]]).astype(np.int64)
    b_off = np.concatenate([[0], np.cumsum(n.astype(np.int64))[:-1]]).astype(np.int64)
    A0, b0, x, info, _ = _run(n, a_off, b_off, prec, seed=int(n[0]))
    assert np.all(info == 0), info
    eps = np.finfo(np.float64).eps
    for i, k in enumerate(orders):
        Ai, bi, xi = A0[a_off[i]:a_off[i] + k * k].reshape(k, k), b0[b_off[i]:b_off[i] + k], x[b_off[i]:b_off[i] + k]
        scale = np.abs(Ai).sum(1).max() * np.abs(xi).max() + np.abs(bi).max()
        assert np.abs(bi - Ai @ xi).max() < 16 * k * eps * scale, k
