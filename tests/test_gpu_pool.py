"""Handles made from what earlier ones left (device blocks, streams, events):
blocks with another order's leftovers, several threads and streams at once."""
import ctypes
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _system(n, seed):
    rng = np.random.default_rng(seed)
    A = rng.uniform(-0.5, 0.5, (n, n)) + np.eye(n) * np.sqrt(n)
    b = rng.uniform(-0.5, 0.5, n)
    buf = torch.zeros(n, n + (n & 1), dtype=torch.float64, device="cuda")[:, :n]
    buf.copy_(torch.from_numpy(A))
    return buf, torch.from_numpy(b).cuda(), np.linalg.solve(A, b)


def test_reused_blocks_of_another_order(cuda_dev):
    import charmlu_b200 as lu
    orders = [900, 333, 1024, 901, 334, 900]
    for it in range(2):
        for n in orders:
            A, b, ref = _system(n, n)
            for prec in (lu.LU_PREC_FP16X3, lu.LU_PREC_FP64):
                s = lu.LUSolver(lu.LUConfig(n, 64, precision=prec, lookahead=bool(it), use_graph=bool(n & 1),
                                            ir_target=1e-3))
                if prec == lu.LU_PREC_FP64:
                    W, x = A.clone() if n % 2 == 0 else torch.nn.functional.pad(A, (0, 1))[:, :n], b.clone()
                    s.factor_solve(W, x)
                    assert s.status() == 0
                else:
                    x, info = s.refine_solve(A, b)
                    assert info["status"] == 0
                # well conditioned (kappa < 10): a backward stable solution is this close
                assert np.abs(x.cpu().numpy() - ref).max() <= 1e-11 * np.abs(ref).max(), (n, prec)
                s.close()


def test_threads_with_their_own_streams(cuda_dev):
    import charmlu_b200 as lu
    bad = []

    def work(k):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for it in range(6):
                    n = 256 + 32 * ((k + it) % 5)
                    A, b, ref = _system(n, 10 * k + it)
                    s = lu.LUSolver(lu.LUConfig(n, 64))
                    s.factor_solve(A, b, stream=stream)
                    if s.status(stream) != 0 or np.abs(b.cpu().numpy() - ref).max() > 1e-11 * np.abs(ref).max():
                        bad.append((k, it))
                    s.close()
        except Exception as e:  # reported by the main thread
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("n", [700, 1001])
def test_zeroed_blocks_do_not_wait_for_the_default_stream(cuda_dev, n):
    """GMRES multiplies against a vector of zeros, which may be another handle's
    block; it has to be zero on a non-blocking stream too, with the default
    stream busy."""
    import charmlu_b200 as lu

    def solve(stream):
        s = lu.LUSolver(lu.LUConfig(n, 64, precision=lu.LU_PREC_FP16X3, ir_mode=lu.LU_IR_GMRES))
        x, info = s.refine_solve(A, b, stream=stream)
        return s, x, info

    A, b, ref = _system(n, n)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    s, _, _ = solve(stream)
    s.close()
    # takes two of the blocks and hands them back behind the others, so that the
    # next handle's vectors are not the ones they were
    W, x = torch.nn.functional.pad(A, (0, n & 1))[:, :n], b.clone()  # a copy with rows on 16 bytes
    s = lu.LUSolver(lu.LUConfig(n, 64))
    s.factor_solve(W, x)
    s.close()
    torch.cuda.synchronize()
    torch.cuda._sleep(int(5e8))  # about a quarter of a second
    s, x, info = solve(stream)
    torch.cuda.synchronize()
    assert info["status"] == 0 and info["used_gmres"] == 1
    assert np.abs(x.cpu().numpy() - ref).max() <= 1e-10 * np.abs(ref).max()
    s.close()


def _singular_factor(n, stream):
    """A handle whose status word holds a singular column; the stream has finished."""
    import charmlu_b200 as lu
    A = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    s = lu.LUSolver(lu.LUConfig(n, 64))
    s.factor(A, stream=stream)
    assert s.status(stream) == 1
    return s


def test_a_status_outlives_the_default_streams_work(cuda_dev):
    """Nothing that lu_create left on the default stream clears a later status."""
    stream = torch.cuda.Stream()
    _singular_factor(256, stream).close()
    A = torch.zeros(256, 256, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    import charmlu_b200 as lu
    torch.cuda._sleep(int(5e8))
    s = lu.LUSolver(lu.LUConfig(256, 64))
    s.factor(A, stream=stream)
    torch.cuda.synchronize()
    assert s.status(stream) == 1
    s.close()


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_a_handle_goes_beside_a_capture(cuda_dev, mode):
    """Destroying a handle leaves a capture alone: another thread's, and in relaxed
    mode this thread's."""
    import charmlu_b200 as lu
    n = 256
    s = lu.LUSolver(lu.LUConfig(n, 64))
    s.factor(torch.rand(n, n, dtype=torch.float64, device="cuda"))
    assert s.status() == 0
    y = torch.ones(64, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=mode):
        x = y * 2
        if mode == "relaxed":
            s.close()
        else:
            t = threading.Thread(target=s.close)
            t.start()
            t.join()
        z = x + 1
    g.replay()
    assert torch.equal(z, torch.full_like(z, 3.0))


def test_handles_come_and_go_beside_graph_schedules(cuda_dev):
    """One thread's solver captures its schedule anew for every matrix while
    another thread makes and destroys handles."""
    import charmlu_b200 as lu
    bad, done = [], threading.Event()

    def schedules():
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                s = lu.LUSolver(lu.LUConfig(1024, 128, use_graph=True))
                keep = []
                for it in range(30):
                    A = torch.rand(1024, 1024, dtype=torch.float64, device="cuda")
                    keep.append(A)  # another address, so another capture
                    s.factor(A, stream=stream)
                    if s.status(stream) != 0:
                        bad.append(("status", it))
                s.close()
        except Exception as e:  # reported by the main thread
            bad.append(("schedules", repr(e)))
        done.set()

    def handles():
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                A = torch.rand(256, 256, dtype=torch.float64, device="cuda")
                while not done.is_set():
                    s = lu.LUSolver(lu.LUConfig(256, 64))
                    s.factor(A.clone(), stream=stream)
                    if s.status(stream) != 0:
                        bad.append("status of a short-lived handle")
                    s.close()
        except Exception as e:
            bad.append(("handles", repr(e)))

    threads = [threading.Thread(target=f) for f in (schedules, handles)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_destroy_waits_for_the_handles_work(cuda_dev):
    import charmlu_b200 as lu
    n = 256
    stream = torch.cuda.Stream()
    A = torch.rand(n, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        s = lu.LUSolver(lu.LUConfig(n, 64))
        with torch.cuda.stream(stream):
            torch.cuda._sleep(int(2e8))  # about a tenth of a second
            s.factor(A, stream=stream)
        s.close()
        assert stream.query()


@pytest.mark.parametrize("pooled", [False, True])
def test_handles_are_not_made_inside_a_capture(cuda_dev, pooled):
    """Refused while the calling thread captures, whatever earlier handles left
    behind; so are blocks that an existing handle lacks."""
    import charmlu_b200 as lu
    n = 320
    rt = ctypes.CDLL(next(ln.split()[-1] for ln in open("/proc/self/maps") if "libcudart" in ln))
    A, B = torch.rand(n, n, dtype=torch.float64, device="cuda"), torch.rand(n, 8, dtype=torch.float64, device="cuda")
    first, kept = lu.LUSolver(lu.LUConfig(n, 64)), lu.LUSolver(lu.LUConfig(n, 64))
    piv = first.factor(A)
    first.solve(A, piv, B.clone())
    assert first.status() == 0
    if pooled:
        first.close()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()

    def refused(call):
        sp, graph = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
        assert rt.cudaStreamBeginCapture(sp, 1) == 0  # thread-local mode
        try:
            with pytest.raises(lu.LUError):
                call()
        finally:
            rt.cudaStreamEndCapture(sp, ctypes.byref(graph))
            rt.cudaGetLastError()

    refused(lambda: lu.LUSolver(lu.LUConfig(n, 64)))
    refused(lambda: kept.solve(A, piv, B.clone(), stream=stream))
    # both work afterwards
    X = B.clone()
    kept.solve(A, piv, X)
    assert kept.status() == 0
    lu.LUSolver(lu.LUConfig(n, 64)).close()
    kept.close()
    first.close()


def test_pool_memory_goes_back(cuda_dev, monkeypatch):
    """lu_pool_release frees what closed solvers left; a bound of 0 leaves nothing."""
    import charmlu_b200 as lu
    n = 4096
    A = lu.generate_uniform(n, n, seed=1)
    A.diagonal().add_(float(n) ** 0.5)
    b = lu.generate_uniform(n, 1, seed=2).view(-1)

    def use():
        s = lu.LUSolver(lu.LUConfig(n, 128, precision=lu.LU_PREC_FP16X3))
        x, info = s.refine_solve(A, b)
        assert info["status"] == 0
        s.close()
        return torch.cuda.mem_get_info()[0]

    use()  # kernels loaded, torch's own blocks in place
    lu.pool_release()
    free = torch.cuda.mem_get_info()[0]
    assert use() <= free - 4 * n * n  # the FP32 factors alone
    lu.pool_release()
    assert torch.cuda.mem_get_info()[0] == free
    monkeypatch.setenv("LU_B200_POOL_BYTES", "0")
    assert use() == free
    monkeypatch.setenv("LU_B200_POOL_BYTES", str(1 << 20))
    assert use() >= free - (4 << 20)
    lu.pool_release()
