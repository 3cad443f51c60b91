"""Which launch a panel leaf takes, on the host: every leaf of the widest width that
is promised for its rows fits the SMs of a cooperative grid and the registers."""
import ctypes

import numpy as np
import pytest

NT = 256  # threads per CTA


@pytest.mark.parametrize("esize,rows32,rows16", [(8, 3, 6), (4, 6, 6)])
@pytest.mark.parametrize("sms", [132, 148, 160, 170])
@pytest.mark.parametrize("cluster", [0, 8, 16])
def test_every_promised_leaf_has_a_launch(esize, rows32, rows16, sms, cluster):
    from charmlu_b200 import _lib
    probe = _lib.load().lub_test_leaf_plan
    out = np.zeros(7, dtype=np.int32)
    limit = min(sms, 160)
    edges = {1, 2}
    for rows in (1, 2, 3, 4, 6, 12):
        for ctas in (1, 2, 4, 8, 16, 48, 148, 149, limit - 1, limit, limit + 1, 160, 161):
            for d in (-1, 0, 1):
                edges.add(max(1, rows * ctas * NT + d))
    for M in sorted(edges):
        for max_ctas in (16, 48, 160):
            probe(esize, M, 1, sms, max_ctas, cluster, ctypes.c_void_p(out.ctypes.data))
            widest = int(out[0])
            assert widest == (32 if M <= limit * NT * rows32 else 16 if M <= limit * NT * rows16 else 8), M
            for ncols in (1, 8, 9, 16, 17, 32):
                probe(esize, M, ncols, sms, max_ctas, cluster, ctypes.c_void_p(out.ctypes.data))
                _, rc, W, transport, G, R, rpt = (int(v) for v in out)
                if M > limit * NT * 12:
                    assert rc == -8, M  # LU_ERR_UNSUPPORTED
                    continue
                if ncols > widest:
                    assert rc in (0, -8)
                else:
                    assert rc == 0, (M, ncols)
                if rc != 0:
                    continue
                assert ncols <= W
                assert 1 <= G <= (limit if transport == 1 else max(cluster, 1)), (M, ncols)
                assert G * R >= M and rpt * NT >= R
                if transport == 1:
                    assert (G - 1) * R < M  # no CTA without rows
                assert rpt <= {32: rows32, 16: rows16, 8: 12}[W]
                assert transport == (0 if M <= 2 * NT else 2 if cluster and M <= cluster * NT * rpt else 1)


def test_the_update_leaves_a_panel_beside_it_enough_sms():
    """Under look-ahead the FP32 leaf's cooperative grid fits the SMs that the update
    does not hold, at every height."""
    from charmlu_b200 import _lib
    L = _lib.load()
    out = np.zeros(7, dtype=np.int32)
    for M in [16385, 65536, 73728, 73729, 80000, 82000, 90000, 120000, 148 * 6 * NT]:
        reserve = L.lub_test_panel_reserve(48, 148, M)
        L.lub_test_leaf_plan(4, M, 32, 148, 48, 0, ctypes.c_void_p(out.ctypes.data))
        assert out[1] == 0 and out[4] <= reserve <= 148, M
        assert reserve == 48 or M > 73728
    assert L.lub_test_panel_reserve(0, 148, 90000) == 0  # no SMs kept on request
