"""Shared memory of the batched solver's panels, on the host: for every accepted
order and panel width no pointer reaches past what the kernel asks for."""
import ctypes

import numpy as np
import pytest


@pytest.mark.parametrize("esize", [8, 4])
@pytest.mark.parametrize("nb", [4, 8, 16, 32])
def test_panel_layout_fits_the_shared_memory(esize, nb):
    from charmlu_b200 import _lib
    probe = _lib.load().lub_test_batched_layout
    out = np.zeros(4, dtype=np.int32)
    for n in range(1, 2049):
        assert probe(n, nb, esize, ctypes.c_void_p(out.ctypes.data)) == 0
        width, reached, stage_rows, asked = (int(v) for v in out)
        assert reached <= asked <= 227 * 1024, (n, width, reached)
        assert 64 <= stage_rows <= 256
        # the widths, and with them the order of the sums, of a panel and 128 columns of it
        want = nb
        while want > 4 and (n * (want + 1) + want * 128) * esize > asked:
            want //= 2
        assert width == want, n
