"""A call that fails leaves the caller's result buffer as it was.  Without a device the first allocation fails;
the buffer is larger than the 2 MB below which no helper thread runs."""
import ctypes as C

import numpy as np
import pytest

from chroma_gb300 import gbclover as G


def test_failed_stout_leaves_the_result_alone():
    import torch
    if torch.cuda.is_available():
        pytest.skip("needs the allocation on the device to fail")
    dims = (8, 8, 8, 16)
    u = np.full((8192, 4, 3, 3), 0.25 - 3j)
    out = np.full((8192, 4, 3, 3), (1 + 2j) / 3)
    dp = lambda a: a.view(np.float64).ctypes.data_as(C.POINTER(C.c_double))
    geom = G.Geom((C.c_int * 4)(*dims), 1)
    rc = G.load().gbc_stout_smear(C.byref(geom), 1, 0.1, (C.c_int * 4)(1, 1, 1, 1), dp(u), dp(out))
    assert rc == G.ERR_CUDA
    assert np.all(out == (1 + 2j) / 3)  # no zero bytes
