"""Inference into host memory reaches nothing past the result's end: pages that follow it stay
as untouched as they were (a result that ends at unmapped memory would end the process)."""
import ctypes
import mmap
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def resident_pages(addr, size, page):
    flags = (ctypes.c_ubyte * (size // page))()
    assert ctypes.CDLL(None).mincore(ctypes.c_void_p(addr), ctypes.c_size_t(size), flags) == 0
    return int((np.frombuffer(flags, np.uint8) & 1).sum())


# per-layer and fused inference; one chunk and several (of max_batch rows; of 64 MB of staging)
@pytest.mark.parametrize("dims,members,rows,fused", [([256, 256, 256], 1, 512, 0), ([256, 256, 256], 1, 20000, 0),
                                                     ([256, 256, 256], 3, 5000, 0), ([16, 512, 16], 1, 20000, 0),
                                                     ([64, 64, 256], 1, 100000, 1), ([64, 64, 256], 2, 60000, 1)])
def test_nothing_past_the_result(lib, dims, members, rows, fused):
    from mfree_iwf_gb300.surrogate import Mlp
    mlp = Mlp(dims, members=members, max_batch=512, seed=1)
    mlp.set_option("fused", fused)
    x = np.random.default_rng(rows).uniform(-1, 1, size=(rows, dims[0])).astype(np.float32)
    want = mlp.predict(x)
    page = os.sysconf("SC_PAGESIZE")
    size = want.nbytes
    whole = (size + page - 1) // page * page  # (the result's own last page is written anyway)
    behind = (rows * dims[-1] * 4 + page - 1) // page * page
    mem = mmap.mmap(-1, whole + behind)
    mem.madvise(mmap.MADV_NOHUGEPAGE)  # (a huge page would hold both the result and what follows it)
    keep = ctypes.c_char.from_buffer(mem)
    addr = ctypes.addressof(keep)
    fp = ctypes.POINTER(ctypes.c_float)
    mlp._check(mlp._lib.mf_mlp_predict(mlp._h, x.ctypes.data_as(fp), rows, ctypes.cast(addr, fp)), "mf_mlp_predict")
    got = np.frombuffer(mem, np.float32, want.size).reshape(want.shape).copy()
    past = resident_pages(addr + whole, behind, page)
    mlp.close()
    np.testing.assert_array_equal(got, want)
    assert past == 0
