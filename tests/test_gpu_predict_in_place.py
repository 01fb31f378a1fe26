"""Inference between host arrays with the outputs written over the inputs (one member, outputs
no wider than the inputs): the results of separate arrays."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("dims", [[66, 32, 66], [64, 256, 5]])
@pytest.mark.parametrize("rows", [3, 16, 17, 40000])
def test_outputs_over_inputs(lib, pinned, dims, rows):
    import torch
    from mfree_iwf_gb300.surrogate import Mlp
    mlp = Mlp(dims, members=1, max_batch=16, seed=4)
    x = np.random.default_rng(rows).uniform(-1, 1, size=(rows, dims[0])).astype(np.float32)
    want = mlp.predict(x)[0]
    buf = torch.empty(x.size, dtype=torch.float32, pin_memory=pinned).numpy()
    p = buf.ctypes.data_as(ctypes.POINTER(ctypes.c_float))
    for fused in (1, 0):
        mlp.set_option("fused", fused)
        buf[:] = x.ravel()
        mlp._check(mlp._lib.mf_mlp_predict(mlp._h, p, rows, p), "mf_mlp_predict")
        got = buf[:rows * dims[-1]].reshape(rows, dims[-1])
        if fused:
            np.testing.assert_array_equal(got, want)
        else:  # the per-layer products in another order of accumulation: the inference checks' bound
            assert np.linalg.norm(got - want) < 3e-3 * np.linalg.norm(want)
    mlp.close()
