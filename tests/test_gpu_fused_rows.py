"""Fused inference at the edges of its tiles: 512 rows to a pair of CTAs, in halves of 256, 128
of a half's rows in each CTA; one tile, less and more, several tiles to a pair; outputs in
blocks of 16, handed on before or after the next tile's input (an input as wide as the widest
layer leaves no room before), against the FP64 network oracle with BF16 rounding at the same
points, the rows around the result untouched."""
import ctypes

import numpy as np
import pytest

from oracle import mlp_ref as R

pytestmark = pytest.mark.gpu


def _predict(dims, members, rows):
    import torch
    from mfree_iwf_gb300.surrogate import Mlp
    mlp = Mlp(dims, members=members, max_batch=16, seed=5)
    assert mlp.get_option("fused") == 1
    rng = np.random.default_rng(rows)
    for z in range(members):  # non-zero biases too
        p = mlp.get_params(z)
        mlp.set_params(z, p + rng.normal(scale=0.1, size=p.shape).astype(np.float32))
    x = rng.uniform(-1, 1, size=(rows, dims[0])).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    n = members * rows * dims[-1]
    yd = torch.full((n + 512 * dims[-1],), 7.0, device="cuda", dtype=torch.float32)
    fp = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_float))
    mlp._check(mlp._lib.mf_mlp_predict(mlp._h, fp(xd), rows, fp(yd)), "mf_mlp_predict")
    y = yd.cpu().numpy()
    assert (y[n:] == 7.0).all()
    params = [mlp.get_params(z).astype(np.float64) for z in range(members)]
    mlp.close()
    return x, y[:n].reshape(members, rows, dims[-1]), params


# 3e-3: the bound of the other inference checks (only the FP32 accumulation differs)
@pytest.mark.parametrize("dims", [[6, 256, 256, 66], [256, 48, 16], [64, 64, 33], [5, 16, 1], [130, 256, 256]])
@pytest.mark.parametrize("rows", [1, 127, 129, 256, 257, 511, 512, 513])
def test_rows_at_tile_edges(lib, dims, rows):
    x, y, params = _predict(dims, 3, rows)
    for z in range(3):
        want, _ = R.forward(params[z], dims, x, emulate=True)
        assert np.linalg.norm(y[z] - want) < 3e-3 * np.linalg.norm(want), z


@pytest.mark.parametrize("dims", [[6, 256, 256, 66], [128, 100, 30]])
def test_several_tiles_to_a_pair(lib, dims):
    """300 tiles, more than the pairs of CTAs that a GPU holds at once, the last one ragged."""
    rows = 512 * 99 + 37
    x, y, params = _predict(dims, 3, rows)
    some = np.r_[0:700, rows - 700:rows]
    for z in range(3):
        want, _ = R.forward(params[z], dims, x[some], emulate=True)
        assert np.linalg.norm(y[z][some] - want) < 3e-3 * np.linalg.norm(want), z
        assert np.isfinite(y[z]).all() and (np.abs(y[z]).max(axis=1) > 0).all()


@pytest.mark.parametrize("rows", [8, 17, 8170, 8171, 16343])
def test_host_arrays_in_staged_chunks(lib, rows):
    """Host arrays of fewer rows than max_batch, more, and of one, exactly one and several
    staged chunks (64 MB: 8,171 rows of 5 inputs and 8 x 256 outputs) give the device
    arrays' outputs bit for bit (rows are independent of the chunks); a smaller call after
    a larger one reuses its staging."""
    import torch
    from mfree_iwf_gb300.surrogate import Mlp
    mlp = Mlp([5, 32, 256], members=8, max_batch=16, seed=2)
    x = np.random.default_rng(rows).uniform(-1, 1, size=(rows, 5)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    yd = torch.empty((8, rows, 256), device="cuda", dtype=torch.float32)
    fp = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_float))
    mlp._check(mlp._lib.mf_mlp_predict(mlp._h, fp(xd), rows, fp(yd)), "mf_mlp_predict")
    want = yd.cpu().numpy()
    np.testing.assert_array_equal(mlp.predict(x), want)
    for n in (rows, rows // 2 + 1):
        np.testing.assert_array_equal(mlp.predict(x[:n]), want[:, :n])
    mlp.close()
