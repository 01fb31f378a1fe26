"""The training step's kernels at the edges of their 64x64 tiles: batches and widths of one
tile, one row more or less, several tiles and a ragged last one, against the FP64 network
oracle with BF16 rounding at the same points."""
import numpy as np
import pytest

from oracle import mlp_ref as R

pytestmark = pytest.mark.gpu


# 5e-3: the bound of the other gradient checks (only the FP32 accumulation differs)
@pytest.mark.parametrize("dims,members", [([3, 20, 2], 2), ([6, 64, 80, 66], 1), ([17, 144, 256, 33, 5], 3)])
@pytest.mark.parametrize("rows", [1, 63, 64, 65, 200])
def test_gradients_at_tile_edges(lib, dims, members, rows):
    from mfree_iwf_gb300.surrogate import Mlp
    m = Mlp(dims, members=members, max_batch=200, seed=11)
    rng = np.random.default_rng(rows)
    for stale in (200, rows):  # the second batch leaves rows of the first behind it
        x = rng.uniform(-1, 1, (members, stale, dims[0])).astype(np.float32)
        y = rng.normal(size=(members, stale, dims[-1])).astype(np.float32)
        g, loss = m.gradients(x, y)
    for z in range(members):
        want, le = R.gradients(m.get_params(z).astype(np.float64), dims, x[z], y[z], emulate=True)
        assert np.linalg.norm(g[z] - want) < 5e-3 * np.linalg.norm(want), z
        assert abs(loss[z] - le) <= 1e-3 * le
    m.close()


def test_train_continues_across_calls(lib):
    """Two calls of five steps draw the batches and count the steps of one call of ten (at
    a constant learning rate, where the schedule does not depend on the call's length)."""
    from mfree_iwf_gb300.surrogate import Mlp
    rng = np.random.default_rng(2)
    x = rng.uniform(-1, 1, (300, 6)).astype(np.float32)
    y = rng.normal(size=(300, 4)).astype(np.float32)
    out = []
    for calls in ((10,), (5, 5)):
        m = Mlp([6, 64, 4], members=2, max_batch=48, seed=5)
        m.set_data(x, y)
        loss = np.concatenate([m.train(n, 1e-3, 1e-3) for n in calls])
        out.append((loss, m.get_params(0), m.get_params(1)))
        m.close()
    np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-6)  # (the loss adds its blocks in any order)
    for a, b in zip(out[0][1:], out[1][1:]):
        np.testing.assert_array_equal(a, b)
