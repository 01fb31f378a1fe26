"""The grid of one small body (a single launch, up to 1,024 rows) at the edges of its rule:
the general kernels' cells and order, hence the same bits."""
import numpy as np
import pytest

from mfree_iwf_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


def states(sc, precision, general):
    import mfree_iwf_gb300 as M
    sim = M.from_scenario(sc, precision=precision)
    sim.set_option("mask_failed", general)  # (a context that masks failed bodies takes the general grid)
    sim.step(3)
    n = sim.launch_count()
    out = sim.get_state(0)
    sim.close()
    return out, n


@pytest.mark.parametrize("precision", ["fp64_strict", "fp64", "mixed"])
@pytest.mark.parametrize("rows", [31, 257, 1023, 1024, 1025])
def test_edges_of_the_single_body_grid(lib, precision, rows):
    sc = S.c1_rings(dx=2e-3)
    b = sc.bodies[0]
    assert b.n > 1025
    x, y = b.arrays["x"], b.arrays["y"]
    near = np.argsort((x - x[0]) ** 2 + (y - y[0]) ** 2, kind="stable")[:rows]  # (a piece with fewer cells than rows)
    b.arrays = {f: v[near] for f, v in b.arrays.items()}
    b.arrays["vx"] += 1.5 * np.sin(200.0 * b.arrays["y"])
    (one, n1), (general, n2) = states(sc, precision, 0), states(sc, precision, 1)
    assert (n1 < n2) == (rows <= 1024)
    for f in ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy"):
        np.testing.assert_array_equal(one[f], general[f], err_msg=f)
