"""The weak form's mixed Gauss-point pass runs at one of two register budgets, by how many
waves of blocks its Gauss points make: the same bits at both."""
import numpy as np
import pytest

from mfree_iwf_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [7, 31])
def test_plate_in_a_batch_equals_plate_alone(lib, copies):
    """7 plates make one wave of blocks of 128 Gauss points on 152 SMs either way, 31 one
    wave of 16 blocks an SM and two of 12."""
    import mfree_iwf_gb300 as M
    sc = S.c3_plate(dx=1e-3, seed=3)
    sc.bodies = sc.bodies[:1]
    one = S.c3_plate(dx=1e-3, seed=3)
    one.bodies = one.bodies[:1]
    sc.bodies = sc.bodies * copies
    out = []
    for s in (one, sc):
        sim = M.from_scenario(s, precision="mixed")
        sim.step(3)
        out.append(sim.get_state(len(s.bodies) - 1))
        sim.close()
    for f in ("x", "y", "vx", "vy"):
        np.testing.assert_array_equal(out[0][f], out[1][f], err_msg=f)
