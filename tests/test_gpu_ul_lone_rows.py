"""Updated-Lagrangian rows without neighbours: a state that is not finite, or an h of zero, ends
the step with the error that it ends with among neighbours; a sound lone particle flies on."""
import numpy as np
import pytest

from mfree_iwf_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64_strict", "fp64", "mixed"])
@pytest.mark.parametrize("field,value", [("vx", 1.0), ("Sxx", np.nan), ("Sxy", np.nan), ("Syy", np.inf), ("h", 0.0)])
def test_lone_row(lib, precision, field, value):
    import mfree_iwf_gb300 as M
    sc = S.c1_rings(dx=1e-3)
    a = sc.bodies[0].arrays
    a["x"][7], a["y"][7] = 0.045, 0.0  # the middle of a ring, beyond every reach
    assert np.sort(np.hypot(a["x"] - a["x"][7], a["y"] - a["y"][7]))[1] > 4 * a["h"][7]
    a["vx"][:] = 1.0
    a["vy"][:] = 0.0
    x0 = a["x"][7]
    a[field][7] = value
    sim = M.from_scenario(sc, precision=precision)
    if np.isfinite(value) and value:
        sim.step(2)
        got = sim.get_state(0)
        assert abs(got["x"][7] - x0 - 2 * sc.dt) < 1e-15 and got["vx"][7] == 1.0 and got["Sxx"][7] == 0.0
    else:
        with pytest.raises(M.MfError) as e:
            sim.step(2)
        assert e.value.name == "MF_ERR_NONFINITE"
    sim.close()
