"""A velocity that is not a number: the fast FP64 passes' sign tests take it as the reference's
comparisons do (not approaching), so after a step the same rows as in the parity form are
not finite."""
import numpy as np
import pytest

from mfree_iwf_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("method", [S.METHOD_UL, S.METHOD_TL])
def test_rows_not_finite_after_a_step(lib, method, sign):
    import mfree_iwf_gb300 as M
    hit = []
    for precision in ("fp64_strict", "fp64"):
        sc = S.c1_rings(dx=2e-3, method=method)
        sim = M.from_scenario(sc, precision=precision)
        sim.step(1)
        s = sim.get_state(0)
        s["vy"][40] = np.copysign(np.nan, sign)
        sim.set_state(0, s)
        with pytest.raises(M.MfError) as e:
            sim.step(1)
        assert e.value.name == "MF_ERR_NONFINITE"
        got = sim.get_state(0)
        sim.close()
        hit.append({f: ~np.isfinite(got[f]) for f in ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy")})
    for f in hit[0]:
        np.testing.assert_array_equal(hit[0][f], hit[1][f], err_msg=f)
    assert hit[0]["x"].any()
    if method == S.METHOD_TL:  # (the updated-Lagrangian grid of such positions is one cell: every row is reached)
        assert not hit[0]["x"].all()
