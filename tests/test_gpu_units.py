"""Steps in mass units apart by a power of two: densities, masses, moduli and stresses scale
exactly, positions and velocities do not change.  Stresses whose squares overflow or underflow
the format, and densities whose cubes do, are part of the range."""
import numpy as np
import pytest

from mfree_iwf_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


def moved(precision, k, stress, speed, method=S.METHOD_UL):
    import mfree_iwf_gb300 as M
    sc = S.c1_rings(dx=4e-3, method=method)
    a, u = sc.bodies[0].arrays, 2.0 ** k
    a["vx"] = speed * np.sin(200.0 * a["y"])
    a["vy"] = speed * np.cos(150.0 * a["x"])
    for f, w in (("Sxx", 90.0), ("Sxy", 70.0), ("Syy", 50.0)):
        a[f] = u * stress * np.sin(w * a["x"] + 60.0 * a["y"])
    for f in ("m", "rho"):
        a[f] = u * a[f]
    sc.E *= u
    sc.rho0 *= u
    sim = M.from_scenario(sc, precision=precision)
    sim.step(3)
    out = sim.get_state(0)
    sim.close()
    for f in ("rho", "Sxx", "Sxy", "Syy"):
        out[f] = out[f] / u
    return out


# the mixed form: every FP32 operation scales exactly.  FP64: reciprocals far from 1 take the
# plain division, which may differ by an ulp from the seeded step; 1e-9 is the form's bound
@pytest.mark.parametrize("precision,k,stress,speed,tol", [
    ("mixed", 50, 1e6, 2.0, 0.0), ("mixed", -50, 1e-2, 1e-6, 0.0),
    ("fp64", 490, 1e8, 2.0, 1e-9), ("fp64_strict", 490, 1e8, 2.0, 1e-9)])
def test_mass_units(lib, precision, k, stress, speed, tol):
    want, got = moved(precision, 0, stress, speed), moved(precision, k, stress, speed)
    for f in want:
        assert np.linalg.norm(got[f] - want[f]) <= tol * np.linalg.norm(want[f]), f


# the run-walk passes of the mixed form, with viscosity
@pytest.mark.parametrize("k", [50, -60])
def test_mass_units_total_lagrangian(lib, k):
    want, got = (moved("mixed", q, 1e4, 2.0, S.METHOD_TL) for q in (0, k))
    for f in want:
        np.testing.assert_array_equal(got[f], want[f], err_msg=f)
