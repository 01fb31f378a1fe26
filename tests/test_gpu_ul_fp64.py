"""The FP64 updated-Lagrangian pair pass (four lanes a row, FP32 candidate test) against
the CPU oracle where its branches change: few and many neighbours (a row's list of pairs
is worked off when it fills), positions too far from the origin for the FP32 test, and
neighbour counts on lattices whose pairs lie exactly on the search radius."""
import numpy as np
import pytest

import oracle
from mfree_iwf_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


def moving_rings(hdx, shift=0.0):
    sc = S.c1_rings(dx=4e-3, hdx=hdx, nbh_eps=1e-6)
    a = sc.bodies[0].arrays
    a["vx"] += 2.0 * np.sin(200.0 * a["y"])
    a["vy"] += 2.0 * np.cos(150.0 * a["x"])
    for f in ("Sxx", "Sxy", "Syy"):
        a[f] += 1e4 * np.sin(90.0 * a["x"] + 70.0 * a["y"])
    a["x"] += shift
    return sc


# 1e-9: the form's bound against the reference (summation order, last bits of atan2)
@pytest.mark.parametrize("precision", ["fp64_strict", "fp64"])
@pytest.mark.parametrize("hdx,shift", [(1.3, 0.0), (1.7, 0.0), (2.7, 0.0), (1.3, 2e6)])
def test_pair_pass_against_oracle(lib, oracle_bin, precision, hdx, shift):
    import mfree_iwf_gb300 as M
    sc = moving_rings(hdx, shift)
    want = oracle.run(sc, 5).dumps[-1]["bodies"][0]
    sim = M.from_scenario(sc, precision=precision)
    sim.step(5)
    got = sim.get_state(0)
    sim.close()
    for f in ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy"):
        e = np.linalg.norm(got[f] - want[f]) / np.linalg.norm(want[f])
        assert e < 1e-9, (f, e)


@pytest.mark.parametrize("hdx", [1.0, 1.3, 2.0])
def test_capacity_is_the_exact_count(lib, hdx):
    import mfree_iwf_gb300 as M
    sc = moving_rings(hdx)
    sc.nbh_eps = 0.0  # with h a multiple of dx / 2 some pairs lie on 2h exactly
    sc.dt = 1e-300    # the four stages see the same positions, hence the same counts
    sim = M.from_scenario(sc, precision="fp64_strict")
    most = int(sim.neighbor_counts(0).max())
    sim.close()
    for cap, fails in ((most + 1, False), (most, True)):
        sim = M.from_scenario(sc, precision="fp64_strict", max_nbh=cap)
        if fails:
            with pytest.raises(M.MfError) as e:
                sim.step(1)
            assert e.value.name == "MF_ERR_NBH_OVERFLOW"
        else:
            sim.step(1)
        sim.close()
