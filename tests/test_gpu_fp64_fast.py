"""The fast FP64 passes against the CPU oracle where their branches change: with and
without the velocity gradient, viscosity and contact, moving and resting Gauss points,
row counts that do not fill a warp or a block."""
import numpy as np
import pytest

import oracle
from mfree_iwf_gb300 import scenarios as S

pytestmark = pytest.mark.gpu

CASES = [S.tensile_tl(7), S.tensile_tl(21), S.rings_tl_contact(13), S.rings_tl_contact(21), S.tensile_tl_weak(7),
         S.tensile_tl_weak(17), S.rotation_tl_weak(15), S.rotation_tl_fem(15), S.rings_tl_weak_contact(21)]


# 1e-8: the fast FP64 form's bound against the reference (contraction and reciprocals by
# multiplication change the last bits of each term)
@pytest.mark.parametrize("sc", CASES, ids=[c.name for c in CASES])
def test_fast_passes_against_oracle(lib, oracle_bin, sc):
    import mfree_iwf_gb300 as M
    for b in sc.bodies:  # a state in which every pair term is at work
        a = b.arrays
        a["vx"] += 0.3 * np.sin(40.0 * a["y"])
        a["vy"] += 0.3 * np.cos(30.0 * a["x"])
    want = oracle.run(sc, 20).dumps[-1]["bodies"]
    sim = M.from_scenario(sc, precision="fp64")
    sim.step(20)
    got = [sim.get_state(k) for k in range(len(sc.bodies))]
    sim.close()
    for f in ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy"):
        w = np.concatenate([b[f] for b in want])
        e = np.linalg.norm(np.concatenate([b[f] for b in got]) - w)
        assert e <= 1e-8 * np.linalg.norm(w), (f, e)
