"""The updated-Lagrangian pair passes against the CPU oracle where their branches change:
few and many neighbours (a row's list of pairs is worked off when it fills), positions too
far from the origin for the FP32 candidate test, neighbour counts on lattices whose pairs
lie exactly on the search radius, pipelines that leave actions out."""
import numpy as np
import pytest

import oracle
from mfree_iwf_gb300 import actions as A
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


DROP = {"none": [], "xsph": [A.CORRECTORS_XSPH], "viscosity": [A.CORRECTORS_MGHN_ARTIFICIAL_VISCOSITY],
        "artificial stress": [A.CORRECTORS_MGHN_ARTIFICIAL_STRESS], "weights": [A.RIEMANN_UPDATE_INTEGRATION_WEIGHTS],
        "momentum": [A.CONTMECH_MOMENTUM_UL], "stress": [A.DERIVE_STRESS_MONAGHAN, A.CONTMECH_MOMENTUM_UL],
        "rates": [A.DERIVE_VELOCITY, A.MATERIAL_STRESS_RATE_JAUMANN, A.CONTMECH_CONTINUITY]}


# FP64: as above.  Mixed: a pair sum of ~20 FP32 terms of ~10 roundings each is good to
# ~1e-6 of its terms; five steps move the state by less than itself
@pytest.mark.parametrize("precision,tol", [("fp64_strict", 1e-9), ("fp64", 1e-9), ("mixed", 1e-5)])
@pytest.mark.parametrize("drop", list(DROP))
def test_partial_pipelines_against_oracle(lib, oracle_bin, precision, tol, drop):
    """Pipelines that leave actions out: the pair pass skips their terms."""
    import mfree_iwf_gb300 as M
    sc = moving_rings(1.3)
    sc.actions = [a for a in sc.actions if a not in DROP[drop]]
    want = oracle.run(sc, 5).dumps[-1]["bodies"][0]
    sim = M.from_scenario(sc, precision=precision)
    sim.step(5)
    got = sim.get_state(0)
    sim.close()
    for f in ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy"):
        e = np.linalg.norm(got[f] - want[f]) / np.linalg.norm(want[f])
        assert e < tol, (f, e)


@pytest.mark.parametrize("hdx", [1.3, 1.7, 2.7])
def test_mixed_pair_pass_close_to_oracle(lib, oracle_bin, hdx):
    """Few and many candidates per stencil column (a mask holds 32)."""
    import mfree_iwf_gb300 as M
    sc = moving_rings(hdx)
    want = oracle.run(sc, 5).dumps[-1]["bodies"][0]
    sim = M.from_scenario(sc, precision="mixed")
    sim.step(5)
    got = sim.get_state(0)
    sim.close()
    for f in ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy"):
        e = np.linalg.norm(got[f] - want[f]) / np.linalg.norm(want[f])
        assert e < 1e-5, (f, e)


def test_large_batch_equals_instances_alone(lib):
    """From 2^19 rows on the mixed pair pass runs at another register budget: the same
    bits as an instance alone."""
    import mfree_iwf_gb300 as M
    ens = S.c4_ensemble(30)
    assert ens.n_total >= 1 << 19
    for b in ens.bodies:
        b.arrays["vx"] += 0.5 * np.sin(200.0 * b.arrays["y"])
    sim = M.from_scenario(ens, precision="mixed")
    sim.step(3)
    for k in (0, 29):
        b = ens.bodies[k]
        one = S.Scenario(method=ens.method, bodies=[b], actions=ens.actions, dt=b.params["dt"], nu=b.params["nu"],
                         E=b.params["E"], rho0=b.params["rho0"], wdeltap=b.params["wdeltap"], corr_exp=ens.corr_exp,
                         mghn_eps=ens.mghn_eps, alpha=ens.alpha, beta=ens.beta, eta=ens.eta, xsph_eps=ens.xsph_eps,
                         nbh_eps=ens.nbh_eps)
        alone = M.from_scenario(one, precision="mixed")
        alone.step(3)
        got, want = sim.get_state(k), alone.get_state(0)
        alone.close()
        for f in ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy"):
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)
    sim.close()


@pytest.mark.parametrize("precision", ["fp64_strict", "fp64", "mixed"])
@pytest.mark.parametrize("dx,instances", [(1e-3, 1), (4e-3, 1), (None, 5), (1e-3, 161)])
def test_small_body_grid_equals_general(lib, precision, dx, instances):
    """The grid of small bodies (a block each) against the general kernels, which a context
    that masks failed bodies always takes: the same cells and order, hence the same bits."""
    import mfree_iwf_gb300 as M
    sc = S.c1_rings(dx=dx) if instances == 1 else S.c4_ensemble(instances, dx_range=(3e-3, 4e-3))
    if instances > 152:  # (a block per SM: bodies up to 4608 rows take this grid too)
        sc.bodies[7] = S.c4_ensemble(1, dx_range=(dx, dx)).bodies[0]
    for b in sc.bodies:
        b.arrays["vx"] += 1.5 * np.sin(200.0 * b.arrays["y"])
        b.arrays["x"][: 3] -= 0.05  # (and a few particles apart from the rest: empty cells)
    out = []
    for general in (0, 1):
        sim = M.from_scenario(sc, precision=precision)
        sim.set_option("mask_failed", general)
        try:
            sim.step(4)
        except M.MfError as e:  # a particle without neighbours counts itself: none expected
            pytest.fail(str(e))
        out.append([sim.get_state(k) for k in range(len(sc.bodies))])
        sim.close()
    for a, b in zip(*out):
        for f in ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy"):
            np.testing.assert_array_equal(a[f], b[f], err_msg=f)


def test_small_body_grid_with_scattered_particles(lib):
    """A body whose cells outnumber its particles (the mixed form allows it up to three a
    particle and context): the counters stand in the cell table itself."""
    import mfree_iwf_gb300 as M
    out = []
    for general in (0, 1):
        sc = S.c4_ensemble(3, dx_range=(2e-3, 4e-3))
        a = sc.bodies[1].arrays
        a["x"][0] -= 1.2  # a particle far off stretches the box to more than two cells a particle
        sim = M.from_scenario(sc, precision="mixed")
        sim.set_option("mask_failed", general)
        sim.step(3)
        out.append([sim.get_state(k) for k in range(3)])
        sim.close()
    for a, b in zip(*out):
        for f in ("x", "y", "vx", "vy", "rho", "Sxx"):
            np.testing.assert_array_equal(a[f], b[f], err_msg=f)


@pytest.mark.parametrize("hdx", [1.0, 1.3, 2.0, 2.7, 3.5])
@pytest.mark.parametrize("drop", ["none", "xsph", "rates"])
def test_row_by_lanes_equals_row_by_thread(lib, hdx, drop):
    """Few rows: eight lanes a row, whose list of neighbours fills and is worked off; a batch
    of the same body with many rows walks a row with one thread: the same bits."""
    import mfree_iwf_gb300 as M
    sc = moving_rings(hdx)
    sc.actions = [a for a in sc.actions if a not in DROP[drop]]
    out = []
    for copies in (1, 60):
        sc.bodies = sc.bodies[:1] * copies
        sim = M.from_scenario(sc, precision="mixed")
        assert (sc.bodies[0].n * copies > 152 * 64) == (copies > 1)
        sim.step(5)
        out.append(sim.get_state(copies - 1))
        sim.close()
    for f in ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy"):
        np.testing.assert_array_equal(out[0][f], out[1][f], err_msg=f)
