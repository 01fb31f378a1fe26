"""The launch counter against the kernels a step is made of (the grid's sort is CUB's and not
counted)."""
import pytest

from mfree_iwf_gb300 import scenarios as S

pytestmark = pytest.mark.gpu


def per_step(sc, precision, options=(), monitor=0, graph=False):
    import mfree_iwf_gb300 as M
    sim = M.from_scenario(sc, precision=precision, graph=graph)
    for k, v in options:
        sim.set_option(k, v)
    if monitor:
        sim.set_monitor(monitor)
    sim.step(1)  # (what the first step alone needs)
    n = sim.launch_count()
    sim.step(3)
    n = sim.launch_count() - n
    sim.close()
    assert n % 3 == 0
    return n // 3


# a stage: grid (general: boxes set, boxes, geometry, keys; of small bodies: 1 launch for one
# body, 2 for several), gather, pair pass; the mixed form builds grid and records once a step
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("precision,one,several,general", [("fp64_strict", 4 * 3, 4 * 4, 4 * 6), ("fp64", 4 * 3, 4 * 4, 4 * 6),
                                                           ("mixed", 1 + 1 + 4, 2 + 1 + 4, 4 + 1 + 4)])
def test_updated_lagrangian(lib, precision, one, several, general, graph):
    small, batch, large = S.c1_rings(dx=4e-3), S.c4_ensemble(3, dx_range=(3e-3, 4e-3)), S.c1_rings(dx=1e-3)
    assert small.n_total <= 1024 < large.n_total and max(b.n for b in batch.bodies) <= 1024
    assert per_step(small, precision, graph=graph) == one
    assert per_step(batch, precision, graph=graph) == several
    assert per_step(large, precision, graph=graph) == general
    assert per_step(batch, precision, [("mask_failed", 1)], graph=graph) == general
    assert per_step(batch, precision, monitor=8, graph=graph) == several + 2


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("precision", ["fp64_strict", "fp64", "mixed"])
def test_contact_adds_two(lib, precision, graph):
    """Boundary and query: the passes A and B of four stages and the clock beside them."""
    sc = S.rings_tl_contact(21)
    assert per_step(sc, precision, graph=graph) == 4 * 2 + 1 + 2


# a stage: two neighbourhoods or the element functions, stress points, particles (mixed: the
# float-float inputs of the neighbourhoods too); smoothing: a neighbourhood and two launches
@pytest.mark.parametrize("precision", ["fp64_strict", "fp64", "mixed"])
def test_weak_updated_lagrangian(lib, precision):
    for sc in (S.tensile_ul_weak(7), S.tensile_ul_fem(7)):
        fem = sc.bodies[0].quads is not None and len(sc.bodies[0].quads) > 0
        ff = 1 if precision == "mixed" and not fem else 0
        want = 4 * ((1 if fem else 2 + ff) + 2) + (1 if any(len(b.bcs) for b in sc.bodies) else 0)
        want += 3 + ff if sc.do_smooth else 0
        assert per_step(sc, precision) == want
