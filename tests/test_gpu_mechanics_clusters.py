"""The force assembly with a cell on one or several CTAs of a cluster: which of
the two kernels and how many CTAs a cell follows from the form, the cell's size
and how many cells there are, so the cases below cover one to sixteen CTAs, cells
of fewer vertices than one warp a CTA, and types run side by side.

Tolerances: FP64 1e-12 of the oracle (the stage tolerance: reordered sums);
FP32 forces of the same cell on other numbers of CTAs 1e-6 (the volume's FP64 sum
is ordered by CTA, so the volume force may round to the next float, 6e-8);
whole runs 1e-10 (FP64) and 1e-4 (FP32) of the oracle, the run tolerances."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _mods():
    from hemocell_gb300 import _lib as L
    from hemocell_gb300 import cases as C
    from oracle import oracle as orc
    return L, C, orc


def _deformed(C, t, seed=3):
    xyz = C.place_cells(t.mesh, np.array([[23.5, 23.5, 23.5]]), np.array([[0.3, 0.2, 0.1]]))
    rng = np.random.default_rng(seed)
    return (xyz - 23.5) * np.exp([0.02, -0.01, -0.01]) + 23.5 + 0.01 * rng.standard_normal(xyz.shape)


@pytest.mark.parametrize("variant", [0, 2])
@pytest.mark.parametrize("kind,n", [("rbc42", 1), ("rbc42", 45), ("rbc42", 120), ("rbc162", 30), ("rbc642", 1),
                                    ("rbc642", 80), ("plt162", 7), ("wbc642", 2), ("wbc2562", 1), ("wbc2562", 12)])
def test_forces_on_any_number_of_ctas(built, kind, n, variant):
    L, C, orc = _mods()
    t = {"rbc42": lambda: C.rbc_type(80), "rbc162": lambda: C.rbc_type(320), "rbc642": lambda: C.rbc_type(600),
         "plt162": lambda: C.plt_type(320), "wbc642": lambda: C.wbc_type(1280), "wbc2562": lambda: C.wbc_type(5120)}[kind]()
    xyz = _deformed(C, t)
    one = {}
    for form, count in ((0, n), (1, n), (1, 1)):
        case = C.Case("c", (48, 48, 48), (1, 1, 1), types=[t], cells=[(0, xyz)] * count)
        hc = case.build(form=form)
        tt = hc.tuning()
        tt[6] = variant
        hc.set_tuning(tt)
        v = 1e-3 * np.random.default_rng(7).standard_normal(xyz.shape)
        hc.write_vertices(None, np.tile(v, (count, 1)), None)
        hc.stage(5)
        f = hc.read_vertices()[2].reshape(count, -1, 3)
        assert hc.device_status() == 0
        hc.close()
        assert np.all(f == f[0])            # every copy of the cell, the same bits
        one[form, count] = f[0]
    o = orc.apply_case(C.Case("c", (48, 48, 48), (1, 1, 1), types=[t], cells=[(0, xyz)]))
    o.write_vertices(None, v, None)
    o.stage("mechanics", forced=1)
    assert rel_l2(one[0, n], o.read_vertices()[2]) < 1e-12
    assert rel_l2(one[1, n], one[1, 1]) < 1e-6


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("launch", [0, 1])
def test_types_side_by_side(built, form, launch):
    """All three models in one box, several cells of each, over steps with graph
    replay and a state change in between, against the oracle."""
    L, C, orc = _mods()
    types = [C.rbc_type(320), C.plt_type(80, radius_m=1.0e-6, aspect=0.4), C.wbc_type(320)]
    rng = np.random.default_rng(2)
    cells = []
    for t, centres in ((0, [(10, 10, 8), (10, 10, 16), (10, 30, 10), (30, 10, 10)]), (1, [(22, 22, 6), (22, 22, 34)]),
                       (2, [(30, 30, 28)])):
        for c in centres:
            cells.append((t, C.place_cells(types[t].mesh, np.array([c], float), rng.uniform(-3, 3, (1, 3)))))
    case = C.Case("three", (40, 40, 40), (1, 1, 1), types=types, cells=cells, body_mode=L.HC_BODY_KOLMOGOROV,
                  body=(1e-5, 0.0, 0.0))
    hc = case.build(form=form, launch=launch)
    o = orc.apply_case(case)
    for n in (7, 12):
        hc.iterate(n)
        o.step(n)
        hc.setExternalVector(L.HC_BODY_KOLMOGOROV, (2e-5, 0.0, 0.0))
        o.set_body_force(L.HC_BODY_KOLMOGOROV, (2e-5, 0.0, 0.0))
    x, v, _ = hc.read_vertices()
    xo, vo, _ = o.read_vertices()
    tol = 1e-10 if form == 0 else 1e-4
    assert rel_l2(x, xo) < tol and rel_l2(v, vo) < tol
    assert rel_l2(hc.read_fluid()[1], o.read_fluid()[1]) < tol
    assert hc.device_status() == 0
    hc.close()
