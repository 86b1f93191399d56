"""Several cell types in one step, a large cell among small ones and more than a
handful of cells: the types' launches are chained, in batched mode with the advance
and the spread in them and inside a graph, against the oracle.  Tolerances as for
whole runs: 1e-10 (FP64) and 1e-4 (FP32)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("launch", [0, 1])
@pytest.mark.parametrize("kind", ["large", "many"])
def test_chained_types(built, form, launch, kind):
    from hemocell_gb300 import _lib as L
    from hemocell_gb300 import cases as C
    from oracle import oracle as orc
    large = kind == "large"
    types = [C.rbc_type(600 if large else 80), C.plt_type(80, radius_m=1.0e-6, aspect=0.4), C.wbc_type(320)]
    rng = np.random.default_rng(2)
    centres = [(t, c) for t, c in ((0, (10, 10, 8)), (0, (10, 10, 18)), (1, (22, 22, 6)), (1, (22, 22, 34)),
                                   (2, (30, 30, 20)))]
    if not large:
        centres += [(1, (4.0 + 6 * i, 36.0, 4.0 + 6 * j)) for i in range(6) for j in range(3)]
    cells = [(t, C.place_cells(types[t].mesh, np.array([c], float), rng.uniform(-3, 3, (1, 3)))) for t, c in centres]
    case = C.Case("chain", (44, 44, 40), (1, 1, 1), types=types, cells=cells, body_mode=L.HC_BODY_KOLMOGOROV,
                  body=(1e-5, 0.0, 0.0))
    hc = case.build(form=form, launch=launch)
    assert hc.tuning()[6] == 2 and (len(cells) > 16 or max(t.mesh.nv for t in types) > 256)
    o = orc.apply_case(case)
    for n in (7, 1, 12):
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
