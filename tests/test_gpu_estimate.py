"""hc_estimate_device_bytes bounds what a handle holds once every readback has
sized its staging: fully fluid periodic boxes (the largest fluid-node list) with
one cell, several cells and all three models, in both forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("n,kind", [(32, "rbc642"), (64, "rbc642"), (33, "rbc42"), (40, "three"), (64, "wbc2562")])
def test_estimate_bounds_the_handle(built, form, n, kind):
    from hemocell_gb300 import cases as C
    from hemocell_gb300.hemocell import estimate_device_bytes
    types = {"rbc642": lambda: [C.rbc_type(600)], "rbc42": lambda: [C.rbc_type(80)],
             "three": lambda: [C.rbc_type(320), C.plt_type(80), C.wbc_type(320)],
             "wbc2562": lambda: [C.wbc_type(5120)]}[kind]()
    centre = np.full((1, 3), 0.5 * n)
    cells = [(k, C.place_cells(t.mesh, centre, np.zeros((1, 3)))) for k, t in enumerate(types)]
    case = C.Case("e", (n, n, n), (1, 1, 1), types=types, cells=cells)
    hc = case.build(form=form)
    hc.iterate(1)
    hc.read_fluid()
    hc.read_vertices()
    hc.read_bins()
    held = hc.stats().device_bytes
    hc.close()
    assert held <= estimate_device_bytes(case.dims, form, case.nvertices, len(cells))
