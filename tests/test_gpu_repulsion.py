"""Repulsion where cells overlap: nodes holding vertices of one and of several
cells, up to several a node, pairs of one vertex spread over more than one round
of a warp, vertex counts that do not fill a warp, on periodic axes (images) and
next to walls, with either term alone and both, against the oracle.  Tolerances:
FP64 1e-12 (the stage tolerance), FP32 1e-5 (as the other repulsion stage test)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("terms", ["cells", "walls", "both"])
@pytest.mark.parametrize("ncells", [1, 2, 3])
def test_overlapping_cells(built, form, terms, ncells):
    from hemocell_gb300 import cases as C
    from oracle import oracle as orc
    n = (19, 21, 16)
    flags, walls = C.shear_walls(n, 1000.0)
    types = [C.rbc_type(320), C.plt_type(80, radius_m=1.0e-6, aspect=0.4)]
    rng = np.random.default_rng(31)
    cells = []
    for k in range(ncells):
        t = k % 2
        # across the periodic edges in x and y, the first close to the lower wall
        c = np.array([[0.4 + 0.7 * k, 20.2 + 0.3 * k, 3.9 + 2.0 * k]])
        a = np.array([[-np.pi / 2, 0.0, 0.0]]) + 0.1 * rng.standard_normal((1, 3))
        cells.append((t, C.place_cells(types[t].mesh, c, a)))
    case = C.Case("overlap", n, (1, 1, 0), flags=flags, walls=walls, types=types, cells=cells)
    hc = case.build(form=form)
    o = orc.apply_case(case)
    if terms != "walls":
        hc._check(hc._lib.hc_set_repulsion(hc._h, 1e-4, 1.7, 1))
        o.set_repulsion(1e-4, 1.7, 1)
    if terms != "cells":
        hc._check(hc._lib.hc_set_boundary_repulsion(hc._h, 5e-5, 1.6, 1))
        o.set_boundary_repulsion(5e-5, 1.6, 1)
    hc.stage(7)
    o.stage("repulsion")
    f, fo = hc.read_repulsion(), o.read_repulsion()
    assert hc.device_status() == 0
    if terms != "walls" and ncells > 1 or terms != "cells":
        assert np.abs(fo).max() > 0
    assert rel_l2(f, fo) < (1e-12 if form == 0 else 1e-5)
    g = hc.read_repulsion()
    hc.stage(7)
    assert np.array_equal(g, hc.read_repulsion())   # no order of arrival in the sums
    hc.close()
