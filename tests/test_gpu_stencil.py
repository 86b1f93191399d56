"""Interpolation and spread with a vertex's stencil shared by two lanes and its
solid nodes read from one byte, where that can go wrong: solid nodes among the
stencils, blocks across a periodic end, blocks that begin beyond a non-periodic
one, last warps of 2 and 10 vertices, both launch modes (the fused spread and
advance, and the single kernels).

Tolerances: the run tolerances of the oracle, 1e-10 (FP64) and 1e-4 (FP32)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("launch", [0, 1])
@pytest.mark.parametrize("triangles,where", [(80, "solid"), (320, "solid"), (600, "solid"), (80, "edge"), (600, "edge")])
def test_stencils_at_walls_and_ends(built, triangles, where, form, launch):
    from hemocell_gb300 import _lib as L
    from hemocell_gb300 import cases as C
    from oracle import oracle as orc
    dims = (26, 24, 24)
    t = C.rbc_type(triangles)
    # across the periodic x end
    xyz = C.place_cells(t.mesh, np.array([[25.4, 11.6, 11.7]]), np.array([[0.4, 0.3, 0.2]]))
    flags = None
    if where == "edge":
        # the lowest vertex a third of a node below the first y node
        xyz[:, 1] -= xyz[:, 1].min() + 0.3
    else:
        rng = np.random.default_rng(4)
        base = np.floor(xyz).astype(int)
        nodes = np.unique(np.concatenate([base + [s >> 2, s >> 1 & 1, s & 1] for s in range(8)]), axis=0)
        # a quarter of the stencil nodes that no vertex comes close to
        gap = np.abs(nodes[:, None, :] - xyz[None]).max(2).min(1)
        nodes = nodes[gap > 0.6]
        nodes = nodes[rng.random(len(nodes)) < 0.25]
        assert len(nodes) > 3
        f = np.zeros(dims[::-1], np.uint8)
        f[nodes[:, 2], nodes[:, 1], nodes[:, 0] % dims[0]] = 1
        flags = f.ravel()
    case = C.Case("stencil", dims, (1, 0, 0), flags=flags, types=[t], cells=[(0, xyz)], body_mode=L.HC_BODY_UNIFORM,
                  body=(1e-5, 0.0, 0.0))
    hc = case.build(form=form, launch=launch)
    o = orc.apply_case(case)
    rng = np.random.default_rng(6)
    force = 1e-4 * rng.standard_normal(xyz.shape)
    hc.write_vertices(None, None, force)
    o.write_vertices(None, None, force)
    hc.iterate(5)
    o.step(5)
    tol = 1e-10 if form == 0 else 1e-4
    x, v, _ = hc.read_vertices()
    xo, vo, _ = o.read_vertices()
    assert rel_l2(x, xo) < tol and rel_l2(v, vo) < tol
    assert rel_l2(hc.read_fluid()[1], o.read_fluid()[1]) < tol
    assert hc.device_status() == 0
    hc.close()
