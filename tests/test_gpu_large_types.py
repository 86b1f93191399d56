"""The largest cell types that one CTA's shared memory holds: hexagonal tubes of
6 L + 2 vertices with a pole at each end (valence 5 and 6), up to the 4730 vertices
of the FP64 form and the 9272 of the FP32 form that 232,448 bytes take.

Tolerances: FP64 forces 1e-10 of the oracle (the tube is 900 times its radius long,
so the sums of the volume lose 3 digits of the stage tolerance 1e-12 at most);
FP32 0.05: positions relative to the tube's end round to 6e-8 of its length, 1e-4
of an edge, against strains of 0.02, and the area terms double that."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def tube(rings, step=0.15):
    """Rings of six vertices along x, poles at both ends, outward faces."""
    from hemocell_gb300.hemocell import Mesh
    a = np.arange(6) * np.pi / 3
    ring = [np.stack([np.full(6, k * step), step * np.cos(a + k * np.pi / 6), step * np.sin(a + k * np.pi / 6)], 1)
            for k in range(rings)]
    xyz = np.concatenate([[[-0.5 * step, 0, 0]], *ring, [[(rings - 0.5) * step, 0, 0]]])
    tris = []
    for j in range(6):
        j1 = (j + 1) % 6
        tris.append((0, 1 + j1, 1 + j))
        for k in range(rings - 1):
            p, q, r, s = 1 + 6 * k + j, 1 + 6 * k + j1, 7 + 6 * k + j, 7 + 6 * k + j1
            tris += [(p, q, r), (q, s, r)]
        last = 1 + 6 * (rings - 1)
        tris.append((last + j, last + j1, 6 * rings + 1))
    return Mesh(xyz=np.ascontiguousarray(xyz), tris=np.array(tris, np.int32))


@pytest.mark.parametrize("variant", [0, 1, 2])
@pytest.mark.parametrize("form,rings", [(0, 787), (0, 788), (1, 1543), (1, 1544), (1, 1545)])
def test_largest_types(built, form, rings, variant):
    from hemocell_gb300 import cases as C
    from hemocell_gb300 import _lib as L
    from oracle import oracle as orc
    mesh = tube(rings)
    assert mesh.nv == 6 * rings + 2 and mesh.nf == 2 * mesh.nv - 4
    t = C.CellTypeSpec("tube", L.HC_MODEL_RBC_HIGH_ORDER, C.RBC_MATERIAL, mesh)
    rng = np.random.default_rng(5)
    xyz = mesh.xyz * np.exp([0.02, -0.01, -0.01]) + 4.0 + 0.002 * rng.standard_normal(mesh.xyz.shape)
    case = C.Case("tube", (264, 8, 8), (1, 1, 1), types=[t], cells=[(0, xyz)])
    hc = case.build(form=form)
    tt = hc.tuning()
    tt[6] = variant
    hc.set_tuning(tt)
    hc.stage(5)
    f = hc.read_vertices()[2]
    assert hc.device_status() == 0
    hc.close()
    o = orc.apply_case(case)
    o.stage("mechanics", forced=1)
    assert rel_l2(f, o.read_vertices()[2]) < (1e-10 if form == 0 else 0.05)


def test_beyond_the_largest_is_refused(built):
    from hemocell_gb300 import cases as C
    from hemocell_gb300 import _lib as L
    from hemocell_gb300.hemocell import HemoCellError
    for form, rings in ((0, 795), (1, 1560)):
        t = C.CellTypeSpec("tube", L.HC_MODEL_RBC_HIGH_ORDER, C.RBC_MATERIAL, tube(rings))
        with pytest.raises(HemoCellError):
            C.Case("tube", (16, 8, 8), (1, 1, 1), types=[t]).build(form=form)
