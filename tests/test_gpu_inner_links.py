"""The inner links (cytoskeleton and rigid core) of the FP32 form in the staged and
in the vertex-centric force assembly: with every other material constant zero both
take the same operations in the same order, so the forces are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("triangles,count", [(320, 1), (1280, 3), (1280, 90)])
def test_inner_links_same_bits(built, triangles, count):
    from hemocell_gb300 import cases as C
    t = C.wbc_type(triangles)
    m = t.material
    t.material = type(m)(kLink=0.0, kBend=0.0, kVolume=0.0, kArea=0.0, eta_m=0.0, kInnerRigid=m.kInnerRigid,
                         kCytoskeleton=m.kCytoskeleton, coreRadius=3.8e-6, radius=m.radius)
    xyz = C.place_cells(t.mesh, np.array([[24.0, 24.0, 24.0]]), np.array([[0.3, 0.2, 0.1]]))
    rng = np.random.default_rng(3)
    xyz = (xyz - 24.0) * 0.97 + 24.0 + 0.02 * rng.standard_normal(xyz.shape)
    f = []
    for variant in (0, 2):
        hc = C.Case("i", (48, 48, 48), (1, 1, 1), types=[t], cells=[(0, xyz)] * count).build(form=1)
        tt = hc.tuning()
        tt[6], tt[2] = variant, 256
        hc.set_tuning(tt)
        hc.stage(5)
        f.append(hc.read_vertices()[2])
        assert hc.device_status() == 0
        hc.close()
    assert np.count_nonzero(f[0]) > 0.9 * f[0].size
    assert np.array_equal(f[0], f[1])
