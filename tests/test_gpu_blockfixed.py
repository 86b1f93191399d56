"""The FP64 collision and node velocity at nodes that the block fixed-point code
refuses (fast, dense or not finite) next to ones that it takes, and at scales far
below and above the usual, in every collide-stream kernel and node-velocity form,
against the oracle.  Tolerance 1e-12, the stage tolerance."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

W = np.array([1 / 3] + [1 / 18] * 3 + [1 / 36] * 6 + [1 / 18] * 3 + [1 / 36] * 6)
FORMS = [(128, 1, 0x101), (64, 2, 0x000), (32, 4, 0x200), (0, 2, 0x300), (16, 8, 0x1300)]


def _box(C, form=0):
    n = (21, 17, 15)
    flags, walls = C.shear_walls(n, 4000.0)
    t = C.rbc_type(80)
    xyz = C.place_cells(t.mesh, np.array([[10.0, 8.0, 7.0]]), np.array([[0.3, -0.2, 0.1]]))
    return C.Case("fixed", n, (1, 1, 0), tau=0.8, flags=flags, walls=walls, types=[t], cells=[(0, xyz)])


@pytest.mark.parametrize("bx,by,t7", FORMS)
@pytest.mark.parametrize("kind", ["mixed", "small", "rest", "not_finite"])
def test_refused_nodes(built, bx, by, t7, kind):
    from hemocell_gb300 import cases as C
    from oracle import oracle as orc
    case = _box(C)
    hc = case.build()
    t = hc.tuning()
    t[0], t[1], t[7] = bx, by, t7
    hc.set_tuning(t)
    o = orc.apply_case(case)
    rng = np.random.default_rng(17)
    amp = {"mixed": 1e-2, "small": 1e-9, "rest": 0.0, "not_finite": 1e-2}[kind]
    d = W[:, None] * amp * rng.standard_normal((19, case.N))
    F = 1e-3 * amp * rng.standard_normal((3, case.N))
    if kind in ("mixed", "not_finite"):
        # a third of the nodes out of bounds, every one well conditioned (rho
        # >= 0.3): |u| up to one at rho near one, and rho of 0.3 to 0.45 or 2 to 3
        fast = rng.random(case.N) < 0.2
        a = 1.5 * W[1:10, None] * rng.uniform(-1, 1, (9, int(fast.sum())))
        d[1:10, fast] += a
        d[10:, fast] -= a
        dense = rng.random(case.N) < 0.15
        rho = np.where(rng.random(int(dense.sum())) < 0.5, rng.uniform(0.3, 0.45, int(dense.sum())),
                       rng.uniform(2.0, 3.0, int(dense.sum())))
        d[:, dense] = W[:, None] * (rho - 1.0) + 0.1 * d[:, dense]
        F[:, rng.random(case.N) < 0.1] *= 1e4
    if kind == "not_finite":
        d[3, 700] = np.nan
        d[11, 2400] = np.inf
        F[1, 3100] = np.nan
    f = W[:, None] + d
    for s in (hc, o):
        s.write_populations(f)
        s.write_force_field(F)
    hc.stage(1)
    o.stage("collide_stream")
    hc.stage(2)
    o.stage("interpolate")
    fluid = case.flags_array() == 0
    a, b = hc.read_populations()[:, fluid] - W[:, None], o.read_populations()[:, fluid] - W[:, None]
    va, vb = hc.read_vertices()[1], o.read_vertices()[1]
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    ok = np.isfinite(b)
    assert ok.sum() > 0.9 * ok.size
    if kind == "rest":
        assert np.abs(a - b).max() < 1e-15 and np.abs(va - vb).max() < 1e-15
    else:
        # the unshifted populations carry 1e-16 of their weights
        assert rel_l2(a[ok], b[ok]) < 1e-12 + (1e-16 / amp if kind == "small" else 0.0)
        both = np.isfinite(vb)
        assert np.array_equal(np.isfinite(va), both)
        assert rel_l2(va[both], vb[both]) < 1e-12 + (1e-16 / amp if kind == "small" else 0.0)
    hc.close()
