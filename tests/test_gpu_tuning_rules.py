"""hc_set_tuning with what hc_get_tuning returned changes nothing: launch shapes
that the rules chose stay the rules', and follow cells that are added later."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("launch", [0, 1])
def test_round_trip_keeps_the_rules(built, form, launch):
    from hemocell_gb300 import cases as C
    t = C.rbc_type(600)
    rng = np.random.default_rng(4)
    centres = np.array([[6.0 + 9.0 * i, 6.0 + 9.0 * j, 6.0 + 9.0 * k] for i in range(3) for j in range(3)
                        for k in range(2)])
    xyz = C.place_cells(t.mesh, centres, rng.uniform(-3, 3, (len(centres), 3)))
    nv = t.mesh.nv
    seen = []
    for trip in (False, True):
        hc = C.Case("r", (32, 32, 32), (1, 1, 1), types=[t]).build(form=form, launch=launch)
        shapes = [hc.tuning()]
        for first, last in ((0, 1), (1, 18)):
            if trip:
                hc.set_tuning(hc.tuning())
            hc.add_cells_xyz(0, xyz[first * nv:last * nv])
            shapes.append(hc.tuning())
            hc.iterate(2)
        # a caller's own choice stays
        own = hc.tuning()
        own[2] = 256
        hc.set_tuning(own)
        hc.set_flags(np.zeros(32 ** 3, np.uint8))
        assert hc.tuning() == own
        assert hc.device_status() == 0
        hc.close()
        seen.append(shapes)
    assert seen[0] == seen[1]


def test_the_shapes_in_use_are_the_ones_reported(built):
    """A handful of small FP32 cells is assembled vertex by vertex (variant 0),
    which hc_get_tuning says; a large cell among them changes that."""
    from hemocell_gb300 import cases as C
    small, large = C.rbc_type(320), C.rbc_type(600)
    hc = C.Case("s", (32, 32, 32), (1, 1, 1), types=[small, large]).build(form=1, launch=1)
    hc.add_cells_xyz(0, C.place_cells(small.mesh, np.array([[9.0, 9.0, 9.0]]), np.zeros((1, 3))))
    assert hc.tuning()[6] == 0
    hc.add_cells_xyz(1, C.place_cells(large.mesh, np.array([[22.0, 22.0, 22.0]]), np.zeros((1, 3))))
    assert hc.tuning()[6] == 2
    hc.iterate(3)
    assert hc.device_status() == 0
    hc.close()
