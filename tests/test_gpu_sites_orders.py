"""The per-site kernel in both layouts at every assignment order, with and without ik,
on rows of even and odd length: a box repeated twice along each axis (5,184 sites: lanes
per mesh plane) and three times (17,496: a lane per site) on an as much finer mesh has
the forces of the single box.  Bounds as for the larger boxes: FP64 1e-10; mixed 1e-5
RMS."""
import numpy as np
import pytest

from conftest import rel_max, rel_rms
from molmodel_b200 import ElecLJ, water_box

from test_gpu_sites import Repeated

pytestmark = pytest.mark.gpu


# rows of 14 and 21, 16 and 24, 20 and 30 points; ik wants an even number of points
@pytest.mark.parametrize("mesh,ik", [(7, False), (8, True), (10, False), (10, True)])
@pytest.mark.parametrize("order", [2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_both_layouts(mesh, ik, order, precision):
    wb = water_box(6, seed=order)
    out = []
    for r in (1, 2, 3):
        s = Repeated(wb, r)
        pot = ElecLJ(precision=precision, rspace_cutoff=6.0, ewald_screening=0.35, neighbor_list_width=1.0,
                     use_p3m=True, p3m_grid_spacing=wb.box / mesh, p3m_assignment_order=order,
                     p3m_ik_differentiate=ik).init(s)
        out.append(pot.compute(s.positions))
        assert pot.settings()["mesh"] == (r * mesh,) * 3
        pot.close()
    for r, many in zip((2, 3), out[1:]):
        m = r ** 3
        want = np.tile(out[0]["f"], (m, 1))
        if precision == "fp64":
            assert rel_max(many["f"], want) < 1e-10
        else:
            assert rel_rms(many["f"], want) < 1e-5
        tol = 1e-10 if precision == "fp64" else 1e-5
        for k in ("elec", "lj"):
            assert abs(many[k] - m * out[0][k]) < tol * m * abs(out[0]["elec"]), k
