"""The site kernel where it reads mesh rows by 16 bytes (more than 40,000 sites, rows of a
multiple of 16 bytes; order 5 and the ik forms), and on rows that are not: a box repeated
four times along each axis on an as much finer mesh has the forces of the single box.
Bounds as for the other sizes: FP64 1e-10; mixed 1e-5 RMS."""
import numpy as np
import pytest

from conftest import rel_max, rel_rms
from molmodel_b200 import ElecLJ, water_box

from test_gpu_sites import Repeated

pytestmark = pytest.mark.gpu


# rows of 32 points, and of 36 with a start at each of a word's places; ik wants an even number
@pytest.mark.parametrize("mesh", [8, 9])
@pytest.mark.parametrize("order,ik", [(5, False), (4, True), (5, True), (6, True), (7, True)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_rows_by_16_bytes(mesh, order, ik, precision):
    wb = water_box(6, seed=order)
    mesh = mesh + 1 if ik and mesh % 2 else mesh
    out = []
    for r in (1, 4):
        s = Repeated(wb, r)
        pot = ElecLJ(precision=precision, rspace_cutoff=6.0, ewald_screening=0.35, neighbor_list_width=1.0,
                     use_p3m=True, p3m_grid_spacing=wb.box / mesh, p3m_assignment_order=order,
                     p3m_ik_differentiate=ik).init(s)
        out.append(pot.compute(s.positions))
        assert pot.settings()["mesh"] == (r * mesh,) * 3 and (r == 1 or s.nsite > 40000)
        pot.close()
    want = np.tile(out[0]["f"], (64, 1))
    if precision == "fp64":
        assert rel_max(out[1]["f"], want) < 1e-10
    else:
        assert rel_rms(out[1]["f"], want) < 1e-5
    tol = 1e-10 if precision == "fp64" else 1e-5
    for k in ("elec", "lj"):
        assert abs(out[1][k] - 64 * out[0][k]) < tol * 64 * abs(out[0]["elec"]), k
