"""The mesh solve's own transforms, at lengths that take every radix as first and as
second factor, odd and even along each axis, unequal along the three, and around the
largest plane the FP64 form's blocks hold, against the oracle's P3M (FP64 form 1e-10;
mixed form 1e-5 RMS, the bound of its reciprocal-space forces)."""
import numpy as np
import pytest

from conftest import rel_max, rel_rms
from molmodel_b200 import ElecLJ, _lib
from oracle.oracle import make_config, port

pytestmark = pytest.mark.gpu


class Ions:
    def __init__(self, box, seed, n=120):
        rng = np.random.default_rng(seed)
        self.nsite, self.box = n, np.asarray(box, dtype=np.float64)
        self.positions = rng.uniform(0, 1, (n, 3)) * self.box
        self.groups = np.stack([np.arange(n), np.arange(n) + 1], 1)
        self.exclusions = np.zeros((0, 2), dtype=np.int64)
        self.site_mask = np.full(n, 1, dtype=np.int32)
        self.q = np.where(np.arange(n) % 2, 0.3, -0.3)
        self.sigma, self.epsilon, self.rscreen = np.zeros(n), np.zeros(n), np.zeros(n)


# (6, 4, 9) ... : products of 2..10 and 12; (8, 144, 100) and (8, 120, 112): an FP64
# plane too large for a block; (14, 98, 7), (5, 10, 12): lengths without two radices
MESHES = [(6, 4, 9), (10, 12, 14), (15, 16, 18), (20, 21, 24), (25, 27, 28), (30, 32, 35), (36, 40, 42), (45, 48, 49),
          (9, 50, 54), (56, 9, 60), (63, 64, 10), (12, 70, 72), (80, 14, 81), (84, 90, 16), (18, 96, 100),
          (108, 20, 120), (144, 21, 8), (8, 144, 100), (14, 98, 7), (5, 10, 12)]


@pytest.mark.parametrize("mesh", MESHES)
@pytest.mark.parametrize("ik", [False, True])
def test_mesh_lengths(mesh, ik):
    # 0.9 A a point keeps the spectrum's tail in reach of every axis; the shortest box
    # edge still holds the cutoff
    spacing = max(0.9, 6.5 / min(mesh))
    s = Ions(np.array(mesh) * spacing, seed=sum(mesh))
    cfg = dict(rspace_cutoff=3.0, ewald_screening=0.35, use_p3m=True, p3m_grid_spacing=spacing,
               p3m_assignment_order=4, p3m_ik_differentiate=ik, include_rspace=False, include_self=False)
    o = port().eleclj(make_config(s.box, bctype=_lib.MMNB_ORTHORHOMBIC, **cfg), s.nsite, s.groups, s.exclusions,
                      s.site_mask, s.q, s.sigma, s.epsilon, s.rscreen).eval(s.positions)
    for precision in ("fp64", "mixed"):
        if ik and np.prod(mesh) % 2:
            continue  # refused
        pot = ElecLJ(precision=precision, **cfg).init(s, bctype=_lib.MMNB_ORTHORHOMBIC)
        assert pot.settings()["mesh"] == mesh
        for _ in range(2):  # the mesh is left as the next evaluation needs it
            g = pot.compute(s.positions)
        pot.close()
        if precision == "fp64":
            assert rel_max(g["f"], o["f"]) < 1e-10
            assert abs(g["elec"] - o["elec"]) < 1e-10 * abs(o["elec"])
        else:
            assert rel_rms(g["f"], o["f"]) < 1e-5
