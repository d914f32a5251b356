"""The per-site kernel in the layout of large boxes (a lane per site, whole 16-byte
words of a mesh row where the row has only such), and the list's cell sort on both
sides of its one-block limit with crowded cells.

A box repeated r times along each axis on an r times finer mesh has the forces of
the single box, whose small layout other tests hold against the oracle.  Bounds:
FP64 1e-10; mixed 1e-5 RMS (each box differs from the exact field by less)."""
import numpy as np
import pytest

from conftest import rel_max, rel_rms
from molmodel_b200 import ElecLJ, water_box
from oracle.oracle import make_config, port

pytestmark = pytest.mark.gpu


class Repeated:
    """`wb` repeated r times along each axis (r = 1: itself)"""

    def __init__(self, wb, r):
        k = np.stack(np.meshgrid(*[np.arange(r)] * 3, indexing="ij"), -1).reshape(-1, 3)
        m = len(k)
        self.nsite, self.box = wb.nsite * m, wb.box * r
        self.positions = (wb.positions[None] + k[:, None] * wb.box).reshape(-1, 3)
        off = wb.nsite * np.arange(m)[:, None, None]
        self.groups = (wb.groups[None] + off).reshape(-1, 2)
        self.exclusions = (wb.exclusions[None] + off).reshape(-1, 2)
        for a in ("site_mask", "q", "sigma", "epsilon"):
            setattr(self, a, np.tile(getattr(wb, a), m))
        self.rscreen = np.zeros(self.nsite)


# rows of 30 points (whole words in FP64 only), 60, 40 and 48 (in both forms) and
# 35 (in neither), of 41,472 and 81,000 sites: above the limit
@pytest.mark.parametrize("mesh,rep,order,ik", [(6, 5, 5, False), (15, 4, 5, False), (10, 4, 4, True), (7, 5, 7, False),
                                               (8, 5, 2, True), (6, 5, 3, True), (12, 4, 6, False)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lane_per_site(mesh, rep, order, ik, precision):
    wb = water_box(6, seed=mesh)
    out = []
    for r in (1, rep):
        pot = ElecLJ(precision=precision, rspace_cutoff=6.0, ewald_screening=0.35, neighbor_list_width=1.0,
                     use_p3m=True, p3m_grid_spacing=wb.box / mesh, p3m_assignment_order=order,
                     p3m_ik_differentiate=ik).init(Repeated(wb, r))
        g = pot.compute(Repeated(wb, r).positions)
        assert pot.settings()["mesh"] == (r * mesh,) * 3
        pot.close()
        out.append(g)
    one, many = out
    m = rep ** 3
    want = np.tile(one["f"], (m, 1))
    if precision == "fp64":
        assert rel_max(many["f"], want) < 1e-10
        tol = 1e-10
    else:
        assert rel_rms(many["f"], want) < 1e-5
        tol = 1e-5
    for k in ("elec", "lj"):
        assert abs(many[k] - m * one[k]) < tol * m * abs(one["elec"]), k


class Clustered:
    """single charged sites, `crowd` of them within a cell of the list"""

    def __init__(self, n, crowd, seed):
        rng = np.random.default_rng(seed)
        self.nsite, self.box = n, 30.0
        self.positions = rng.uniform(0, self.box, (n, 3))
        at = rng.permutation(n)[:crowd]
        self.positions[at] = 7.0 + rng.uniform(-0.3, 0.3, (crowd, 3))
        self.groups = np.stack([np.arange(n), np.arange(n) + 1], 1)
        self.exclusions = np.zeros((0, 2), dtype=np.int64)
        self.site_mask = np.full(n, 1, dtype=np.int32)
        self.q = np.where(np.arange(n) % 2, 0.3, -0.3)
        self.sigma, self.epsilon, self.rscreen = np.zeros(n), np.zeros(n), np.zeros(n)


# cells at and past the size ordered by one thread; last one-block and first two-kernel
# sizes (2048, 2049), one cell (7 groups: n = 1) and several passes of the block
@pytest.mark.parametrize("n,crowd", [(7, 7), (300, 16), (300, 17), (2048, 60), (2049, 16), (2049, 60), (6000, 120)])
def test_cell_sort(n, crowd):
    s = Clustered(n, crowd, seed=n + crowd)
    cfg = dict(rspace_cutoff=5.0, neighbor_list_width=1.0, ewald_screening=0.4, kspace_cutoff=2.0)
    pot = ElecLJ(**cfg).init(s)
    pot.compute(s.positions)
    o = port().eleclj(make_config(s.box, **cfg), s.nsite, s.groups, s.exclusions, s.site_mask, s.q, s.sigma,
                      s.epsilon, s.rscreen)
    o.eval(s.positions)
    canon = lambda p: np.unique(np.sort(np.asarray(p), axis=1), axis=0)
    assert np.array_equal(canon(pot.pairlist()), canon(o.nbrlist().pairs()))
    cells, ncell = pot.cells(n)
    assert ncell == o.nbrlist().ncell() and np.array_equal(cells, o.nbrlist().cells(n))
