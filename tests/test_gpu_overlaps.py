"""A box whose sites overlap, as a packed box does before it is relaxed: the mixed form's
pair energy and virial past the range of one fixed-point word (2^31), each row's within
it.  Pairs of LJ sites 0.9 A apart: 8.4e6 kcal/mol a pair.  FP32 terms with r^-12 of
coordinates good to 1e-7: the bounds are the mixed form's energy bound and, the virial
being 12 times the energy with the same relative error, the same for it."""
import numpy as np
import pytest

from molmodel_b200 import ElecLJ
from oracle.oracle import make_config, port

pytestmark = pytest.mark.gpu

ENERGY_TOL = 5e-5


class Overlaps:
    """n^3 pairs of sites, each site its own group, 5 A between pairs"""

    def __init__(self, n):
        rng = np.random.default_rng(n)
        step = 5.0
        c = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3) * step
        d = rng.normal(size=c.shape)
        d *= 0.45 / np.linalg.norm(d, axis=1)[:, None]
        self.positions = np.stack([c - d, c + d], 1).reshape(-1, 3)
        self.nsite, self.box = 2 * n ** 3, n * step
        k = np.arange(self.nsite)
        self.groups = np.stack([k, k + 1], 1)
        self.exclusions = np.zeros((0, 2), dtype=np.int64)
        self.site_mask = np.full(self.nsite, 2, dtype=np.int32)
        self.q, self.rscreen = np.zeros(self.nsite), np.zeros(self.nsite)
        self.sigma, self.epsilon = np.full(self.nsite, 3.4), np.full(self.nsite, 0.25)


@pytest.mark.parametrize("n", [6, 10])  # 1.8e9: within the word; 8.4e9
def test_energy_and_virial_of_overlapping_sites(n):
    s = Overlaps(n)
    cfg = dict(rspace_cutoff=9.0, neighbor_list_width=1.0, ewald_screening=0.35, kspace_cutoff=3.0)
    o = port().eleclj(make_config(s.box, **cfg), s.nsite, s.groups, s.exclusions, s.site_mask, s.q, s.sigma,
                      s.epsilon, s.rscreen).eval(s.positions)
    mass = np.ones(s.nsite)
    w64, e64, _ = ElecLJ(precision="fp64", **cfg).init(s).virial(s.positions, mass)
    p = ElecLJ(precision="mixed", **cfg).init(s)
    w, e, _ = p.virial(s.positions, mass)
    lj = p.compute(s.positions)["lj"]
    assert abs(e64["lj"] - o["lj"]) <= 1e-10 * abs(o["lj"])
    assert abs(lj - o["lj"]) <= ENERGY_TOL * abs(o["lj"])
    assert abs(e["lj"] - o["lj"]) <= ENERGY_TOL * abs(o["lj"])
    assert abs(w - w64) <= ENERGY_TOL * abs(w64)
