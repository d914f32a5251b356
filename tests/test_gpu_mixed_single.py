"""The mixed form's pair kernel for groups of one site, against the FP64 oracle: rows
shorter than a warp and longer, with and without exclusions across groups, screening
radii and the virial's term.  Bounds of the mixed form's other general tests."""
import numpy as np
import pytest

from conftest import rel_rms
from molmodel_b200 import ElecLJ
from oracle.oracle import make_config, port

pytestmark = pytest.mark.gpu

RMS_TOL = 1e-5
ENERGY_TOL = 5e-5


class Lattice:
    """n^3 sites on a jittered lattice, every third uncharged, every fifth without LJ"""

    def __init__(self, n, step, excluded, screened):
        rng = np.random.default_rng(n)
        c = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
        self.nsite, self.box = n ** 3, n * step
        self.positions = (c + rng.uniform(-0.15, 0.15, c.shape)) * step
        k = np.arange(self.nsite)
        self.groups = np.stack([k, k + 1], 1)
        pairs = np.stack([k[:-1], k[1:]], 1)[rng.random(self.nsite - 1) < 0.3]
        self.exclusions = pairs if excluded else np.zeros((0, 2), dtype=np.int64)
        self.site_mask = np.where(k % 3, 1, 0) | np.where(k % 5, 2, 0)
        self.q = np.where(k % 3, rng.choice([-4.0, 4.0], self.nsite), 0.0)
        self.sigma, self.epsilon = np.where(k % 5, 2.6, 0.0), np.where(k % 5, 0.15, 0.0)
        self.rscreen = np.where(k % 4, 0.0, 1.5) if screened else np.zeros(self.nsite)


@pytest.mark.parametrize("excluded", [False, True])
@pytest.mark.parametrize("screened", [False, True])
@pytest.mark.parametrize("n,step,rc", [(5, 4.0, 4.5), (9, 2.9, 8.0), (12, 2.5, 9.0)])
def test_single_sites(n, step, rc, screened, excluded):
    s = Lattice(n, step, excluded, screened)
    cfg = dict(rspace_cutoff=rc, neighbor_list_width=0.7, ewald_screening=0.4, kspace_cutoff=4.0)
    o = port().eleclj(make_config(s.box, **cfg), s.nsite, s.groups, s.exclusions, s.site_mask, s.q, s.sigma,
                      s.epsilon, s.rscreen).eval(s.positions)
    g = ElecLJ(precision="mixed", **cfg).init(s).compute(s.positions)
    assert rel_rms(g["f"], o["f"]) < RMS_TOL
    for k in ("elec", "lj"):
        assert abs(g[k] - o[k]) < ENERGY_TOL * (abs(o["elec"]) + abs(o["lj"])), k
    if not screened:
        mass = np.ones(s.nsite)
        w, _, _ = ElecLJ(precision="mixed", **cfg).init(s).virial(s.positions, mass)
        w64, _, _ = ElecLJ(precision="fp64", **cfg).init(s).virial(s.positions, mass)
        assert abs(w - w64) < ENERGY_TOL * (abs(w64) + abs(o["elec"]) + abs(o["lj"]))
