"""Exclusions across groups in the FP64 pair kernel for any groups: a row's excluded sites
as masks while they lie within 64 indices, searched for past that, rows of both kinds and
of none in one box.  Against the oracle, 1e-10: the FP64 form's bound."""
import numpy as np
import pytest

from conftest import rel_max
from molmodel_b200 import ElecLJ
from oracle.oracle import make_config, port

pytestmark = pytest.mark.gpu


class Lattice:
    """n^3 groups of k sites; site i of every third group excludes the sites `reach`
    indices on (those in its own group too), a few pairs anywhere in the box"""

    def __init__(self, n, k, reach, anywhere):
        rng = np.random.default_rng(100 * k + reach)
        c = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3) * 3.0
        body = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 1, 0], [1, 0, 1], [0, 1, 1], [1, 1, 1]])[:k]
        self.nsite, self.box = n ** 3 * k, n * 3.0
        self.positions = (c[:, None] + 1.1 * body + rng.uniform(-0.1, 0.1, (n ** 3, k, 3))).reshape(-1, 3)
        g = np.arange(n ** 3) * k
        self.groups = np.stack([g, g + k], 1)
        i = np.arange(self.nsite)[(np.arange(self.nsite) // k) % 3 == 0]
        ex = [np.stack([i, i + d], 1)[i + d < self.nsite] for d in (1, 2, reach)]
        ex.append(rng.integers(0, self.nsite, (anywhere, 2)))
        ex = np.concatenate(ex)
        self.exclusions = ex[ex[:, 0] != ex[:, 1]]
        self.site_mask = rng.choice([1, 2, 3, 3, 3], self.nsite).astype(np.int32)
        self.q = np.where(self.site_mask & 1, rng.choice([-4.0, 4.0], self.nsite), 0.0)
        self.sigma, self.epsilon = np.full(self.nsite, 2.0), np.full(self.nsite, 0.1)
        self.rscreen = np.zeros(self.nsite)


# spans of 64 and 65 indices, and far ones
@pytest.mark.parametrize("k,reach", [(1, 3), (1, 31), (1, 32), (1, 63), (1, 64), (1, 65), (3, 5), (3, 61), (3, 62),
                                     (3, 200), (8, 10), (8, 56), (8, 57), (8, 300)])
@pytest.mark.parametrize("anywhere", [0, 40])
def test_exclusions_across_groups(k, reach, anywhere):
    s = Lattice(8 if k < 8 else 7, k, reach, anywhere)
    cfg = dict(rspace_cutoff=8.0, neighbor_list_width=1.0, ewald_screening=0.35, kspace_cutoff=3.0)
    o = port().eleclj(make_config(s.box, **cfg), s.nsite, s.groups, s.exclusions, s.site_mask, s.q, s.sigma,
                      s.epsilon, s.rscreen).eval(s.positions)
    g = ElecLJ(**cfg).init(s).compute(s.positions, want_fields=True)
    assert rel_max(g["f"], o["f"]) < 1e-10
    assert rel_max(g["phi"], o["phi"]) < 1e-10
    for e in ("elec", "lj"):
        assert abs(g[e] - o[e]) < 1e-10 * (abs(o["elec"]) + abs(o["lj"])), e
