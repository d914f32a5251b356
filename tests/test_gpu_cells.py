"""The list's cell sort with crowded cells: around the size past which a block counts
a cell's groups instead of walking the cell's list (512), in the one-block form and in
the two-kernel form, one such cell and two, and cells in several chunks of counts.  The
pair set and the cells are the oracle's."""
import numpy as np
import pytest

from molmodel_b200 import ElecLJ
from oracle.oracle import make_config, port

pytestmark = pytest.mark.gpu


class Crowds:
    """single charged sites, `crowds` of them each in a cell of the list"""

    def __init__(self, n, crowds, seed):
        rng = np.random.default_rng(seed)
        self.nsite, self.box = n, 36.0
        self.positions = rng.uniform(0, self.box, (n, 3))
        at = np.split(rng.permutation(n)[:sum(crowds)], np.cumsum(crowds)[:-1])
        for k, i in enumerate(at):
            self.positions[i] = (5.0 + 9.0 * k) + rng.uniform(-0.2, 0.2, (len(i), 3))
        self.groups = np.stack([np.arange(n), np.arange(n) + 1], 1)
        self.exclusions = np.zeros((0, 2), dtype=np.int64)
        self.site_mask = np.full(n, 1, dtype=np.int32)
        self.q = np.where(np.arange(n) % 2, 0.3, -0.3)
        self.sigma, self.epsilon, self.rscreen = np.zeros(n), np.zeros(n), np.zeros(n)


@pytest.mark.parametrize("n,crowds", [(512, (512,)), (1500, (513,)), (2048, (700, 600)), (2049, (511, 513)),
                                      (5000, (514,)), (5000, (900, 40, 700)), (20000, (30, 520, 17))])
def test_crowded_cells(n, crowds):
    s = Crowds(n, crowds, seed=n)
    cfg = dict(rspace_cutoff=4.0, neighbor_list_width=0.5, ewald_screening=0.4, kspace_cutoff=2.0)
    pot = ElecLJ(**cfg).init(s)
    pot.compute(s.positions)
    o = port().eleclj(make_config(s.box, **cfg), s.nsite, s.groups, s.exclusions, s.site_mask, s.q, s.sigma,
                      s.epsilon, s.rscreen)
    o.eval(s.positions)
    cells, ncell = pot.cells(n)
    assert ncell == o.nbrlist().ncell() and np.array_equal(cells, o.nbrlist().cells(n))
    canon = lambda p: np.unique(np.sort(np.asarray(p), axis=1), axis=0)  # noqa: E731
    assert np.array_equal(canon(pot.pairlist()), canon(o.nbrlist().pairs()))
