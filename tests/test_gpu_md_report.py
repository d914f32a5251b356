"""A run's start and end kernels over more integrators than one launch takes, with logs
that fit the report and logs that do not: every replica's energies are those of the
same replica run by itself (mixed form: bitwise)."""
import numpy as np
import pytest

from molmodel_b200 import ElecLJ, maxwell_boltzmann, water_box_n
from molmodel_b200.md import MDyn, ReplicaBatch

pytestmark = pytest.mark.gpu


def replica(k):
    wb = water_box_n(27 + k % 5, seed=k)
    pot = ElecLJ(precision="mixed", rspace_cutoff=3.5, ewald_screening=0.6, neighbor_list_width=0.4, use_p3m=True,
                 p3m_grid_spacing=1.1, p3m_assignment_order=4).init(wb)
    md = MDyn(pot, wb.masses, timestep=0.0005)
    md.set_state(wb.positions, maxwell_boltzmann(wb, 200.0, seed=k))
    return md


# 2^17 words of log: 3 steps n from 662 steps of 66 replicas on
@pytest.mark.parametrize("n,steps", [(1, 1), (66, 3), (66, 663)])
def test_batch_energies(n, steps):
    mds = [replica(k) for k in range(n)]
    got = ReplicaBatch(mds).run(steps)
    for k in {0, n // 2, n - 2, n - 1} - {-1}:
        alone = replica(k).run(steps)
        assert got[k].shape == (steps, 3) and np.array_equal(got[k], alone), k
