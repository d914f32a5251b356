"""A kspace_cutoff with more wave vectors than an int counts (from 1008 on) is a bad
argument, to a handle whose forces take the k-sum and to the potential at points; the
handle stays usable."""
import numpy as np
import pytest

from molmodel_b200 import ElecLJ, _lib, water_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kc", [1008.0, 1e6])
def test_cutoff_past_the_index_range(kc):
    wb = water_box(6, seed=1)
    cfg = dict(rspace_cutoff=7.0, ewald_screening=0.35, kspace_cutoff=kc)
    with pytest.raises(_lib.MmnbError) as ex:
        ElecLJ(**cfg).init(wb)
    assert ex.value.status == 1, ex.value.status  # MMNB_ERR_ARG
    p = ElecLJ(use_p3m=True, p3m_grid_spacing=1.0, **cfg).init(wb)
    for _ in range(2):
        with pytest.raises(_lib.MmnbError) as ex:
            p.electrostatic_potential_at_gridpoints(wb.positions, wb.positions[:3] + 1.0)
        assert ex.value.status == 1, ex.value.status
    assert np.isfinite(p.compute(wb.positions)["f"]).all()
