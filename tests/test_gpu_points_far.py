"""Potential at points many boxes away, and of sites many boxes away: past 2^30 box
lengths a wrapped coordinate is rounding (and may lie outside the box), so such points,
and all points of such sites, take every site one by one; the minimum image's rounding
is the oracle's, so the values are too (1e-10, the FP64 form's bound).

Without the k-sum: a phase k.r of such a coordinate is rounding in either code."""
import numpy as np
import pytest

from conftest import rel_max
from molmodel_b200 import ElecLJ, water_box
from oracle.oracle import make_config, port

pytestmark = pytest.mark.gpu

CFG = dict(rspace_cutoff=6.0, smoothing_width=0.7, ewald_screening=0.4, include_kspace=False)


def check(wb, r, pts):
    o = port().eleclj(make_config(wb.box, **CFG), wb.nsite, wb.groups, wb.exclusions, wb.site_mask, wb.q, wb.sigma,
                      wb.epsilon, np.zeros(wb.nsite))
    phi = ElecLJ(**CFG).init(wb).electrostatic_potential_at_gridpoints(r, pts)
    ref = o.phi_at_points(r, pts)
    # (a displacement rounded to zero gives infinity in either)
    some = np.isfinite(ref)
    assert np.array_equal(phi[~some], ref[~some])
    assert not some.any() or rel_max(phi[some], ref[some]) < 1e-10


def box_multiples(box):
    """near, and on both sides of 2^30 box lengths (in whole boxes and a bit), then far"""
    return [k * box + 3.25 for k in (2.0 ** 20, 2.0 ** 29, 2.0 ** 30, 2.0 ** 31, -2.0 ** 31)] + \
        [1e14, 1e18, -1e18, 3e18, 3e19, -3e19, 1e25, 1e100, -1e300]


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [6, 9])
def test_far_points(n, axis):
    wb = water_box(n, seed=n)
    far = box_multiples(wb.box)
    pts = np.random.default_rng(axis).uniform(0, wb.box, (4 * len(far), 3))
    pts[::2, axis] = np.repeat(far, 2)
    check(wb, wb.positions, pts)


@pytest.mark.parametrize("where", [2.0 ** 29, 2.0 ** 31, 1e17])
def test_far_sites(where):
    wb = water_box(6, seed=2)
    r = wb.positions.copy()
    r[5] += np.round(where) * wb.box
    r[40, 2] -= np.round(where) * wb.box
    check(wb, r, np.random.default_rng(3).uniform(0, wb.box, (50, 3)))
