"""Site pairs past the erfc table's end (r^2 > 1.2 rc^2, anchors within the cutoff) in
the FP64 pair kernel for any groups: erfc and exp, as the reference has them.  One such
pair alone, so its potential and field are the whole answer: 1e-12 relative (a few
ulp of erfc and exp, whose argument (eta r)^2 <= 40 carries its own rounding)."""
import math

import numpy as np
import pytest

from molmodel_b200 import ElecLJ

pytestmark = pytest.mark.gpu

RC = 9.0


class Pair:
    """two groups of two sites: anchors that carry nothing `apart` from one another, a
    charge `out` beyond each"""

    def __init__(self, apart, out):
        self.nsite, self.box = 4, 40.0
        u = np.array([2.0, -1.0, 2.0]) / 3
        a = np.array([11.0, 12.0, 13.0])
        self.positions = np.array([a, a - out * u, a + apart * u, a + (apart + out) * u])
        self.groups = np.array([[0, 2], [2, 4]])
        self.exclusions = np.zeros((0, 2), dtype=np.int64)
        self.site_mask = np.array([0, 1, 0, 1], dtype=np.int32)
        self.q = np.array([0.0, 1.5, 0.0, -2.0])
        self.sigma = self.epsilon = self.rscreen = np.zeros(4)


@pytest.mark.parametrize("eta", [0.2, 0.26, 0.35, 0.5])
@pytest.mark.parametrize("apart,out", [(7.9, 1.0), (7.9, 1.5), (7.0, 2.1)])
def test_pair_past_the_table(eta, apart, out):
    s = Pair(apart, out)
    g = ElecLJ(rspace_cutoff=RC, smoothing_width=1.0, ewald_screening=eta, include_kspace=False,
               include_self=False).init(s).compute(s.positions, want_fields=True)
    d = s.positions[1] - s.positions[3]
    r2 = float(d @ d)
    r = math.sqrt(r2)
    assert r2 > 1.2 * RC * RC
    b0 = math.erfc(eta * r) / r
    b1 = (b0 + 2 * eta / math.sqrt(math.pi) * math.exp(-eta * eta * r2)) / r2
    assert abs(g["phi"][1] - s.q[3] * b0) <= 1e-12 * abs(s.q[3] * b0)
    e = s.q[3] * b1 * d
    assert np.abs(g["evec"][1] - e).max() <= 1e-12 * np.abs(e).max()
    f = s.q[1] * e
    assert np.abs(g["f"][1] - f).max() <= 1e-12 * np.abs(f).max()
