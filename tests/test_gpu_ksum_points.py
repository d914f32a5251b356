"""The Ewald k-sum's kernels and the potential at points at the sizes where
their tiles and cells can go wrong, against sums over all wave vectors and all
sites (numpy, FP64) and the oracle.  1e-10 relative, the FP64 form's bound: a
term is a few products of phases good to an ulp, so sums of up to 33,000 terms
stay within ~1e-13 of their RMS."""
import numpy as np
import pytest

from conftest import rel_max
from molmodel_b200 import ElecLJ, water_box
from oracle.oracle import make_config, port

pytestmark = pytest.mark.gpu

TOL = 1e-10


class Ions:
    """Charges in groups of one, some of them outside the box."""

    def __init__(self, n, seed):
        rng = np.random.default_rng(seed)
        self.nsite = n
        self.box = np.array([11.0, 13.5, 9.25])
        self.positions = rng.uniform(-1.5, 2.5, (n, 3)) * self.box
        self.groups = np.stack([np.arange(n), np.arange(n) + 1], 1)
        self.exclusions = np.zeros((0, 2))
        self.site_mask = np.ones(n, dtype=np.int32)
        self.q = rng.normal(size=n)
        self.sigma = self.epsilon = self.rscreen = np.zeros(n)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 97])
# nmax 0 (no wave vectors), 1, a sum in shared memory, one that is not (tiles of 16 sites too)
@pytest.mark.parametrize("kc", [0.9, 1.0, 5.5, 25.0])
def test_ksum_potential_and_field(n, kc):
    s = Ions(n, seed=n)
    eta = 0.1 * kc + 0.2
    p = ElecLJ(rspace_cutoff=4.0, ewald_screening=eta, kspace_cutoff=kc, include_rspace=False,
               include_self=False).init(s, bctype=2)
    out = p.compute(s.positions, want_fields=True)
    m = int(kc)
    g = np.arange(-m, m + 1)
    k = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    n2 = (k ** 2).sum(1)
    k = k[(n2 > 0) & (n2 <= kc * kc)] * (2 * np.pi / s.box)
    if len(k) == 0:
        assert not out["phi"].any() and not out["f"].any()
        return
    k2 = (k ** 2).sum(1)
    a = 4 * np.pi / s.box.prod() * np.exp(-k2 / (4 * eta ** 2)) / k2
    e = np.exp(1j * (s.positions @ k.T))
    t = a * (s.q @ e) * e.conj()
    assert rel_max(out["phi"], t.real.sum(1)) < TOL
    field = -(t.imag @ k)
    scale = np.sqrt((np.abs(t) ** 2 @ k2).mean())
    assert np.abs(out["evec"] - field).max() < TOL * scale


@pytest.mark.parametrize("stretch", [(1.0, 1.0, 1.0), (1.0, 1.4, 2.3), (2.6, 1.0, 1.1)])
# one cell or all cells of an axis in reach, up to more cells than are reached
@pytest.mark.parametrize("n,rc", [(2, 2.5), (3, 4.0), (7, 4.0), (7, 9.5), (10, 5.0)])
def test_points_in_and_around_cells(n, rc, stretch):
    wb = water_box(n, seed=n)
    rng = np.random.default_rng(n)
    box = wb.box * np.array(stretch)
    r = wb.positions * np.array(stretch)
    # whole molecules moved by box vectors, and a crowd in one corner
    r = (r.reshape(-1, 3, 3) + rng.integers(-2, 3, (wb.nwater, 1, 3)) * box).reshape(-1, 3)
    r[:wb.nsite // 4] = rng.uniform(0, 0.2, (wb.nsite // 4, 3)) * box

    class S:
        nsite, groups, exclusions, sigma, epsilon, q = (wb.nsite, wb.groups, wb.exclusions, wb.sigma, wb.epsilon, wb.q)
        site_mask = np.where(np.arange(wb.nsite) % 7 == 3, 0, wb.site_mask).astype(np.int32)
        rscreen = np.where(np.arange(wb.nsite) % 3 == 0, 1.6, 0.0)
    S.box = box
    pts = np.concatenate([rng.uniform(-1, 2, (70, 3)) * box, r[::5] + rng.normal(scale=0.3, size=r[::5].shape),
                          np.zeros((1, 3)), box[None, :], box[None, :] / 2])
    cfg = dict(rspace_cutoff=rc, smoothing_width=0.7, ewald_screening=0.4, kspace_cutoff=3.0)
    o = port().eleclj(make_config(box, bctype=2, **cfg), S.nsite, S.groups, S.exclusions, S.site_mask, S.q, S.sigma,
                      S.epsilon, S.rscreen)
    phi = ElecLJ(**cfg).init(S, bctype=2).electrostatic_potential_at_gridpoints(r, pts)
    ref = o.phi_at_points(r, pts)
    # the middle of an odd lattice is a site: the distance there is rounding (or
    # zero), and so is the sum of its 1/r and the screening's -1/r
    d = pts[:, None, :] - r[None, :, :]
    d -= box * np.floor(d / box + 0.5)
    off = (d ** 2).sum(-1).min(1) > 1e-12
    assert off.sum() >= len(pts) - 1
    assert rel_max(phi[off], ref[off]) < TOL


def test_points_with_a_coordinate_that_is_not_finite():
    """As in a sum over all pairs: a bad site gives NaN everywhere, a bad point at that point."""
    wb = water_box(5, seed=1)
    p = ElecLJ(rspace_cutoff=6.0, ewald_screening=0.4).init(wb)
    pts = np.random.default_rng(1).uniform(0, wb.box, (9, 3))
    for bad in (np.nan, np.inf):
        r = wb.positions.copy()
        r[7, 1] = bad
        assert np.isnan(p.electrostatic_potential_at_gridpoints(r, pts)).all()
        q = pts.copy()
        q[4, 2] = bad
        phi = p.electrostatic_potential_at_gridpoints(wb.positions, q)
        assert np.isnan(phi[4]) and np.isfinite(np.delete(phi, 4)).all()
