"""The pair kernels for groups of any size, at the group sizes, row counts and
screening parameters where their queues, teams of warps and short-range branch can
go wrong, against the oracle (FP64 form: 1e-10; mixed form: 1e-5 RMS, both the
forms' bounds)."""
import numpy as np
import pytest

from conftest import rel_max, rel_rms
from molmodel_b200 import ElecLJ, water_box_n
from oracle.oracle import make_config, port

pytestmark = pytest.mark.gpu

TOL = 1e-10


class Grouped:
    """Water sites regrouped by the given sizes in turn, with sites that carry
    charge, LJ, both or neither, and exclusions within and across groups."""

    def __init__(self, nwater, sizes, seed, neutral_sites=True):
        wb = water_box_n(nwater, seed)
        rng = np.random.default_rng(seed)
        n = self.nsite = wb.nsite
        self.box, self.positions = wb.box, wb.positions
        edges, k = [0], 0
        while edges[-1] < n:
            edges.append(min(n, edges[-1] + sizes[k % len(sizes)]))
            k += 1
        self.groups = np.stack([edges[:-1], edges[1:]], 1)
        kind = rng.integers(0, 4, n) if neutral_sites else np.full(n, 3)
        self.site_mask = kind.astype(np.int32)
        self.q = np.where(kind & 1, wb.q, 0.0)
        self.sigma = np.where(kind & 2, rng.uniform(0.5, 1.2, n), 0.0)
        self.epsilon = np.where(kind & 2, rng.uniform(0.01, 0.1, n), 0.0)
        self.rscreen = np.zeros(n)
        i = rng.integers(0, n - 4, n // 6)
        self.exclusions = np.concatenate([wb.exclusions, np.stack([i, i + rng.integers(1, 4, len(i))], 1)])


def check(s, **kw):
    cfg = dict(rspace_cutoff=6.0, ewald_screening=0.4, kspace_cutoff=4.0)
    cfg.update(kw)
    g = ElecLJ(**cfg).init(s).compute(s.positions, want_fields=True)
    o = port().eleclj(make_config(s.box, **cfg), s.nsite, s.groups, s.exclusions, s.site_mask, s.q, s.sigma,
                      s.epsilon, s.rscreen).eval(s.positions)
    for k in ("f", "phi", "evec"):
        assert rel_max(g[k], o[k]) < TOL, k
    for k in ("elec", "lj", "total"):
        assert abs(g[k] - o[k]) <= TOL * abs(o[k]), k


# one site to eight a group, and mixtures: the queues' batches and carries
@pytest.mark.parametrize("sizes", [(1,), (2,), (1, 2, 3), (4, 1), (5, 3), (8,), (7, 1, 8, 2)])
def test_group_sizes(sizes):
    check(Grouped(125, sizes, seed=sum(sizes)))


# rows for teams of four and two warps, and for single warps taking several rows
@pytest.mark.parametrize("nwater", [64, 433, 900, 2100])
def test_row_counts(nwater):
    check(Grouped(nwater, (3,), seed=nwater))


# eta times the table's lower end below and above the series' range; geometric
# combining; a table too large for two copies (small rc); no switch
@pytest.mark.parametrize("kw", [dict(ewald_screening=0.2), dict(ewald_screening=0.42), dict(ewald_screening=0.6),
                                dict(geometric_combining_for_sigma=1), dict(rspace_cutoff=3.0),
                                dict(smoothing_width=0.0)])
def test_parameters(kw):
    check(Grouped(216, (3, 4), seed=9), **kw)


def test_screened_charges():
    s = Grouped(216, (3, 2), seed=4)
    s.rscreen = np.where(np.arange(s.nsite) % 4 == 0, 1.5, 0.0)
    check(s)


# rigid water: the series' range, one copy of the table, and waters that differ
@pytest.mark.parametrize("eta", [0.2, 0.42, 0.6])
@pytest.mark.parametrize("uniform", [True, False])
def test_rigid_water(eta, uniform):
    wb = water_box_n(1000, 3)

    class S:
        nsite, box, groups, exclusions, site_mask = wb.nsite, wb.box, wb.groups, wb.exclusions, wb.site_mask
        q, sigma, epsilon, rscreen, positions = wb.q.copy(), wb.sigma, wb.epsilon, wb.rscreen, wb.positions
    if not uniform:
        S.q[0] *= 1.01
    check(S, ewald_screening=eta)


@pytest.mark.parametrize("sizes", [(1,), (2,), (1, 2, 3), (4, 1), (5, 3), (8,), (7, 1, 8, 2)])
def test_mixed_group_sizes(sizes):
    s = Grouped(216, sizes, seed=sum(sizes))
    s.rscreen = np.where(np.arange(s.nsite) % 5 == 0, 1.5, 0.0)
    cfg = dict(rspace_cutoff=7.0, ewald_screening=0.4, kspace_cutoff=4.0)
    o = port().eleclj(make_config(s.box, **cfg), s.nsite, s.groups, s.exclusions, s.site_mask, s.q, s.sigma,
                      s.epsilon, s.rscreen).eval(s.positions)
    ref = None
    # fixed-point sums: the same bits whatever the list holds beyond the cutoff
    for width in (0.3, 1.5):
        g = ElecLJ(precision="mixed", neighbor_list_width=width, **cfg).init(s).compute(s.positions, want_fields=True)
        assert rel_rms(g["f"], o["f"]) < 1e-5
        assert rel_rms(g["phi"], o["phi"]) < 1e-5
        assert abs(g["total"] - o["total"]) < 5e-5 * abs(o["total"])
        if ref is not None:
            assert np.array_equal(g["f"], ref["f"]) and g["lj"] == ref["lj"]
        ref = g
