"""The work that users of molmodel_b200 have it do, as cases to be timed.

Each case is one call (or one short run) through the package's public entry
points, in the form a simulation or fitting program makes it:

  host     ElecLJ.add_to_energy_and_forces on host arrays: the reference's own
           per-step call, k-sum or P3M
  device   an evaluation on device arrays, replayed from its captured graph
  md       MDyn.run: ten steps of rigid-water dynamics
  batch    ReplicaBatch.run: ten steps of a set of replicas of uneven size
  fit      ElecLJ.forward and site_gradients: one frame of a force-matching fit
  charges  ElecLJ.set_params and compute with the site fields: one sweep of a
           self-consistent charge solve
  virial   ElecLJ.virial: the pressure of a constant-pressure run
  points   ElecLJ.electrostatic_potential_at_gridpoints: a potential grid

The systems are this package's synthetic water boxes (any number of waters)
and solutions: the same water lattice in which about one pair of cells in eight
holds a six-site solute of two groups, with 1-4 pairs scaled and exclusions across
its groups.  Settings are those of the repository's configurations: cutoff 9 A,
switch 1 A, screening 0.35 / A, skin 1.5 A, lists rebuilt every ten evaluations,
P3M at about 1.04 A spacing and order 5 (the charge sweeps use the package's
own default mesh, 0.5 A and order 3).

The mixed-precision form's numbers are FP32 sums (about 4e-6 RMS), and a
program that picks it keeps forces, velocities and energies in float32, as
trajectory files and training sets hold them: the mixed cases end with that
conversion.  The FP64 form's outputs are kept as they come.
"""
import itertools
import math

import numpy as np
import torch

from molmodel_b200 import ElecLJ, maxwell_boltzmann, water_box_n
from molmodel_b200.md import MDyn, ReplicaBatch
from molmodel_b200.remd import replica_sizes, temperature_ladder
from molmodel_b200.units import e_to_charge_unit
from molmodel_b200.water import (EPSILON_O, MASS_H, MASS_O, SIGMA_O, SITE_HAS_LJ, SITE_HAS_Q, box_length, water_box)

RC, SWITCH, ETA, SKIN, REBUILD = 9.0, 1.0, 0.35, 1.5, 10
STEPS = 10  # dynamics steps per pass


def listed():
    return [
        # the smallest box in use: a k-sum evaluation per step from host arrays
        dict(name="host_fp64_ksum_216", kind="host", system="water", size=216, precision="fp64", kcut=7.0),
        # the per-step host call of a program that keeps its own integrator
        dict(name="host_mixed_4096", kind="host", system="water", size=4096, precision="mixed", spacing=1.04, order=5),
        # the headline box, positions resident on the device, in both forms
        dict(name="device_mixed_32768", kind="device", system="water", size=32768, precision="mixed", spacing=1.04,
             order=5),
        dict(name="device_fp64_32768", kind="device", system="water", size=32768, precision="fp64", spacing=1.04,
             order=5),
        # molecules in water: groups of two to four sites, exclusions across
        # groups and scaled 1-4 pairs, an odd total
        dict(name="device_fp64_solution_17", kind="device", system="solution", size=17, precision="fp64",
             spacing=1.04, order=5),
        dict(name="device_mixed_solution_32", kind="device", system="solution", size=32, precision="mixed",
             spacing=1.04, order=5),
        # dynamics of a medium box in plain FP64
        dict(name="md_fp64_4096", kind="md", system="water", size=4096, precision="fp64", spacing=1.04, order=5),
        # replica exchange: twelve boxes of 256 to 4096 waters advanced together
        dict(name="batch_mixed_12", kind="batch", system="water", size=12, precision="mixed", spacing=1.04, order=5),
        # one frame of a force-matching fit on the 512-water box
        dict(name="fit_fp64_512", kind="fit", system="water", size=512, precision="fp64", spacing=1.04, order=5),
        # one sweep of a charge solve on the default mesh
        dict(name="charges_fp64_1331", kind="charges", system="water", size=1331, precision="fp64", spacing=0.5,
             order=3),
        # the pressure of a medium box with mesh differentiation by ik
        dict(name="virial_mixed_ik_6000", kind="virial", system="water", size=6000, precision="mixed", spacing=1.04,
             order=4, ik=True),
        # a potential grid around the sites of a medium box
        dict(name="points_fp64_4096", kind="points", system="water", size=4096, precision="fp64", npoint=5000,
             kcut=6.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "host", "device", "device", "device", "md", "batch", "fit", "charges", "virial",
                       "points"])
    c = dict(kind=kind, system="water", precision=rng.choice(["fp64", "mixed"]))
    c["spacing"] = round(rng.uniform(0.8, 1.2), 3)
    c["order"] = rng.choice([3, 4, 5, 5, 5, 6])
    if kind == "host":
        if rng.random() < 0.4:
            # the k-sum is for small boxes
            c.update(size=_log_int(rng, 216, 1000), kcut=float(rng.randint(5, 8)))
            del c["spacing"], c["order"]
        else:
            c["size"] = _log_int(rng, 216, 32768)
    elif kind == "device":
        if rng.random() < 0.4:
            c.update(system="solution", size=rng.randint(8, 32))
        else:
            c["size"] = _log_int(rng, 216, 32768)
    elif kind == "md":
        c["size"] = _log_int(rng, 216, 8192)
    elif kind == "batch":
        c["size"] = rng.randint(2, 12)
    elif kind == "fit":
        c["size"] = _log_int(rng, 216, 4096)
    elif kind == "charges":
        c.update(size=_log_int(rng, 216, 4096), spacing=round(rng.uniform(0.5, 1.1), 3))
    elif kind == "virial":
        c.update(size=_log_int(rng, 216, 8192), ik=rng.random() < 0.4)
    else:
        c.update(size=_log_int(rng, 216, 4096), npoint=_log_int(rng, 500, 5000), kcut=float(rng.randint(4, 7)))
        del c["spacing"], c["order"]
    return c


# ---- systems -----------------------------------------------------------------

class Solution:
    """Water and a six-site solute ([C, H, H, H] and [O, H]) on an n^3 water
    lattice; a solute takes two cells that follow one another along z."""

    # body frame, C-O along z, its middle at the origin; charges in e
    BODY = np.array([[0, 0, -0.715], [1.028, 0, -1.079], [-0.514, 0.890, -1.079], [-0.514, -0.890, -1.079],
                     [0, 0, 0.715], [0.896, 0, 1.017]])
    CHARGE = np.array([0.145, 0.04, 0.04, 0.04, -0.683, 0.418])
    SIGMA = np.array([3.5, 2.5, 2.5, 2.5, 3.12, 0.0])
    EPSILON = np.array([0.066, 0.03, 0.03, 0.03, 0.17, 0.0])
    MASS = np.array([12.011, MASS_H, MASS_H, MASS_H, MASS_O, MASS_H])
    EXCLUDED = np.array([[0, 1], [0, 2], [0, 3], [1, 2], [1, 3], [2, 3], [0, 4], [1, 4], [2, 4], [3, 4], [0, 5],
                         [4, 5]])
    FOURTH = np.array([[1, 5], [2, 5], [3, 5]])

    def __init__(self, n, seed):
        rng = np.random.default_rng(seed)
        wb = water_box(n, seed)
        self.box = wb.box
        step = wb.box / n
        water = wb.positions.reshape(n, n, n, 3, 3)
        taken = np.zeros((n, n, n), dtype=bool)
        # a quarter of every other column's pairs: no two solutes side by side
        x, y = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
        column = ((x + y) % 2 == 0) & (x < n - n % 2) & (y < n - n % 2)
        pairs = np.argwhere((rng.random((n, n, n // 2)) < 0.25) & column[:, :, None])
        taken[pairs[:, 0], pairs[:, 1], 2 * pairs[:, 2]] = True
        taken[pairs[:, 0], pairs[:, 1], 2 * pairs[:, 2] + 1] = True
        w = water[~taken]
        nw, ns = len(w), len(pairs)
        a = rng.uniform(0, 2 * np.pi, ns)
        flip = rng.choice([-1.0, 1.0], ns)
        rot = np.zeros((ns, 3, 3))
        rot[:, 0, 0], rot[:, 0, 1] = np.cos(a), -np.sin(a) * flip
        rot[:, 1, 0], rot[:, 1, 1] = np.sin(a), np.cos(a) * flip
        rot[:, 2, 2] = flip
        mid = (pairs * np.array([1, 1, 2]) + np.array([0.5, 0.5, 1.0])) * step
        s = mid[:, None, :] + np.einsum("nij,sj->nsi", rot, self.BODY)
        self.positions = np.concatenate([w.reshape(-1, 3), s.reshape(-1, 3)])
        self.nsite = len(self.positions)
        o, b = 3 * np.arange(nw), 3 * nw + 6 * np.arange(ns)
        g = np.concatenate([np.stack([o, o + 3], 1), np.stack([b, b + 4, b + 4, b + 6], 1).reshape(-1, 2)])
        self.groups = g.astype(np.int32)
        we = np.array([[0, 1], [0, 2], [1, 2]])
        self.exclusions = np.concatenate([(o[:, None, None] + we).reshape(-1, 2),
                                          (b[:, None, None] + self.EXCLUDED).reshape(-1, 2)]).astype(np.int32)
        self.pairs14 = (b[:, None, None] + self.FOURTH).reshape(-1, 2).astype(np.int32)

        def per_site(w3, s6):
            return np.concatenate([np.tile(np.asarray(w3, dtype=np.float64), nw), np.tile(s6, ns)])

        self.q = e_to_charge_unit(per_site([-0.8476, 0.4238, 0.4238], self.CHARGE))
        self.sigma = per_site([SIGMA_O, 0, 0], self.SIGMA)
        self.epsilon = per_site([EPSILON_O, 0, 0], self.EPSILON)
        self.rscreen = np.zeros(self.nsite)
        self.site_mask = np.where(self.sigma > 0, SITE_HAS_Q | SITE_HAS_LJ, SITE_HAS_Q).astype(np.int32)
        self.masses = per_site([MASS_O, MASS_H, MASS_H], self.MASS)


def _system(case, seed):
    """The case's system, its molecules off their lattice points by up to 0.15 A."""
    if case["system"] == "solution":
        s = Solution(case["size"], seed)
    else:
        s = water_box_n(case["size"], seed)
        s.pairs14 = None
    jitter = np.random.default_rng(seed + 1).uniform(-0.15, 0.15, (len(s.groups), 3))
    if case["system"] == "solution":
        nw = int(np.sum(s.groups[:, 1] - s.groups[:, 0] == 3))
        jitter[nw + 1::2] = jitter[nw::2]  # a solute's two groups move together
    s.positions = s.positions + np.repeat(jitter, s.groups[:, 1] - s.groups[:, 0], axis=0)
    return s


def _settings(case):
    d = dict(precision=case["precision"], rspace_cutoff=RC, smoothing_width=SWITCH, ewald_screening=ETA,
             neighbor_list_width=SKIN, rebuild_interval=REBUILD)
    if "kcut" in case:
        d["kspace_cutoff"] = case["kcut"]
    if "order" in case:
        d.update(use_p3m=True, p3m_grid_spacing=case["spacing"], p3m_assignment_order=case["order"],
                 p3m_ik_differentiate=bool(case.get("ik", False)))
    if case["system"] == "solution":
        d.update(elec_1_4_scale_factor=0.5, lj_1_4_scale_factor=0.5)
    return d


# ---- preparing and running ---------------------------------------------------

_work_stream = None


def _stream():
    """The one stream the program evaluates on."""
    global _work_stream
    if _work_stream is None:
        _work_stream = torch.cuda.Stream()
    return _work_stream


def _replicas(case, seed):
    sizes = replica_sizes(case["size"])
    temps = temperature_ladder(case["size"])
    for k, n in enumerate(sizes):
        yield _system(dict(case, size=int(n)), 1000 * seed + k), temps[k]


def _loss_gradient(n, seed):
    """dL/dF of a force-matching loss: twice a force difference of a few percent."""
    return np.random.default_rng(seed + 2).normal(scale=1.0, size=(n, 3))


def _charges(s, seed):
    """Charges that a sweep has arrived at: the model's, each water's shifted."""
    d = np.random.default_rng(seed + 3).normal(scale=0.02, size=(s.nsite // 3, 2))
    return s.q + e_to_charge_unit(np.column_stack([d.sum(1), -d[:, 0], -d[:, 1]]).reshape(-1))


def _points(s, case, seed):
    return np.random.default_rng(seed + 4).uniform(0, s.box, size=(case["npoint"], 3))


class State:
    pass


_open = []  # a program's potentials and integrators stay open until it ends


def prepare(case, seed):
    st = State()
    _open.append(st)
    st.case = case
    kind = case["kind"]
    if kind == "batch":
        st.pots, st.mds = [], []
        for k, (s, t) in enumerate(_replicas(case, seed)):
            pot = ElecLJ(**_settings(case)).init(s)
            md = MDyn(pot, s.masses, timestep=0.002)
            md.set_state(s.positions, maxwell_boltzmann(s, t, seed=seed + k))
            st.pots.append(pot)
            st.mds.append(md)
        st.batch = ReplicaBatch(st.mds)
        return st
    s = _system(case, seed)
    st.pot = ElecLJ(**_settings(case)).init(s, pairs14=s.pairs14)
    st.sys = s
    st.r = np.ascontiguousarray(s.positions)
    if kind == "host":
        st.r = torch.from_numpy(st.r).pin_memory().numpy()
        st.f = np.zeros((s.nsite, 3))
    elif kind == "device":
        st.pot.set_stream(_stream().cuda_stream)
        st.pot.compute(st.r)
        st.d_r = torch.from_numpy(st.r).cuda()
        st.d_f = torch.zeros(s.nsite, 3, dtype=torch.float64, device="cuda")
        st.d_e = torch.zeros(4, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        st.pot.graph_capture(st.d_r.data_ptr(), st.d_f.data_ptr(), st.d_e.data_ptr())
        st.f32 = torch.zeros(s.nsite, 3, device="cuda")
        st.e32 = torch.zeros(4, device="cuda")
        torch.cuda.synchronize()
    elif kind == "md":
        st.md = MDyn(st.pot, s.masses, timestep=0.002)
        st.md.set_state(st.r, maxwell_boltzmann(s, 300.0, seed=seed))
    elif kind == "fit":
        st.g = _loss_gradient(s.nsite, seed)
    elif kind == "charges":
        st.q = _charges(s, seed)
    elif kind == "points":
        st.points = _points(s, case, seed)
    return st


def _kept(x, case):
    """A result as the program keeps it: float32 with the mixed form."""
    if case["precision"] == "fp64":
        return x
    if isinstance(x, dict):
        return {k: _kept(v, case) for k, v in x.items()}
    return np.float32(x) if isinstance(x, float) else x.astype(np.float32)


def _energies(d):
    """The energies of a result as one record: charges and molecules close to
    neutral make any one of them nearly cancel."""
    return np.array([d["elec"], d["lj"], d["lj_correction"], d["total"]])


def run(st):
    case, kind = st.case, st.case["kind"]
    if kind == "host":
        st.f.fill(0.0)
        u = st.pot.add_to_energy_and_forces(0.0, st.f, st.r)
        return _kept(dict(f=st.f, e=_energies(dict(st.pot.energy, total=u))), case)
    if kind == "device":
        with torch.cuda.stream(_stream()):
            st.d_f.zero_()
            st.pot.graph_launch()
            if case["precision"] == "fp64":
                return dict(f=st.d_f, e=st.d_e)
            st.f32.copy_(st.d_f)
            st.e32.copy_(st.d_e)
            return dict(f=st.f32, e=st.e32)
    if kind == "md":
        e = st.md.run(STEPS)
        r, v = st.md.state()
        return _kept(dict(e=e, r=r, v=v), case)
    if kind == "batch":
        return [[_kept(x, case) for x in (e, *md.state())] for e, md in zip(st.batch.run(STEPS), st.mds)]
    if kind == "fit":
        out = st.pot.forward(st.r)
        return _kept(dict(f=out["f"], e=_energies(out), **st.pot.site_gradients(st.g)), case)
    if kind == "charges":
        s = st.sys
        st.pot.set_params(s.site_mask, st.q, s.sigma, s.epsilon, s.rscreen)
        out = st.pot.compute(st.r, want_fields=True)
        return _kept(dict(f=out["f"], phi=out["phi"], evec=out["evec"], e=_energies(out)), case)
    if kind == "virial":
        w, e, f = st.pot.virial(st.r, st.sys.masses)
        return _kept(dict(w=w, e=_energies(e), f=f), case)
    return st.pot.electrostatic_potential_at_gridpoints(st.r, st.points)


# ---- the work a pass cannot do without ---------------------------------------

def _sites(case):
    """(groups, sites, site pairs of a group pair, of them with LJ) of the case's system."""
    if case["system"] == "solution":
        n = case["size"]
        pairs = 0.125 * n * n * (n // 2)
        nw = n ** 3 - 2 * pairs
        groups, sites = nw + 2 * pairs, 3 * nw + 6 * pairs
        per = sites / groups
        return groups, sites, per * per, ((nw + 5 * pairs) / groups) ** 2
    return case["size"], 3 * case["size"], 9.0, 1.0


def _evaluation(case):
    groups, sites, per, lj = _sites(case)
    box = box_length(groups)
    pairs = groups / 2 * (4 / 3 * math.pi * RC ** 3) * groups / box ** 3
    flops = pairs * (40 * per + 20 * lj + 30)
    if "order" in case:
        m = (box / case["spacing"]) ** 3
        ik = 4 if case.get("ik") else 1
        flops += sites * case["order"] ** 3 * (2 + 8) + (1 + ik) * 2.5 * m * math.log2(m)
    elif case["kind"] == "host":
        # a structure factor and a field sum: a sine and a cosine each
        flops += 2 * math.pi / 3 * case["kcut"] ** 3 * sites * 2 * 30
    # positions, charge and LJ parameters read, force and potential written
    return sites * (24 + 24 + 24 + 8), flops


def work(case):
    kind = case["kind"]
    if kind == "batch":
        # sizes log-uniform on [256, 4096]
        b, f = _evaluation(dict(case, size=int(3840 / math.log(16))))
        return dict(bytes=STEPS * case["size"] * 2.2 * b, flops=STEPS * case["size"] * f)
    if kind == "points":
        groups, sites, _, _ = _sites(case)
        near = (4 / 3 * math.pi * RC ** 3) * sites / box_length(groups) ** 3
        nk = 2 * math.pi / 3 * case["kcut"] ** 3
        return dict(bytes=sites * 32 + case["npoint"] * 32,
                    flops=case["npoint"] * near * 25 + nk * (sites + case["npoint"]) * 30)
    b, f = _evaluation(case)
    if kind == "md":
        return dict(bytes=STEPS * 2.2 * b, flops=STEPS * f)
    if kind == "fit":
        return dict(bytes=2.2 * b, flops=2.5 * f)
    return dict(bytes=b, flops=f)


# ---- the same numbers in plain 64-bit torch ----------------------------------

def _anchor_pairs(anchor, box):
    """Unordered anchor pairs within the cutoff and their lattice shifts (integers)."""
    n = len(anchor)
    out = []
    rows = max(1, (1 << 25) // n)
    idx = torch.arange(n, device=anchor.device)
    for a in range(0, n, rows):
        d = anchor[a:a + rows, None, :] - anchor[None, :, :]
        d -= box * torch.floor(d / box + 0.5)
        ok = ((d * d).sum(-1) <= RC * RC) & (idx[None, :] > idx[a:a + rows, None])
        i, j = ok.nonzero(as_tuple=True)
        out.append(torch.stack([i + a, j]))
    ij = torch.cat(out, 1)
    d = anchor[ij[0]] - anchor[ij[1]]
    return ij[0], ij[1], -torch.floor(d / box + 0.5)


def _switch(r2):
    z = ((r2 - (RC - SWITCH) ** 2) / (RC ** 2 - (RC - SWITCH) ** 2)).clamp(min=0)
    return 1 + z ** 3 * (-10 + z * (15 - 6 * z))


def _spline(x, order):
    """Cardinal B-spline weights: first mesh point and (n, order) weights."""
    if order % 2:
        j = torch.floor(x.detach() + 0.5)
        w = x - j + 0.5
    else:
        j = torch.floor(x.detach())
        w = x - j
    m = [torch.ones_like(w)]
    for k in range(2, order + 1):
        zero = torch.zeros_like(w)
        prev = [zero] + m + [zero]
        m = [((w + i) * prev[i + 1] + (k - w - i) * prev[i]) / (k - 1) for i in range(k)]
    return j.long() - ((order + 1) // 2 - 1), torch.stack(m[::-1], -1)


def _influence(mesh, box, order, ik, dev):
    """The optimal influence function (alias sums over |p| <= 2) and the wave vectors."""
    j = [torch.fft.fftfreq(mesh, 1 / mesh, device=dev, dtype=torch.float64)] * 2
    j.append(torch.fft.rfftfreq(mesh, 1 / mesh, device=dev, dtype=torch.float64))
    j = [torch.where(x == -mesh / 2, -x, x) for x in j]
    shape = [(-1, 1, 1), (1, -1, 1), (1, 1, -1)]
    k = [2 * math.pi / box * x.reshape(s) for x, s in zip(j, shape)]
    num = d1 = d2 = 0.0
    for p in itertools.product(range(-2, 3), repeat=3):
        kp = [2 * math.pi / box * (x + q * mesh).reshape(s) for x, q, s in zip(j, p, shape)]
        u2 = 1.0
        for x, q, s in zip(j, p, shape):
            u2 = u2 * torch.sinc(x / mesh + q).pow(2 * order).reshape(s)
        kp2 = kp[0] ** 2 + kp[1] ** 2 + kp[2] ** 2
        zero = kp2 == 0
        g = torch.where(zero, 0.0, 4 * math.pi / torch.where(zero, 1.0, kp2) * torch.exp(-kp2 / (4 * ETA ** 2)))
        u2 = torch.where(zero, 0.0, u2)
        if ik:
            num = num + g * u2 * sum(a * b for a, b in zip(k, kp))
            d1 = d1 + u2
        else:
            num = num + g * kp2 * u2
            d1, d2 = d1 + u2, d2 + u2 * kp2
    den = d1 * d1 * sum(x * x for x in k) if ik else d1 * d2
    den[0, 0, 0] = 1.0
    num[0, 0, 0] = 0.0
    return num / den / box ** 3, k


def _mesh_size(box, spacing):
    x = math.floor(box / spacing + 0.5)
    best = 1
    cand = sorted({a * b * c * d for a in (2 ** i for i in range(10)) for b in (3 ** i for i in range(7))
                   for c in (5 ** i for i in range(5)) for d in (7 ** i for i in range(4))})
    for v in cand:
        if v <= x and abs(x - v) < abs(x - best):
            best = v
    return best


class Exact:
    """The energy of a system as a function of its positions, charges, LJ
    parameters and a box scale, in plain 64-bit torch."""

    def __init__(self, s, case, dev="cuda"):
        t = lambda x, d=torch.float64: torch.as_tensor(np.array(x), dtype=d, device=dev)  # noqa: E731
        self.case, self.dev, self.box = case, dev, float(s.box)
        self.r, self.q = t(s.positions), t(s.q)
        self.sigma, self.epsilon = t(s.sigma), t(s.epsilon)
        self.has_lj = t((s.site_mask & SITE_HAS_LJ) != 0, torch.bool)
        self.excl = t(np.sort(s.exclusions, axis=1), torch.int64)
        p14 = s.pairs14 if s.pairs14 is not None else np.zeros((0, 2))
        self.p14 = t(p14, torch.int64)
        g = t(s.groups, torch.int64)
        width = int((g[:, 1] - g[:, 0]).max())
        site = g[:, :1] + torch.arange(width, device=dev)
        live = site < g[:, 1:]
        self.anchor = g[:, 0]
        i, j, self.shift = _anchor_pairs(self.r[self.anchor], self.box)
        self.ai, self.aj = self.anchor[i], self.anchor[j]
        self.si = site[i][:, :, None].expand(-1, width, width).reshape(-1)
        self.sj = site[j][:, None, :].expand(-1, width, width).reshape(-1)
        ok = (live[i][:, :, None] & live[j][:, None, :]).reshape(-1)
        pair = torch.arange(len(i), device=dev).repeat_interleave(width * width)
        n = len(self.r)
        ex = torch.unique(self.excl[:, 0] * n + self.excl[:, 1])
        self.excl = torch.stack([ex // n, ex % n], 1)
        key = torch.minimum(self.si, self.sj) * n + torch.maximum(self.si, self.sj)
        at = torch.searchsorted(ex, key).clamp(max=len(ex) - 1)
        ok &= ex[at] != key
        self.si, self.sj, self.pair = self.si[ok], self.sj[ok], pair[ok]
        self.lj = (self.has_lj[self.si] & self.has_lj[self.sj]).nonzero().squeeze(1)

    def _lj(self, i, j, r2, sigma, epsilon):
        s6 = (0.25 * (sigma[i] + sigma[j]) ** 2 / r2) ** 3
        return 4 * torch.sqrt(epsilon[i] * epsilon[j]) * (s6 * s6 - s6)

    def _near(self, r, i, j, box):
        d = r[i] - r[j]
        d = d - box * torch.floor((d / box).detach() + 0.5)
        return (d * d).sum(-1)

    def tail(self, sigma, epsilon, box):
        """2 pi / V sum_ab n_a n_b int (1 - S) u_ab r^2 dr, by quadrature."""
        sg, ep = sigma[self.has_lj], epsilon[self.has_lj]
        cls, of = torch.unique(torch.stack([sg, ep], 1).detach(), dim=0, return_inverse=True)
        cnt = torch.zeros(len(cls), dtype=torch.float64, device=self.dev).index_add_(0, of, torch.ones_like(sg))
        # each class at the mean of its sites, so that its sites share its derivative
        sg, ep = (torch.zeros_like(cnt).index_add(0, of, x) / cnt for x in (sg, ep))
        x, w = np.polynomial.legendre.leggauss(64)
        rr = torch.as_tensor(RC - SWITCH + SWITCH * (x + 1) / 2, device=self.dev)
        ww = torch.as_tensor(w * SWITCH / 2, device=self.dev) * (1 - _switch(rr * rr)) * rr * rr
        i12 = (ww * rr ** -12).sum() + RC ** -9 / 9
        i6 = (ww * rr ** -6).sum() + RC ** -3 / 3
        s6 = (0.5 * (sg[:, None] + sg[None, :])) ** 6
        e = 4 * torch.sqrt(ep[:, None] * ep[None, :]) * cnt[:, None] * cnt[None, :]
        return 2 * math.pi / box ** 3 * (e * (s6 * s6 * i12 - s6 * i6)).sum()

    def mesh(self, r, q, scale):
        """Site potential on the P3M mesh and, with ik, the site field."""
        case, box = self.case, self.box * scale
        m, order, ik = _mesh_size(self.box, case["spacing"]), case["order"], bool(case.get("ik", False))
        base, w = _spline(r * (m / box), order)
        idx = torch.remainder(base[..., None] + torch.arange(order, device=self.dev), m)
        at = ((idx[:, 0, :, None, None] * m + idx[:, 1, None, :, None]) * m + idx[:, 2, None, None, :]).reshape(-1)
        ww = (w[:, 0, :, None, None] * w[:, 1, None, :, None] * w[:, 2, None, None, :]).reshape(len(r), -1)
        rho = torch.zeros(m ** 3, dtype=torch.float64, device=self.dev)
        rho = rho.index_add(0, at, (ww * q[:, None]).reshape(-1)).reshape(m, m, m)
        g, k = _influence(m, self.box, order, ik, self.dev)
        spec = torch.fft.rfftn(rho) * (g / scale)
        back = lambda x: (torch.fft.irfftn(x, (m, m, m), norm="forward").reshape(-1)[at].reshape(ww.shape) * ww).sum(1)  # noqa: E731
        return back(spec), torch.stack([back(-1j * kd / scale * spec) for kd in k], 1) if ik else None

    def waves(self):
        kc = self.case["kcut"]
        n = int(kc)
        half = [v for v in itertools.product(range(n + 1), range(-n, n + 1), range(-n, n + 1))
                if v > (0, 0, 0) and sum(x * x for x in v) <= kc * kc + 1e-8]
        k = 2 * math.pi / self.box * torch.tensor(half, dtype=torch.float64, device=self.dev)
        k2 = (k * k).sum(1)
        return k, 4 * math.pi / self.box ** 3 * torch.exp(-k2 / (4 * ETA ** 2)) / k2

    def energy(self, r=None, q=None, sigma=None, epsilon=None, scale=1.0, fixed_switch=False):
        """(electrostatic, LJ pairs, LJ tail, site field of the ik mesh or None)"""
        r = self.r if r is None else r
        q = self.q if q is None else q
        sigma = self.sigma if sigma is None else sigma
        epsilon = self.epsilon if epsilon is None else epsilon
        box, eta = self.box * scale, ETA / scale
        da = r[self.ai] - r[self.aj] + self.shift * box
        sw = _switch((da * da).sum(-1))
        if fixed_switch:
            sw = sw.detach()
        d = r[self.si] - r[self.sj] + (self.shift * box)[self.pair]
        r2 = (d * d).sum(-1)
        rr = torch.sqrt(r2)
        elec = (q[self.si] * q[self.sj] * torch.special.erfc(eta * rr) / rr * sw[self.pair]).sum()
        k = self.lj
        lj = (self._lj(self.si[k], self.sj[k], r2[k], sigma, epsilon) * sw[self.pair[k]]).sum()
        i, j = self.excl.unbind(1)
        re = torch.sqrt(self._near(r, i, j, box))
        elec = elec - (q[i] * q[j] * torch.special.erf(eta * re) / re).sum()
        if len(self.p14):
            i, j = self.p14.unbind(1)
            x2 = self._near(r, i, j, box)
            elec = elec - 0.5 * (q[i] * q[j] / torch.sqrt(x2)).sum()
            m = self.has_lj[i] & self.has_lj[j]
            lj = lj - 0.5 * self._lj(i[m], j[m], x2[m], sigma, epsilon).sum()
        field = None
        if "order" in self.case:
            phi, field = self.mesh(r, q, scale)
            elec = elec + 0.5 * (q * phi).sum()
        else:
            k, a = self.waves()
            x = r @ k.T
            elec = elec + (a * ((q @ torch.cos(x)) ** 2 + (q @ torch.sin(x)) ** 2)).sum()
        elec = elec - eta / math.sqrt(math.pi) * (q * q).sum() - math.pi / (2 * eta ** 2 * box ** 3) * q.sum() ** 2
        return elec, lj, self.tail(sigma, epsilon, box), field

    def forces(self, **kw):
        """(forces, elec, LJ pairs, tail); the ik mesh's force is charge times
        its site field, every other term's the gradient of its energy."""
        r = self.r.clone().requires_grad_()
        elec, lj, tail, field = self.energy(r=r, **kw)
        u = elec + lj
        if field is None:
            f = -torch.autograd.grad(u, r)[0]
        else:
            q = kw.get("q", self.q)
            mesh = 0.5 * (q * self.mesh(r, q, 1.0)[0]).sum()
            f = -torch.autograd.grad(u - mesh, r)[0] + (q[:, None] * field).detach()
        return f, float(elec.detach()), float(lj.detach()), float(tail.detach())

    def potential_at(self, pts):
        p = torch.as_tensor(pts, dtype=torch.float64, device=self.dev)
        out = []
        for a in range(0, len(p), 1000):
            d = self.r[None, :, :] - p[a:a + 1000, None, :]
            d -= self.box * torch.floor(d / self.box + 0.5)
            r2 = (d * d).sum(-1)
            rr = torch.sqrt(r2)
            out.append((torch.where(r2 <= RC * RC, torch.special.erfc(ETA * rr) / rr * _switch(r2), 0.0) * self.q).sum(1))
        k, a = self.waves()
        x, y = self.r @ k.T, p @ k.T
        c, s = self.q @ torch.cos(x), self.q @ torch.sin(x)
        return torch.cat(out) + 2 * (a * (c * torch.cos(y) + s * torch.sin(y))).sum(1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("md", "batch"):
        return None  # ten steps of dynamics
    s = _system(case, seed)
    x = Exact(s, case)
    if kind == "points":
        return x.potential_at(_points(s, case, seed)).cpu().numpy()

    def record(elec, lj, tail):
        return np.array([elec, lj + tail, tail, elec + lj + tail])

    if kind in ("host", "device"):
        f, elec, lj, tail = x.forces()
        return dict(f=f.cpu().numpy(), e=record(elec, lj, tail))
    if kind == "charges":
        q = torch.as_tensor(_charges(s, seed), device=x.dev).requires_grad_()
        elec = x.energy(q=q)[0]
        phi = torch.autograd.grad(elec, q)[0]
        q = q.detach()
        r = x.r.clone().requires_grad_()
        e = -torch.autograd.grad(x.energy(r=r, q=q, fixed_switch=True)[0], r)[0] / q[:, None]
        f, elec, lj, tail = x.forces(q=q)
        return dict(f=f.cpu().numpy(), phi=phi.cpu().numpy(), evec=e.cpu().numpy(),
                    e=record(elec, lj, tail))
    if kind == "virial":
        f, elec, lj, tail = x.forces()
        g = torch.as_tensor(np.array(s.groups), dtype=torch.int64, device=x.dev)
        mol = torch.repeat_interleave(torch.arange(len(g), device=x.dev), g[:, 1] - g[:, 0])
        m = torch.as_tensor(s.masses, device=x.dev)
        com = torch.zeros(len(g), 3, dtype=torch.float64, device=x.dev).index_add(0, mol, m[:, None] * x.r)
        com = com / torch.zeros(len(g), dtype=torch.float64, device=x.dev).index_add(0, mol, m)[:, None]
        scale = torch.ones((), dtype=torch.float64, device=x.dev).requires_grad_()
        u = sum(x.energy(r=x.r + (scale - 1) * com[mol], scale=scale)[:3])
        w = float(torch.autograd.grad(u, scale)[0])
        # with ik the mesh force is not the gradient of the mesh energy, and the
        # virial is built on the forces: no value for it here
        return dict(w=None if case.get("ik") else w, e=record(elec, lj, tail), f=f.cpu().numpy())
    r = x.r.clone().requires_grad_()
    par = [x.q.clone().requires_grad_(), x.sigma.clone().requires_grad_(), x.epsilon.clone().requires_grad_()]
    elec, lj, tail, _ = x.energy(r, *par)
    f = -torch.autograd.grad(elec + lj, r, create_graph=True)[0]
    g = torch.as_tensor(_loss_gradient(s.nsite, seed), device=x.dev)
    du = torch.autograd.grad(elec + lj + tail, par, retain_graph=True)
    dl = torch.autograd.grad((f * g).sum(), par)
    out = dict(f=f.detach().cpu().numpy(), e=record(float(elec.detach()), float(lj.detach()), float(tail.detach())))
    for name, a, b in zip(("dq", "dsig", "deps"), du, dl):
        live = torch.ones_like(x.has_lj) if name == "dq" else x.has_lj
        out["du_" + name] = torch.where(live, a, 0.0).cpu().numpy()
        out["dl_" + name] = torch.where(live, b, 0.0).cpu().numpy()
    return out
