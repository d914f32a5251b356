"""mmnb_site_gradients on a mesh whose transforms are the library's plans (98 has no two
radices), and after a first call whose set-up failed: a mixed-form handle makes the
dipole solve's meshes and plans on first use.

The loss is quartic in the charges, so the Richardson-extrapolated differences of the
oracle are exact to rounding; the bounds are those of the other gradient tests."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from molmodel_b200 import ElecLJ, _lib

from adjoint_cases import directional_fd, oracle_eval

MESH, SPACING = (28, 14, 98), 0.9


class Ions:
    def __init__(self, mesh, n=90, seed=2):
        rng = np.random.default_rng(seed)
        self.nsite, self.box = n, np.array(mesh) * SPACING
        self.positions = rng.uniform(0, 1, (n, 3)) * self.box
        self.groups = np.stack([np.arange(n), np.arange(n) + 1], 1)
        self.exclusions = np.zeros((0, 2), dtype=np.int64)
        self.site_mask = np.full(n, 1, dtype=np.int32)
        self.q = np.where(np.arange(n) % 2, 0.3, -0.3)
        self.sigma, self.epsilon, self.rscreen = np.zeros(n), np.zeros(n), np.zeros(n)
        self.pairs14 = None


def config(ik):
    return dict(rspace_cutoff=5.0, ewald_screening=0.5, use_p3m=True, p3m_grid_spacing=SPACING,
                p3m_assignment_order=4, p3m_ik_differentiate=ik)


def handle(s, ik, precision):
    return ElecLJ(precision=precision, **config(ik)).init(s, bctype=_lib.MMNB_ORTHORHOMBIC)


@pytest.mark.gpu
@pytest.mark.parametrize("ik", [False, True])
def test_gradients_on_a_mesh_of_the_librarys_plans(ik):
    s = Ions(MESH)
    cfg = dict(config(ik), bctype=_lib.MMNB_ORTHORHOMBIC)
    targets = oracle_eval(s, cfg, q=s.q * 1.05)["f"]
    v = np.random.default_rng(4).normal(size=s.nsite)
    fd_u, fd_l = directional_fd(s, cfg, "q", v, 1e-3, targets)
    p = handle(s, ik, "fp64")
    assert p.settings()["mesh"] == MESH
    dl_df = 2 * (p.forward(s.positions)["f"] - targets)
    g64 = p.site_gradients(dl_df)
    assert abs(v @ g64["du_dq"] - fd_u) <= 3e-8 * abs(fd_u) + 1e-9
    assert abs(v @ g64["dl_dq"] - fd_l) <= 3e-8 * abs(fd_l) + 1e-9
    m = handle(s, ik, "mixed")
    m.forward(s.positions)
    gm = m.site_gradients(dl_df)
    for key in ("du_dq", "dl_dq"):
        assert np.abs(gm[key] - g64[key]).max() <= 2e-5 * np.abs(g64[key]).max(), key


# cufftPlan3d in front of the library's: the next `plan_skip` calls pass, then
# `plan_failures` return "allocation failed"
SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
int plan_skip = 0, plan_failures = 0;
int cufftPlan3d(int *plan, int nx, int ny, int nz, int type)
{
  static int (*real)(int *, int, int, int, int);
  if (plan_skip > 0)
    plan_skip--;
  else if (plan_failures > 0) {
    plan_failures--;
    return 2;
  }
  if (!real)
    real = (int (*)(int *, int, int, int, int)) dlsym(dlopen("libcufft.so.11", RTLD_LAZY | RTLD_NOLOAD), "cufftPlan3d");
  return real(plan, nx, ny, nz, type);
}
"""


def failing_setup(shim, mesh, ik, skip):
    """Child process: the first two gradient calls' set-up fails, the third's does not."""
    import ctypes
    lib = ctypes.CDLL(shim, mode=ctypes.RTLD_GLOBAL)
    s = Ions(mesh)
    dl_df = np.random.default_rng(6).normal(size=(s.nsite, 3))
    p = handle(s, ik, "mixed")
    p.forward(s.positions)
    for _ in range(2):
        ctypes.c_int.in_dll(lib, "plan_skip").value = skip
        ctypes.c_int.in_dll(lib, "plan_failures").value = 1
        with pytest.raises(_lib.MmnbError) as ex:
            p.site_gradients(dl_df)
        assert ex.value.status == 2, ex.value.status  # MMNB_ERR_CUDA
        assert ctypes.c_int.in_dll(lib, "plan_failures").value == 0
    got = p.site_gradients(dl_df)
    q = handle(s, ik, "mixed")  # never failed
    q.forward(s.positions)
    want = q.site_gradients(dl_df)
    for key in ("du_dq", "dl_dq"):  # (the FP64 dipole mesh is summed with atomic adds)
        assert np.abs(got[key] - want[key]).max() <= 1e-10 * np.abs(want[key]).max(), key


# plans: a mesh of the library's, both forms; ik on a mesh of the own transforms
@pytest.mark.gpu
@pytest.mark.parametrize("mesh,ik", [(MESH, False), (MESH, True), ((20, 18, 24), True)])
@pytest.mark.parametrize("skip", [0, 1])
def test_gradients_after_a_failed_setup(mesh, ik, skip, tmp_path):
    src, shim = tmp_path / "plans.c", tmp_path / "plans.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(shim), str(src), "-ldl"], check=True)
    code = ("import sys; sys.path[:0] = [%r, %r]; import test_gpu_adjoint_setup as t; t.failing_setup(%r, %r, %r, %r)"
            % (ROOT, os.path.join(ROOT, "tests"), str(shim), mesh, ik, skip))
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stdout + done.stderr
