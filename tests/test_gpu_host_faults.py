"""Faults on the host's side of a call, made by stand-ins for two CUDA runtime calls that are linked
in front of the real ones (tests/cpp/cuda_fakes.cpp): allocations that fail, and copies that read
their host arrays as late as the runtime may."""
import os
import subprocess
import sys

import numpy as np
import pytest

from helios_gb300 import _hrt, scenes

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def fake_lib_path(hrt_lib, tmp_path_factory):
    from helios_gb300 import build

    objs = [os.path.join(build.BUILD, os.path.splitext(s)[0] + ".o") for s in build.SOURCES]
    out = str(tmp_path_factory.mktemp("fakes") / "libhrt_fakes.so")
    r = subprocess.run([build.nvcc(), *build.ARCH, "-shared", "-o", out, *objs, os.path.join(ROOT, "tests", "cpp", "cuda_fakes.cpp"),
                        "-Xcompiler", "-fPIC", "-Xlinker", "--wrap=cudaMallocAsync", "-Xlinker",
                        "--wrap=cudaMemcpyAsync"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return out


@pytest.fixture
def fakes(fake_lib_path, monkeypatch):
    monkeypatch.setattr(_hrt, "_lib", None)
    lib = _hrt.load(fake_lib_path)
    lib.fake_fail_allocations.argtypes = [_hrt.C.c_size_t, _hrt.C.c_size_t]
    yield lib
    lib.fake_fail_allocations(0, 0)
    lib.fake_late_copies(0)


def _solve(n, sources, nb=1, **k):
    S = len(sources)
    d = {"band_launch": np.ones(nb, np.uint8), "sources": sources, "source_flux": np.full((S, nb), 300.0),
         "rho": np.full((S, n, nb), 0.3), "tau": np.full((S, n, nb), 0.2), "diffuse_flux": np.full(nb, 100.0),
         "direct_rays": np.full(nb, 400), "diffuse_rays": np.full(nb, 64), "depth": np.full(nb, 1),
         "emission": np.zeros(nb, np.uint8), "seed": 3}
    return dict(d, **k)


def _voxel_context():
    leaves = scenes.mixed_canopy(700, 1.0, seed=2, height=1.0)
    vox = scenes.voxel_grid((0.0, 0.0, 0.05), (1.3, 1.3, 1.0), (6, 5, 4), 1.5)
    c = _hrt.Context(0)
    c.update_geometry(np.concatenate([leaves.T, vox.T]), np.concatenate([leaves.ptype, vox.ptype]),
                      np.concatenate([leaves.twosided, vox.twosided]), None, (0.0, 0.0),
                      np.concatenate([np.zeros(leaves.n), vox.lad]))
    return c, leaves.n


@pytest.mark.parametrize("what", ["cells", "second tree", "sun cells", "sun entries", "sun frames"])
def test_optional_buffers_without_memory(fakes, what):
    """Buffers that a call can do without: the cells of a voxel lattice, the tree of the surfaces beside
    it, and the grids of a direct pass.  Without memory for them the call gives the same fluxes."""
    c, ns = _voxel_context()
    c.build_accel()
    n = c.n
    d = _solve(n, [{"type": 0, "position": (0.3, 0.2, 0.9)}])
    want = c.run_band(d).astype(np.float64)
    size = {"cells": 2 * 16 * 6 * 5 * 4, "second tree": 64 * (ns - 1 + 8), "sun cells": 8 * 8 * n, "sun entries": 8 * 16 * n,
            "sun frames": 32 * 384}
    sun = what.startswith("sun")  # cells are as large as the transforms: fail them from the solve on
    fakes.fake_fail_allocations(0 if sun else size[what], 0)
    c, _ = _voxel_context()
    c.build_accel()
    failed = fakes.fake_failed()
    fakes.fake_fail_allocations(size[what] if sun else 0, 0)
    got = c.run_band(d).astype(np.float64)
    assert failed + fakes.fake_failed() > 0
    assert np.all(np.abs(got - want) <= 2.4e-7 * np.abs(want))


@pytest.mark.parametrize("spare", [0, 1 << 30])
def test_server_grids_take_what_the_budget_leaves(fakes, spare):
    """With a budget of just the scene's footprint the server makes no grids of its suns, and with room it
    does (their allocation fails here, which changes nothing): the fluxes are those of the scene alone."""
    sc = scenes.mixed_canopy(4000, 2.0, seed=1)
    n = sc.n
    sun = (0.3, 0.2, 0.9)
    c = _hrt.Context(0)
    c.update_geometry(sc.T, sc.ptype, sc.twosided)
    c.build_accel()
    want = c.run_band(_solve(n, [{"type": 0, "position": sun}], direct_rays=np.array([100]))).astype(np.float64)
    fakes.fake_fail_allocations(8 * 16 * n, 0)  # the entries of one sun
    srv = _hrt.Server(device=0, workers=1, hbm_budget=n * (529 + 68) + (8 << 20) + spare)
    srv.add_scene(0, sc.T, sc.ptype, sc.twosided, np.full((n, 1), 0.3), np.full((n, 1), 0.2))
    srv.submit(0, 0, 0.0, [1], sun, [300.0], [100.0], 100, 64, 1, 3, keep=True)
    srv.start()
    srv.wait()
    got = srv.result(0, n)["flux"].reshape(n, 1).astype(np.float64)
    srv.close()
    assert (fakes.fake_failed() > 0) == (spare > 0)
    assert np.all(np.abs(got - want) <= 1e-5 * np.maximum(np.abs(want), 1e-3 * np.abs(want).mean()))


LATE = """
import sys
import numpy as np
sys.path.insert(0, {root!r})
sys.path.insert(0, {tests!r})
from helios_gb300 import _hrt
lib = _hrt.load({lib!r})
import test_gpu_host_faults as t
c, ns = t._voxel_context()
c.build_accel()
sources = [{{"type": k % 2, "position": (0.3 + 0.01 * k, 0.2, 0.9 + 6.0 * (k % 2)), "width": (0.3, 0.3)}} for k in range(6)]
rng = np.random.default_rng(1)
d = t._solve(c.n, sources, nb=2, direct_rays=np.full(2, 36), diffuse_peak=np.tile([0.0, 0.0, 1.0], (2, 1)),
             diffuse_ext=np.full(2, 0.4), diffuse_norm=np.full(2, 0.7), depth=np.array([1, 3]))
d["rho"][:, ns:] = rng.uniform(0.0, 0.5, (6, c.n - ns, 2))
sw = dict(sun_dir=rng.uniform(0.1, 1.0, (100, 3)), direct_flux=np.full((100, 1), 300.0),
          diffuse_flux=np.full((100, 1), 80.0), direct_rays=4, diffuse_rays=4, depth=1, seed=5)

def plain():
    sc = t.scenes.mixed_canopy(500, 2.0, seed=4)
    s = _hrt.Context(0)
    s.update_geometry(sc.T, sc.ptype, sc.twosided)
    s.build_accel()
    sw.update(rho=np.full((sc.n, 1), 0.3), tau=np.full((sc.n, 1), 0.2))
    return s

s = plain()
want, wsw = c.run_band(d).astype(np.float64), s.run_sweep(**sw).astype(np.float64)
c, ns = t._voxel_context()
c.build_accel()
s = plain()
lib.fake_late_copies(1)
got, gsw = c.run_band(d).astype(np.float64), s.run_sweep(**sw).astype(np.float64)
assert lib.fake_lates() > 0
lib.fake_late_copies(0)
err = lambda a, b: float((np.abs(a - b) / np.maximum(np.abs(b), 1e-3 * np.abs(b).mean())).max())
assert err(got, want) <= 1e-5 and err(gsw, wsw) <= 1e-5
"""


def test_host_arrays_outlive_their_copies(fake_lib_path):
    """Copies from pageable memory that read their source when the stream reaches them: every array of
    a solve or sweep is still there.  The C library fills freed memory (MALLOC_PERTURB_), so that an
    array freed before its copy gives other fluxes."""
    code = LATE.format(root=ROOT, tests=os.path.join(ROOT, "tests"), lib=fake_lib_path)
    env = dict(os.environ, MALLOC_PERTURB_="165", MALLOC_MMAP_THRESHOLD_=str(1 << 25), MALLOC_TRIM_THRESHOLD_=str(1 << 30),
               GLIBC_TUNABLES="glibc.malloc.tcache_count=0")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, env=env, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]
