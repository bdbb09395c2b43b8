"""Forms of the trace that only some rays or launches reach, against the FP64 oracle: hits are
compared bit for bit, per-primitive fluxes to 1e-4 (the tolerance of the parity tests)."""
import numpy as np
import pytest

from helios_gb300 import _hrt, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(hrt_lib):
    return _hrt.Context(0)


@pytest.mark.parametrize("div", [1, 3, 8])
def test_rays_through_edges_and_corners(gpu, oracle_mod, div):
    """Rays exactly through edges, corners and diagonals of patches and triangles, where an edge
    function is zero and FP64 decides it."""
    sc = scenes.tile_grid((0.0, 0.0, 0.0), (float(div), float(div)), (div, div), twosided=1)
    h = 0.5 * div
    v = np.array([[-h, -h, 1.0], [h, -h, 1.0], [h, h, 1.0], [-h, h, 1.0]])
    T = np.concatenate([sc.T, scenes.triangle_T(v[[0, 0]], v[[1, 2]], v[[2, 3]])])
    ty = np.concatenate([sc.ptype, [scenes.TRIANGLE] * 2]).astype(np.uint32)
    ts = np.ones(ty.size, np.int8)
    g = np.linspace(-h, h, 2 * div + 1)
    x, y = np.meshgrid(g, g)
    o = np.stack([x.ravel(), y.ravel(), np.full(x.size, 3.0)], 1)
    o = np.concatenate([o, o - [0.0, 0.0, 2.5], o - [0.0, 0.0, 6.0]]).astype(np.float32)
    d = np.tile([0.0, 0.0, -1.0], (o.shape[0], 1)).astype(np.float32)
    d[2 * x.size:] *= -1.0
    tilt = np.array([0.5, 0.25, -1.0], np.float32)  # exact in FP32, as are the origins it starts from
    o = np.concatenate([o, o[:x.size] - 2.0 * tilt])
    d = np.concatenate([d, np.tile(tilt, (x.size, 1))])
    gpu.update_geometry(T, ty, ts)
    gpu.build_accel()
    h1, t1, f1 = gpu.trace_rays(o, d)
    h2, t2, f2, _ = oracle_mod.OracleScene(T, ty, ts).trace(o, d)
    assert (h2 >= 0).any()
    assert np.array_equal(h1, h2) and np.array_equal(f1, f2)
    assert np.array_equal(t1[h1 >= 0], t2[h2 >= 0])
