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


@pytest.mark.parametrize("scale,offset", [(1e-3, 0.0), (1.0, 0.0), (1.0, 3.0e4), (1e4, 0.0)])
def test_wide_nodes_enclose_their_children(gpu, oracle_mod, scale, offset):
    """The quantised 4-wide nodes cull no accepted hit at small and large sizes and far from the
    origin of coordinates: fluxes and ray counts of a solve over them equal the oracle's."""
    from helios_gb300.radiation import Context, RadiationModel
    from helpers import run_oracle

    sc = scenes.mixed_canopy(700, 2.0, seed=5)
    T = sc.T.reshape(-1, 4, 4).astype(np.float64)
    T[:, :3, :] *= scale
    T[:, :2, 3] += offset
    ctx = Context()
    uu = ctx.addPrimitives(T.reshape(-1, 16).astype(np.float32), sc.ptype, sc.area * scale ** 2, sc.twosided)
    ctx.setPrimitiveData(uu, "reflectivity_SW", np.full(uu.size, 0.3))
    rad = RadiationModel(ctx)
    rad.addRadiationBand("SW")
    rad.disableEmission("SW")
    sun = rad.addCollimatedRadiationSource(scenes.sun_direction(40.0, 100.0))
    rad.setSourceFlux(sun, "SW", 500.0)
    rad.setDiffuseRadiationFlux("SW", 80.0)
    rad.setDirectRayCount("SW", 36)
    rad.setDiffuseRayCount("SW", 49)
    rad.setScatteringDepth("SW", 1)
    rad.setSeed(11)
    got = rad.runBand("SW").astype(np.float64)
    ref, st = run_oracle(rad, ["SW"], oracle_mod, seed=11)
    floor = 1e-3 * float(np.abs(ref).mean())
    assert float((np.abs(got - ref) / np.maximum(np.abs(ref), floor)).max()) <= 1e-4
    assert rad.last_stats["rays"] == st["rays"]
