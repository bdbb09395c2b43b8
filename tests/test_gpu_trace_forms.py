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


def _direct_model(kind, suns, periodic, rays=400, seed=3):
    """A direct-only solve of at least 0.2 M rays per source, so that collimated sources are binned."""
    from helios_gb300.radiation import Context, RadiationModel

    ctx = Context()
    if kind == "voxels":
        ctx.addScene(scenes.deep_scatter(n_tri=300, n_patch=150, n_disk=150, vox_div=4, domain=2.0, height=1.0, seed=seed))
    elif kind == "far":  # coordinates far larger than the scene
        sc = scenes.mixed_canopy(700, 2.0, seed=seed)
        T = sc.T.copy()
        T[:, [3, 7]] += 2.0e4
        ctx.addPrimitives(T, sc.ptype, sc.area, sc.twosided)
    elif kind == "wide":  # more wide primitives than a grid takes: the tree serves the source
        ctx.addScene(scenes.mixed_canopy(2000, 2.0, seed=seed))
        for k in range(40):
            ctx.addPatch((0.6, 0.7, 3.1 + 0.01 * k), (1.5, 1.4), (0.1, 0.2 * k))
    elif kind == "flat":  # one plane: no extent across a horizontal sun
        ctx.addScene(scenes.tile_grid((0.0, 0.0, 0.0), (4.0, 4.0), (24, 24), twosided=1))
    else:
        ctx.addScene(scenes.mixed_canopy(700, 2.0, seed=seed))
        if kind == "masks":
            mask = np.zeros((8, 8), np.uint8)
            mask[::2] = 1
            for k in range(30):
                ctx.addPatch((0.03 * k, 0.5, 3.2), (0.2, 0.2), (0.3, 0.1 * k), texture_mask=mask)
    rad = RadiationModel(ctx)
    if periodic:
        rad.enforcePeriodicBoundary("xy")
    rad.addRadiationBand("SW")
    rad.disableEmission("SW")
    for k, d in enumerate(suns):
        s = rad.addSphereRadiationSource((0.5, 0.5, 9.0), 0.3) if d is None else rad.addCollimatedRadiationSource(d)
        rad.setSourceFlux(s, "SW", 300.0 + 50.0 * k)
    rad.setDirectRayCount("SW", rays)
    rad.setDiffuseRayCount("SW", 1)
    rad.setSeed(seed)
    return rad


SUNS = [(0.3, -0.4, 0.8), (0.0, 0.0, 1.0), (1.0, 0.0, 0.0), (-0.2, 0.9, -0.3)]


@pytest.mark.parametrize("kind", ["mixed", "voxels", "masks", "far", "wide", "flat"])
@pytest.mark.parametrize("periodic", [False, True])
def test_binned_shadow_rays_equal_the_tree(hrt_lib, kind, periodic):
    """Shadow rays answered by the grid across the sun give the tree's sums: suns from above, along an
    axis and from below, a source that is no sun between them, over every primitive form.  A set
    visit budget sends all of them through the tree.  Strengths are summed in another order in FP64:
    FP32 fluxes agree to two units in the last place."""
    rad = _direct_model(kind, SUNS[:2] + [None] + SUNS[2:], periodic)
    binned = rad.runBand("SW").astype(np.float64)
    rays = rad.last_stats["rays"]
    rad.ctx.set_visit_budget(1 << 30)
    tree = rad.runBand("SW").astype(np.float64)
    assert (tree > 0).any()
    assert np.abs(binned - tree).max() <= 2.4e-7 * np.abs(tree).max()
    assert np.all(np.abs(binned - tree) <= 2.4e-7 * np.abs(tree))
    assert rad.last_stats["rays"] == rays
    rad.ctx.set_visit_budget(0)
    rad.ctx.set_launch_ray_limit(60000)  # several primitive chunks
    assert np.all(np.abs(rad.runBand("SW").astype(np.float64) - tree) <= 2.4e-7 * np.abs(tree))


@pytest.mark.parametrize("nsun", [1, 33])
def test_binned_sweep_equals_the_tree(gpu, nsun):
    """The sweep's suns in one batch and in two (more suns than a batch holds)."""
    sc = scenes.mixed_canopy(2100, 2.0, seed=4)
    rng = np.random.default_rng(1)
    d = scenes.uniform_sphere(rng, nsun).astype(np.float32)
    kw = dict(sun_dir=d, direct_flux=np.full((nsun, 1), 500.0), diffuse_flux=np.zeros((nsun, 1)),
              rho=np.full((sc.n, 1), 0.1), tau=np.full((sc.n, 1), 0.05), direct_rays=100, diffuse_rays=4, depth=0, seed=9)
    gpu.update_geometry(sc.T, sc.ptype, sc.twosided)
    gpu.build_accel()
    binned, rays = gpu.run_sweep(**kw), gpu.last_stats()["rays"]
    again = gpu.run_sweep(**kw)
    gpu.set_visit_budget(1 << 30)
    tree = gpu.run_sweep(**kw)
    gpu.set_visit_budget(0)
    assert gpu.last_stats()["rays"] == rays
    assert np.array_equal(binned, again)
    assert np.all(np.abs(binned - tree) <= 2.4e-7 * np.abs(tree))


@pytest.mark.parametrize("panes,voxels", [(1, False), (16, False), (20, False), (3, True)])
@pytest.mark.parametrize("depth", [0, 2])
def test_stacked_covers_vs_oracle(oracle_mod, panes, voxels, depth):
    """Rays through a stack of covers, up to and beyond the sixteen that a segment takes, with a sky
    (covers take deposits) and scattering (covers are passed by): fluxes of covers and leaves."""
    from helios_gb300.radiation import Context, RadiationModel
    from helpers import run_oracle

    ctx = Context()
    if voxels:
        ctx.addScene(scenes.deep_scatter(n_tri=100, n_patch=60, n_disk=60, vox_div=3, domain=1.0, height=1.0, seed=6))
    else:
        ctx.addScene(scenes.mixed_canopy(200, 2.0, seed=6, height=1.0))
    leaves = np.arange(1, ctx.getPrimitiveCount())
    for k in range(panes):
        u = ctx.addPatch((0.5, 0.5, 1.3 + 0.02 * k), (1.2, 1.2), (0.02 * (k % 3), 0.3 * k))
        ctx.setPrimitiveData(u, "glass_n_SW", 1.3 + 0.01 * k)
        ctx.setPrimitiveData(u, "glass_KL_SW", 0.02)
    ctx.setPrimitiveData(leaves, "reflectivity_SW", np.full(leaves.size, 0.3))
    ctx.setPrimitiveData(leaves, "transmissivity_SW", np.full(leaves.size, 0.2))
    rad = RadiationModel(ctx)
    rad.addRadiationBand("SW")
    rad.disableEmission("SW")
    s = rad.addCollimatedRadiationSource(scenes.sun_direction(25.0, 60.0))
    rad.setSourceFlux(s, "SW", 600.0)
    rad.setDiffuseRadiationFlux("SW", 100.0)
    rad.setDirectRayCount("SW", 49)
    rad.setDiffuseRayCount("SW", 64)
    rad.setScatteringDepth("SW", depth)
    rad.setSeed(21)
    got = rad.runBand("SW").astype(np.float64)
    ref, st = run_oracle(rad, ["SW"], oracle_mod, seed=21)
    floor = 1e-3 * float(np.abs(ref).mean())
    assert float((np.abs(got - ref) / np.maximum(np.abs(ref), floor)).max()) <= 1e-4
    assert rad.last_stats["rays"] == st["rays"]


@pytest.mark.parametrize("boundary", ["x", "y", "xy", "tilted"])
def test_periodic_walls_vs_oracle(oracle_mod, boundary):
    """Walls across x, across y and both, and walls that are not the planes of a box (which take no part
    in the plane test): fluxes and ray counts against the oracle."""
    from helios_gb300.radiation import Context, RadiationModel
    from helpers import run_oracle

    ctx = Context()
    ctx.addScene(scenes.mixed_canopy(400, 1.0, seed=8))
    rad = RadiationModel(ctx)
    rad.enforcePeriodicBoundary("xy" if boundary == "tilted" else boundary)
    if boundary == "tilted":
        faces = rad._bbox_faces()
        faces[1, 2, 0] += np.float32(0.01)
        rad._bbox_faces = lambda: faces
    rad.addRadiationBand("SW")
    rad.disableEmission("SW")
    s = rad.addCollimatedRadiationSource(scenes.sun_direction(55.0, 30.0))
    rad.setSourceFlux(s, "SW", 600.0)
    rad.setDiffuseRadiationFlux("SW", 100.0)
    rad.setDirectRayCount("SW", 25)
    rad.setDiffuseRayCount("SW", 64)
    rad.setSeed(5)
    got = rad.runBand("SW").astype(np.float64)
    ref, st = run_oracle(rad, ["SW"], oracle_mod, seed=5)
    floor = 1e-3 * float(np.abs(ref).mean())
    assert float((np.abs(got - ref) / np.maximum(np.abs(ref), floor)).max()) <= 1e-4
    assert rad.last_stats["rays"] == st["rays"]


def _voxel_scene(form, seed=2):
    """Leaves among voxels that are a full lattice, a lattice with holes, one layer, off the planes of
    any lattice, and a lattice far from the origin of coordinates."""
    rng = np.random.default_rng(seed)
    leaves = scenes.mixed_canopy(300, 1.0, seed=seed, height=1.0)
    div = (5, 4, 1) if form == "layer" else (5, 4, 3)
    vox = scenes.voxel_grid((0.0, 0.0, 0.05), (0.85, 0.85, 1.0), div, rng.uniform(0.0, 3.0, int(np.prod(div))))
    T, lad = vox.T.copy(), vox.lad
    if form == "holes":
        keep = rng.random(T.shape[0]) < 0.5
        T, lad = T[keep], lad[keep]
    if form == "shifted":
        T[::3, 3] += 0.03
    ty = np.concatenate([leaves.ptype, np.full(T.shape[0], scenes.VOXEL, np.uint32)])
    T = np.concatenate([leaves.T, T])
    if form == "far":
        T[:, [3, 7]] += 500.0
    return T, ty, np.concatenate([leaves.twosided, np.ones(lad.size, np.int8)]), np.concatenate([np.zeros(leaves.n), lad])


@pytest.mark.parametrize("form", ["full", "holes", "layer", "shifted", "far"])
@pytest.mark.parametrize("periodic", [False, True])
def test_voxel_lattices_vs_oracle(oracle_mod, form, periodic):
    """Voxels that are marched as a lattice, and some that are not one: fluxes and ray counts."""
    from helios_gb300.radiation import Context, RadiationModel
    from helpers import run_oracle

    T, ty, ts, lad = _voxel_scene(form)
    ctx = Context()
    uu = ctx.addPrimitives(T, ty, 1.0, ts)
    ctx.setPrimitiveData(uu, "leaf_area_density", lad)
    ctx.setPrimitiveData(uu[1:], "reflectivity_SW", np.full(uu.size - 1, 0.4))
    ctx.setPrimitiveData(uu[1:], "transmissivity_SW", np.full(uu.size - 1, 0.3))
    rad = RadiationModel(ctx)
    if periodic:
        rad.enforcePeriodicBoundary("xy")
    rad.addRadiationBand("SW")
    rad.disableEmission("SW")
    s = rad.addCollimatedRadiationSource(scenes.sun_direction(35.0, 200.0))
    rad.setSourceFlux(s, "SW", 600.0)
    rad.setDiffuseRadiationFlux("SW", 100.0)
    rad.setDirectRayCount("SW", 25)
    rad.setDiffuseRayCount("SW", 100)
    rad.setScatteringDepth("SW", 3)
    rad.setSeed(7)
    got = rad.runBand("SW").astype(np.float64)
    ref, st = run_oracle(rad, ["SW"], oracle_mod, seed=7)
    floor = 1e-3 * float(np.abs(ref).mean())
    assert float((np.abs(got - ref) / np.maximum(np.abs(ref), floor)).max()) <= 1e-4
    assert rad.last_stats["rays"] == st["rays"]
    assert rad.ctx.device_status() == 0


@pytest.mark.parametrize("n", [2, 3, 65, 1023, 1024, 1025, 1026, 5000, 140001])
@pytest.mark.parametrize("spread", ["uniform", "line", "same"])
def test_trees_of_all_sizes_hit_what_the_binary_tree_hits(gpu, n, spread):
    """The clustered tree and its 4-wide nodes at the sizes around the last block's and the tiles' limits,
    with equal areas everywhere ("same": all primitives in one place, refused beyond a depth as before):
    a solve over it equals the one over the binary tree, whose nodes the host build pins."""
    rng = np.random.default_rng(n)
    c = rng.uniform(0.0, max(1.0, (n / 50.0) ** (1.0 / 3.0)), (n, 3))
    if spread == "line":
        c[:, 1:] = 0.0
    if spread == "same":
        c[:] = 0.5
    nrm = np.tile([0.0, 0.0, 1.0], (n, 1)) if spread == "same" else scenes.uniform_sphere(rng, n)
    T = scenes.frame_T(c, np.full(n, 0.1), np.full(n, 0.1), nrm, np.zeros(n) if spread == "same" else rng.uniform(0, 6, n))
    gpu.update_geometry(T, np.zeros(n, np.uint32), np.ones(n, np.int8))
    if spread == "same" and n > 1000:  # boxes that all tie chain up, deeper than a tree may be: refused
        with pytest.raises(_hrt.HrtError, match="invalid argument"):
            gpu.build_accel()
        return
    gpu.build_accel()
    assert gpu.device_status() == 0
    R = max(4, 4000 // n)
    solve = {"band_launch": np.array([1], np.uint8), "sources": [{"type": 1, "position": (2.0, 1.0, 9.0), "width": (0.4, 0.0)}],
             "source_flux": np.array([[500.0]]), "rho": np.zeros((1, n, 1)), "tau": np.zeros((1, n, 1)),
             "diffuse_flux": np.array([50.0]), "direct_rays": np.array([R]), "diffuse_rays": np.array([4]),
             "depth": np.array([0]), "emission": np.array([0], np.uint8), "seed": 3}
    wide = gpu.run_band(solve).astype(np.float64)
    rays = gpu.last_stats()["rays"]
    gpu.set_tuning(16 + 1)  # binary nodes for the diffuse pass
    binary = gpu.run_band(solve).astype(np.float64)
    gpu.set_tuning(1)
    assert gpu.last_stats()["rays"] == rays and gpu.device_status() == 0
    assert np.all(np.abs(wide - binary) <= 2.4e-7 * np.abs(binary))


@pytest.mark.parametrize("scale", [1.0, 6.0, 4.0e4])
def test_binned_shadow_rays_from_far_walls(hrt_lib, scale):
    """A horizontal sun through periodic walls as wide as the scene, several times and 40,000 times wider
    (where the tree serves the sun): rays that come back from a wall start where coordinates are
    coarser, and find what the tree finds.  Leaves face the sun, so that many end at the edges of cells."""
    rng = np.random.default_rng(3)
    n, sun = 3000, np.array([0.6, 0.8, 0.0])
    T = scenes.frame_T(rng.uniform(0.0, 1.7, (n, 3)), np.full(n, 0.05), np.full(n, 0.05), np.tile(sun, (n, 1)), np.zeros(n))
    h, z = 2.0 * scale, 3.0
    walls = np.array([[(-h, -h, -z), (-h, h, -z), (-h, h, z), (-h, -h, z)], [(h, -h, -z), (h, h, -z), (h, h, z), (h, -h, z)],
                      [(-h, -h, -z), (h, -h, -z), (h, -h, z), (-h, -h, z)], [(-h, h, -z), (h, h, -z), (h, h, z), (-h, h, z)]],
                     np.float32)
    c = _hrt.Context(0)
    c.update_geometry(T, np.zeros(n, np.uint32), np.ones(n, np.int8), walls, (1.0, 1.0))
    c.build_accel()
    d = {"band_launch": np.array([1], np.uint8), "sources": [{"type": 0, "position": tuple(sun)}],
         "source_flux": np.array([[100.0]]), "rho": np.zeros((1, n, 1)), "tau": np.zeros((1, n, 1)),
         "diffuse_flux": np.array([0.0]), "direct_rays": np.array([400]), "diffuse_rays": np.array([1]),
         "depth": np.array([0]), "emission": np.array([0], np.uint8), "seed": 3}
    binned = c.run_band(d).astype(np.float64)
    c.set_visit_budget(1 << 30)
    tree = c.run_band(d).astype(np.float64)
    assert np.all(np.abs(binned - tree) <= 2.4e-7 * np.abs(tree))


def _direct_ms(c, d, k=7):
    import time

    c.run_band(d, out=False)
    t = []
    for _ in range(k):
        a = time.perf_counter()
        c.run_band(d, out=False)
        t.append(time.perf_counter() - a)
    return 1e3 * sorted(t)[k // 2]


@pytest.mark.parametrize("ground", [0.0, 50.0, 400.0, 5000.0])
def test_shadow_rays_of_clumped_leaves(hrt_lib, ground):
    """One plant of 20,000 leaves alone and on ever wider grounds, where the cells of a sun's grid hold
    hundreds or thousands of leaves: same fluxes as through the tree and not much slower than it."""
    rng = np.random.default_rng(0)
    n = 20000
    at = scenes.uniform_sphere(rng, n) * (rng.uniform(0, 1, n) ** (1 / 3))[:, None] * 1.25
    at[:, 2] += 1.75
    T = scenes.frame_T(at, np.full(n, 0.03), np.full(n, 0.03), scenes.uniform_sphere(rng, n), rng.uniform(0, 6, n))
    if ground:
        one = np.ones(1)
        T = np.concatenate([scenes.frame_T(np.zeros((1, 3)), ground * one, ground * one, np.array([[0.0, 0.0, 1.0]]), 0 * one), T])
    n = T.shape[0]
    c = _hrt.Context(0)
    c.update_geometry(T, np.zeros(n, np.uint32), np.ones(n, np.int8))
    c.build_accel()
    for sun in ((0.0, 0.0, 1.0), (0.6, 0.3, 0.5)):
        d = {"band_launch": np.array([1], np.uint8), "sources": [{"type": 0, "position": sun}], "source_flux": np.array([[100.0]]),
             "rho": np.zeros((1, n, 1)), "tau": np.zeros((1, n, 1)), "diffuse_flux": np.array([0.0]),
             "direct_rays": np.array([100]), "diffuse_rays": np.array([1]), "depth": np.array([0]),
             "emission": np.array([0], np.uint8), "seed": 3}
        got, ms = c.run_band(d).astype(np.float64), _direct_ms(c, d)
        c.set_visit_budget(1 << 30)
        tree, tree_ms = c.run_band(d).astype(np.float64), _direct_ms(c, d)
        c.set_visit_budget(0)
        assert np.all(np.abs(got - tree) <= 2.4e-7 * np.abs(tree))
        assert ms <= 1.5 * tree_ms, (sun, ms, tree_ms)


def test_direct_range_of_a_large_scene(hrt_lib):
    """A range with fewer rays than the scene has primitives is not worth binning them all: it makes the
    launches that it makes through the tree, and a range with more rays makes the grid's."""
    sc = scenes.mixed_canopy(300000, 2.0, seed=1)
    c = _hrt.Context(0)
    c.update_geometry(sc.T, sc.ptype, sc.twosided)
    c.build_accel()
    c.update_materials(np.zeros((1, sc.n, 1)), np.zeros((1, sc.n, 1)), 1, 1)
    c.update_sources([{"type": 0, "position": (0.3, 0.2, 0.9)}])
    c.zero_radiation_buffers(1)
    c.upload_source_fluxes([100.0])

    def launches(count):
        before = c.last_stats()["kernels"]
        c.launch_direct(launch_offset=5, launch_count=count, rays_per_primitive=25, random_seed=3, pass_id=0, nbands_global=1,
                        nbands_launch=1, band_launch_flag=np.ones(1, np.uint8))
        return c.last_stats()["kernels"] - before

    few, many = launches(10000), launches(20000)
    c.set_visit_budget(1 << 30)
    assert few == launches(10000) and many > launches(20000)


@pytest.mark.parametrize("variant,n", [(6, 133), (8, 140), (8, 144), (13, 151), (13, 159)])
def test_deep_stacks_that_fit(hrt_lib, oracle_mod, variant, n):
    """Coincident patches make a chain of nodes whose children are all pushed.  As deep as the stacks in
    shared and local memory together, each lean shape gives the oracle's fluxes and no error."""
    from helpers import oracle_solve

    T = np.concatenate([np.tile(scenes.frame_T(np.full((1, 3), 0.5), np.array([0.1]), np.array([0.1]), np.array([[0.0, 0.0, 1.0]]),
                                               np.zeros(1)), (n, 1)),
                        scenes.frame_T(np.array([[0.5, 0.5, 0.3]]), np.array([0.3]), np.array([0.3]), np.array([[0.0, 0.0, 1.0]]),
                                       np.zeros(1))]).astype(np.float32)
    n += 1
    ty, ts = np.zeros(n, np.uint32), np.ones(n, np.int8)
    c = _hrt.Context(0)
    c.update_geometry(T, ty, ts)
    c.build_accel()
    d = {"band_launch": np.array([1], np.uint8), "sources": [{"type": 0, "position": (0.0, 0.0, 1.0), "width": (0.0, 0.0)}],
         "source_flux": np.zeros((1, 1)), "rho": np.full((1, n, 1), 0.3), "tau": np.full((1, n, 1), 0.2),
         "diffuse_flux": np.array([100.0]), "direct_rays": np.array([0]), "diffuse_rays": np.array([64]),
         "depth": np.array([1]), "emission": np.array([0], np.uint8), "seed": 3}
    c.set_tuning(16 + variant)
    got = c.run_band(d).astype(np.float64)
    full = dict({k: None for k in ("diffuse_ext", "diffuse_norm", "diffuse_peak", "prague", "eps", "temperature")}, **d)
    ref, _ = oracle_mod.OracleScene(T, ty, ts).run_band(oracle_solve(full))
    floor = 1e-3 * float(np.abs(ref).mean())
    assert float((np.abs(got - ref) / np.maximum(np.abs(ref), floor)).max()) <= 1e-4
    assert c.device_status() == 0


@pytest.mark.parametrize("form", ["full", "half", "sparse", "line", "dense leaves"])
def test_lattices_are_marched_where_it_pays(hrt_lib, form):
    """Lattices of voxels that are full, half full, one cell in sixteen, a line of a thousand cells, and
    full among dense leaves: a diffuse pass takes at most 1.4 times as long as the generic trace."""
    div, occupied, ext = {"full": ((10, 10, 10), 1.0, 4.0), "half": ((10, 10, 10), 0.5, 4.0), "sparse": ((40, 40, 40), 1 / 15.5, 4.0),
                          "line": ((1024, 1, 1), 1.0, 4.0), "dense leaves": ((24, 24, 24), 1.0, 1.5)}[form]
    rng = np.random.default_rng(5)
    lv = scenes.mixed_canopy(16000, 16000 * 0.0025 / ext ** 2, seed=2, height=1.0)
    v = scenes.voxel_grid((0.0, 0.0, 0.05), (ext, ext, 1.0), div, rng.uniform(0.0, 2.0, int(np.prod(div))))
    keep = rng.random(v.n) < occupied
    keep[0] = keep[-1] = True
    T, lad = np.concatenate([lv.T, v.T[keep]]), np.concatenate([np.zeros(lv.n), v.lad[keep]])
    n = T.shape[0]
    c = _hrt.Context(0)
    c.update_geometry(T, np.concatenate([lv.ptype, v.ptype[keep]]), np.concatenate([lv.twosided, v.twosided[keep]]), None,
                      (0.0, 0.0), lad)
    c.build_accel()
    d = {"band_launch": np.array([1], np.uint8), "sources": [{"type": 0, "position": (0.0, 0.0, 1.0)}],
         "source_flux": np.zeros((1, 1)), "rho": np.zeros((1, n, 1)), "tau": np.zeros((1, n, 1)), "diffuse_flux": np.array([100.0]),
         "direct_rays": np.array([0]), "diffuse_rays": np.array([100]), "depth": np.array([0]),
         "emission": np.array([0], np.uint8), "seed": 3}
    got, ms = c.run_band(d).astype(np.float64), _direct_ms(c, d)
    c.set_tuning(16 + 4)
    generic, generic_ms = c.run_band(d).astype(np.float64), _direct_ms(c, d)
    assert np.all(np.abs(got - generic) <= 2.4e-7 * np.abs(generic))
    assert ms <= 1.4 * generic_ms, (ms, generic_ms)


@pytest.mark.parametrize("form", ["full", "holes", "layer", "shifted", "far"])
@pytest.mark.parametrize("walls", [False, True])
def test_march_equals_the_tree_of_everything(hrt_lib, form, walls):
    """The march and the generic trace, each forced, give the same fluxes and ray counts; passes of scenes
    of this size run the generic one by themselves."""
    T, ty, ts, lad = _voxel_scene(form)
    n = T.shape[0]
    c = _hrt.Context(0)
    lo, hi = T.reshape(-1, 16)[:, [3, 7, 11]].min(0) - 0.6, T.reshape(-1, 16)[:, [3, 7, 11]].max(0) + 0.6
    (x0, y0, z0), (x1, y1, z1) = lo, hi
    bb = np.array([[(x0, y0, z0), (x0, y1, z0), (x0, y1, z1), (x0, y0, z1)], [(x1, y0, z0), (x1, y1, z0), (x1, y1, z1), (x1, y0, z1)],
                   [(x0, y0, z0), (x1, y0, z0), (x1, y0, z1), (x0, y0, z1)], [(x0, y1, z0), (x1, y1, z0), (x1, y1, z1), (x0, y1, z1)]],
                  np.float32)
    c.update_geometry(T, ty, ts, bb if walls else None, (1.0, 1.0) if walls else (0.0, 0.0), lad)
    c.build_accel()
    d = {"band_launch": np.array([1], np.uint8), "sources": [{"type": 0, "position": (0.0, 0.0, 1.0)}],
         "source_flux": np.zeros((1, 1)), "rho": np.full((1, n, 1), 0.4), "tau": np.full((1, n, 1), 0.3),
         "diffuse_flux": np.array([100.0]), "direct_rays": np.array([0]), "diffuse_rays": np.array([400]), "depth": np.array([2]),
         "emission": np.array([0], np.uint8), "seed": 3}
    got = []
    for mode in (16 + 8, 16 + 4, 0):
        c.set_tuning(mode)
        got.append((c.run_band(d).astype(np.float64), c.last_stats()["rays"]))
    for flux, rays in got[1:]:
        assert rays == got[0][1]
        assert np.all(np.abs(flux - got[0][0]) <= 2.4e-7 * np.abs(got[0][0]))
    assert c.device_status() == 0
