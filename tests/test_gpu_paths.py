"""The path pipeline (csrc/dr_paths.cu) at the sizes where it can go wrong,
against the one-thread-per-path kernel: tiles equal up to the order of the
per-pixel float sums (the tolerance of the other tile tests) and every counter
equal.  The per-path kernel is pinned to the CPU restatement elsewhere."""
import numpy as np
import pytest

from conftest import c0_cfg, depth_texture, golden_octree, occluder_surfaces, settings_from_cfg
from droplet_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def renderer():
    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import Octree

    r = Renderer(0)
    r.upload(Octree(*golden_octree()))
    yield r
    r.close()


def _pair(r, cfg, tile, spp, seed=11):
    """(sun, sky, counters) of the pipeline and of the per-path kernel."""
    r.set_params(settings_from_cfg(cfg))
    got = []
    for kernel in (0, 1):
        r.set_tuning(kernel)
        r.reset_counters()
        sun, sky = r.render_tile(*tile, spp, seed=seed, sample_base=2)
        got.append((sun, sky, r.counters()))
    r.set_tuning()
    return got


def _check(got):
    (s0, k0, c0), (s1, k1, c1) = got
    assert c0 == c1
    for g, p in ((s0, s1), (k0, k1)):
        assert np.allclose(g, p, rtol=2e-5, atol=1e-6 * np.abs(p).max() + 1e-30)


# tile edges (list blocks of 16 x 8 pixels, odd tiles drop a row and a column), samples around the warp and the ticket
@pytest.mark.parametrize("tile", [(30, 30, 2, 2), (20, 22, 3, 5), (9, 14, 17, 9), (5, 3, 50, 47)])
@pytest.mark.parametrize("spp", [1, 31, 33, 130])
def test_tile_and_sample_edges(renderer, tile, spp):
    _check(_pair(renderer, c0_cfg(64, 64), tile, spp))


@pytest.mark.parametrize("events", [0, 1, 40])
def test_event_limits(renderer, events):
    cfg = dict(c0_cfg(64, 64), scattevs=events, sigma_s=60.0, sigma_a=0.1)
    _check(_pair(renderer, cfg, (8, 8, 48, 48), 32))


@pytest.mark.parametrize("flags", [{"depthcomp": True}, {"finite_paths": True}, {"depthcomp": True, "embree": True}])
def test_depth_and_flags(renderer, flags):
    _check(_pair(renderer, dict(c0_cfg(64, 64), depth=depth_texture(64, 64), **flags), (4, 2, 56, 60), 24))


def test_axis_parallel_rays(renderer):
    """The middle row and column of an odd image have a zero direction component
    (they take the octree), and the sun stands exactly on an axis."""
    cfg = c0_cfg(33, 33)
    viewi = np.eye(4, dtype=np.float32)
    viewi[3, :3] = (0.5, 0.5, 3.0)
    cfg.update(viewi=viewi, sun_dir=np.array([0.0, 1.0, 0.0], np.float32))
    got = _pair(renderer, cfg, (0, 0, 33, 33), 48)
    assert got[0][2]["mie_evals"] > 0
    _check(got)


def test_rounds(renderer):
    """More collided samples than the record buffer holds (2^20 for this frame):
    the launch runs in rounds."""
    cfg = dict(c0_cfg(32, 32), sigma_s=400.0, sigma_a=4.0, scattevs=2)
    got = _pair(renderer, cfg, (8, 8, 16, 16), 8192)
    assert got[0][2]["mie_evals"] > 3 * (1 << 20)
    _check(got)


@pytest.mark.parametrize("pool", [N.DR_NONE, 1, 300])
def test_pixels_without_lists(renderer, pool):
    try:
        renderer.set_camera_lists(pool)
        _check(_pair(renderer, c0_cfg(64, 64), (4, 6, 50, 52), 37))
    finally:
        renderer.set_camera_lists(0)


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    ro = 0.5 + rng.uniform(-0.3, 0.3, (n, 3)) - rng.choice([0.0, 1.5], (n, 1)) * d
    rd = d.astype(np.float32)
    rd[0] = (0.0, 0.0, -1.0)  # a zero direction component: takes the octree
    return ro.astype(np.float32), rd


# samples around a warp's share of a ray (64 to 4,096)
@pytest.mark.parametrize("n_rays,nsamp", [(1, 1), (3, 33), (700, 64), (5, 4097), (40, 20000)])
def test_transmittance_counts(renderer, n_rays, nsamp):
    """The escapes equal those the adjoint's replay counts (octree, one sample a thread), sample for sample."""
    renderer.set_params(settings_from_cfg(c0_cfg(64, 64)))
    ro, rd = _rays(n_rays, n_rays)
    got = renderer.probe_transmittance(ro, rd, nsamp, seed=77)
    _, ref = renderer.adjoint_transmittance(ro, rd, np.ones(n_rays), nsamp, 77, len(golden_octree()[1]))
    assert np.array_equal(got, ref)


def test_transmittance_of_long_leaf_lists():
    """Rays with more leaves than a warp keeps (96) are traversed per sample."""
    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import build_octree

    i = np.arange(128)
    org = np.stack([8 * i, 8 * i, 8 * i], 1).astype(np.int32)
    oc = build_octree(org, np.full((128, 512), 0.02, np.float32), 1.0 / 1024, 12)
    with Renderer(0) as r:
        r.upload(oc)
        r.set_params(settings_from_cfg(c0_cfg(64, 64)))
        ro = np.array([[-0.2, -0.2001, -0.1999], [0.5, 0.5, 0.5]], np.float32)
        rd = np.array([[1.0, 1.0001, 0.9999], [0.3, -0.2, 0.9]], np.float32)
        rd /= np.linalg.norm(rd, axis=1, keepdims=True).astype(np.float32)
        assert r.probe_leaf_sequence(ro, rd, 512)[3].max() > 96
        got = r.probe_transmittance(ro, rd, 1000, seed=5)
        _, ref = r.adjoint_transmittance(ro, rd, np.ones(2), 1000, 5, oc.n_leaves)
        assert np.array_equal(got, ref) and got.min() < 1.0


@pytest.mark.parametrize("flags", [{"embree": True}, {"embree": True, "finite_paths": True}, {"embree": False}])
@pytest.mark.parametrize("tile,spp", [((30, 30, 2, 2), 1), ((9, 14, 17, 9), 33), ((2, 2, 60, 60), 40)])
def test_occluder_light(flags, tile, spp):
    """The light of lit shadow segments and escapes, tested against the occluders in
    the warp's queue (embree), in place (finite_paths) or not at all."""
    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import Octree

    with Renderer(0) as r:
        r.set_occluders(occluder_surfaces())
        r.upload(Octree(*golden_octree()))
        _check(_pair(r, dict(c0_cfg(64, 64), **flags), tile, spp))


def test_majorants_with_unreachable_leaves():
    """Leaf nodes that the root does not reach get majorants of their own from
    dr_set_bricks_dev, and leave those of the leaves in the block grid alone: rays
    through every leaf count the escapes of the octree's replay."""
    import torch

    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import Octree

    nodes, bricks, mlevel = golden_octree()
    leaves = np.flatnonzero(nodes["volx"][:, 1] != N.DR_NONE)
    loose = np.repeat(nodes[leaves[:1]], 500)  # nodes without a parent, each with a denser brick
    loose["volx"][:, 1] = len(bricks)
    with Renderer(0) as r:
        r.upload(Octree(np.concatenate([nodes, loose]), np.concatenate([bricks, np.full((1, 512), 7.0, np.float32)]),
                        mlevel))
        r.set_params(settings_from_cfg(c0_cfg(64, 64)))
        b = torch.as_tensor(np.concatenate([0.5 * bricks, np.full((1, 512), 9.0, np.float32)]), device="cuda")
        r.set_bricks_dev(b.data_ptr(), len(bricks) + 1, 1.0)
        r.synchronize()
        maj = r.majorants(len(nodes) + len(loose))
        assert (maj[len(nodes):] == 9.0).all() and maj[:len(nodes)].max() < 9.0
        d = np.random.default_rng(1).normal(size=(len(leaves), 3))
        d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        ro = nodes["ce"][leaves][:, :3] - 2.0 * d
        got = r.probe_transmittance(ro, d, 256, seed=9)
        _, ref = r.adjoint_transmittance(ro, d, np.ones(len(leaves)), 256, 9, len(bricks) + 1)
        assert np.array_equal(got, ref) and got.min() < 1.0


@pytest.mark.parametrize("more", [dict(phase_mode=N.DR_PHASE_HG, hg_g=0.6), dict(env_mode=N.DR_ENV_NONE)])
def test_occluders_without_the_flag(more):
    """Occluders count with DR_KERNEL_EMBREE only, whatever other options choose the
    kernel: pipeline, cell walk and one thread per path render the frame without any."""
    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import Octree

    cfg = dict(c0_cfg(64, 64), **more)
    images = []
    with Renderer(0) as r:
        r.upload(Octree(*golden_octree()))
        for occluders in ([], occluder_surfaces()):
            r.set_occluders(occluders)
            r.set_params(settings_from_cfg(cfg))
            for kernel, traversal in ((0, 0), (0, 1), (1, 0)):
                r.set_tuning(kernel, traversal=traversal)
                images.append(r.render_tile(2, 2, 60, 60, 33, seed=11, sample_base=2))
    for g in images[1:]:
        for a, b in zip(g, images[0]):
            assert np.allclose(a, b, rtol=2e-5, atol=1e-6 * np.abs(b).max() + 1e-30)


def test_counters_repeat_with_occluders():
    """Frames and shadow passes with occluders count the same in every launch."""
    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import Octree

    cfg = dict(c0_cfg(160, 120), depth=depth_texture(160, 120), embree=True, phase_mode=N.DR_PHASE_HG, hg_g=0.6)
    with Renderer(0) as r:
        r.set_occluders(occluder_surfaces())
        r.upload(Octree(*golden_octree()))
        r.set_params(settings_from_cfg(cfg))
        counts = []
        for _ in range(20):
            r.reset_counters()
            r.render_tile(0, 0, 160, 120, 48, seed=5, sample_base=0)
            frame = r.counters()
            r.reset_counters()
            r.render_shadow_tile(0, 0, 160, 120, 48, seed=5, sample_base=0)
            counts.append((frame, r.counters()))
        assert all(c == counts[0] for c in counts)
        r.set_tuning(1)  # one thread per path
        r.reset_counters()
        r.render_tile(0, 0, 160, 120, 48, seed=5, sample_base=0)
        assert r.counters() == counts[0][0]


def test_deep_occluder_tree():
    """A fan of triangles whose boxes all overlap: a deep tree, and rays that go down both sides."""
    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import Octree

    n = 3000  # sizes over five decades make the surface-area splits uneven
    rng = np.random.default_rng(8)
    size = np.geomspace(1e-4, 0.5, n)[:, None, None]
    v = (np.array([1.2, 1.0, 1.2]) + size * (1.0 + rng.normal(size=(n, 3, 3)))).reshape(-1, 3).astype(np.float32)
    with Renderer(0) as r:
        r.set_occluders([(v, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), 2)])
        r.upload(Octree(*golden_octree()))
        got = _pair(r, dict(c0_cfg(64, 64), embree=True), (4, 4, 56, 56), 33)
        _check(got)
        r.set_occluders([])
        r.set_tuning(1)
        free = r.render_tile(4, 4, 56, 56, 33, seed=11, sample_base=2)
        assert got[0][0][..., :3].sum() < 0.9 * free[0][..., :3].sum()


def test_more_tickets_than_32_bits():
    """2^39 + 4096 samples: 2^32 + 32 tickets, nearly all of them through the one leaf before the camera."""
    import torch

    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import build_octree

    org = np.array([[0, 0, 0], [16, 16, 16], [32, 32, 32], [56, 56, 56]], np.int32)
    oc = build_octree(org, np.full((4, 512), 0.01, np.float32), 1.0 / 64, 12)
    spp = 2 ** 27 + 1
    cfg = dict(c0_cfg(1920, 1080), sigma_s=1e-5, sigma_a=1e-7, scattevs=1)
    eye = oc.nodes["ce"][np.flatnonzero(oc.nodes["volx"][:, 1] != N.DR_NONE)[1]][:3]
    viewi = np.array(cfg["viewi"], np.float32).reshape(4, 4)
    viewi[3, :3] = eye  # inside a leaf: every camera ray meets it
    cfg["viewi"] = viewi.reshape(-1)
    with Renderer(0) as r:
        r.upload(oc)
        r.set_params(settings_from_cfg(cfg))
        sun, sky = (torch.zeros((64, 64, 4), device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        r.reset_counters()
        r.render_tile_async(930, 500, 64, 64, spp, 3, 0, sun.data_ptr(), sky.data_ptr())
        r.synchronize()
        c = r.counters()
        assert c["paths"] == 4096 * spp
        assert c["vertices"] >= 4096 * spp and c["gave_up"] == 0


@pytest.mark.parametrize("levels,leaves", [(4, 300), (7, 3000), (9, 6000)])
def test_deep_sparse_octrees(levels, leaves):
    """Scattered leaves in deep octrees: empty nodes of every size between them, so that
    rays cross the upper levels of the grid.  Frames, shadow segments and every counter."""
    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import build_octree

    rng = np.random.default_rng(levels)
    n = 15 * 2 ** (levels - 3)  # blocks a side: the root's 2^levels cells hold them at 7 voxels a block
    cells = rng.choice(n ** 3, leaves, replace=False)
    near = n // 2 + rng.integers(-3, 4, (leaves // 3, 3))  # a third of them close together
    org = np.unique(np.concatenate([np.stack(np.unravel_index(cells, (n, n, n)), 1), near,
                                    [[0, 0, 0], [n - 1] * 3]]), axis=0).astype(np.int32) * 8
    oc = build_octree(org, rng.uniform(0.1, 1.0, (len(org), 512)).astype(np.float32), 1.0 / (8 * n), 12)
    cfg = dict(c0_cfg(96, 80), sigma_s=40.0 * 2 ** levels, sigma_a=2.0, scattevs=12)
    with Renderer(0) as r:
        r.upload(oc)
        got = _pair(r, cfg, (0, 0, 96, 80), 24)
        assert got[0][2]["mie_evals"] > 1000
        _check(got)
        ro, rd = _rays(200, levels)
        _, ref = r.adjoint_transmittance(ro, rd, np.ones(200), 500, 3, oc.n_leaves)
        assert np.array_equal(r.probe_transmittance(ro, rd, 500, seed=3), ref) and ref.min() < 1.0
