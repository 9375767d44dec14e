"""The adjoint's decision tape (csrc/dr_paths.cu, tape_scatter_kernel) where it
ends or does not serve, against the CPU restatement on the same random streams
(the tolerance of the other adjoint tests): paths whose decisions do not fit or
with more shadow segments than a record has bits for are replayed, as are rays
with a zero direction component; and a gradient that is not aligned."""
import numpy as np
import pytest

from conftest import c0_cfg, depth_texture, golden_octree, settings_from_cfg

pytestmark = pytest.mark.gpu


def _adjoint(r, tile, spp, dsun, dsky, n_leaves, shift=0):
    import torch

    ds, dk = (torch.as_tensor(d, device="cuda").contiguous() for d in (dsun, dsky))
    g = torch.zeros(n_leaves * 512 + 4, dtype=torch.float32, device="cuda")
    ga = torch.zeros(1, dtype=torch.float64, device="cuda")
    r.adjoint_tile_async(*tile, spp, 5, 1, ds.data_ptr(), dk.data_ptr(), g.data_ptr() + 4 * shift, ga.data_ptr())
    torch.cuda.synchronize()
    assert not g[:shift].any() and not g[shift + n_leaves * 512:].any()
    return g[shift:shift + n_leaves * 512].double().cpu().numpy().reshape(-1, 512), float(ga.item())


def _axis_cfg():
    viewi = np.eye(4, dtype=np.float32)
    viewi[3, :3] = (0.5, 0.5, 3.0)
    return dict(c0_cfg(33, 33), viewi=viewi.ravel(), sun_dir=np.array([0.0, 1.0, 0.0], np.float32))


# deep: more than 64 events a path, and more decisions than the tape holds
CASES = {
    "no events": (lambda: dict(c0_cfg(64, 64), scattevs=0), (8, 8, 48, 40), 8),
    "one event": (lambda: dict(c0_cfg(64, 64), scattevs=1), (5, 3, 49, 47), 5),
    "deep": (lambda: dict(c0_cfg(64, 64), scattevs=100, sigma_s=2000.0, sigma_a=0.01), (24, 24, 16, 16), 16),
    "axis": (_axis_cfg, (0, 0, 33, 33), 24),
    "depth": (lambda: dict(c0_cfg(64, 64), depth=depth_texture(64, 64), depthcomp=True), (4, 2, 56, 60), 6),
}


@pytest.mark.parametrize("case", list(CASES))
def test_tape_equals_restatement(port, case):
    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import Octree

    make, tile, spp = CASES[case]
    cfg = make()
    nodes, bricks, mlevel = golden_octree()
    rng = np.random.default_rng(4)
    dsun, dsky = (rng.normal(size=(tile[3], tile[2], 4)).astype(np.float32) for _ in range(2))
    dsun[::5, 1::4] = dsky[::5, 1::4] = 0.0  # pixels without a gradient
    keep = []
    g_cpu, a_cpu = port.adjoint_tile(port.scene(nodes, bricks), port.params(cfg, keep), *tile, spp, 5, 1, dsun, dsky)
    with Renderer(0) as r:
        r.upload(Octree(nodes, bricks, mlevel))
        r.set_params(settings_from_cfg(cfg))
        g, a = _adjoint(r, tile, spp, dsun, dsky, len(bricks))
    scale = np.abs(g_cpu).max()
    assert (scale > 0) == (cfg["scattevs"] > 0)
    assert np.allclose(g, g_cpu, rtol=1e-3, atol=1e-4 * scale)
    assert abs(a - a_cpu) <= 1e-4 * abs(a_cpu)


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_unaligned_gradient(shift):
    """More leaves than the gradient is spread over copies for (one copy in
    256 MB), so that the caller's gradient itself is added to."""
    from droplet_b200.renderer import Renderer
    from droplet_b200.scene import build_octree

    k = np.arange(64)
    org = np.stack(np.meshgrid(k, k, np.arange(17), indexing="ij"), -1).reshape(-1, 3).astype(np.int32) * 16
    fld = np.random.default_rng(2).uniform(0.0, 0.4, (len(org), 512)).astype(np.float32)
    oc = build_octree(org, fld, 1.0 / 1024, 12)
    assert oc.n_leaves > 65536
    rng = np.random.default_rng(4)
    d = rng.normal(size=(64, 64, 4)).astype(np.float32)
    with Renderer(0) as r:
        r.upload(oc)
        r.set_params(settings_from_cfg(c0_cfg(64, 64)))
        tile = (0, 0, 64, 64)
        ref, a_ref = _adjoint(r, tile, 16, d, d, oc.n_leaves)
        g, a = _adjoint(r, tile, 16, d, d, oc.n_leaves, shift)
    scale = np.abs(ref).max()
    assert scale > 0
    assert np.allclose(g, ref, rtol=1e-4, atol=1e-5 * scale)
    assert abs(a - a_ref) <= 1e-5 * abs(a_ref)
