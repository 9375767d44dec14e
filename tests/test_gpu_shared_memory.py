"""Dynamic shared memory of the path pipeline: what a launch needs depends on the
phase tables and on the octree's depth, and the limit it runs under belongs to the
kernel, for every context and thread of the process."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from conftest import c0_cfg, mie_table, settings_from_cfg
from droplet_b200 import _native as N

pytestmark = pytest.mark.gpu


def _scene(levels):
    """A cluster of leaves in an octree `levels` deep (two far corners hold it open)."""
    from droplet_b200.scene import build_octree

    n = 15 * 2 ** (levels - 3)
    c = n // 2 + np.arange(-2, 3)
    org = np.stack(np.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3)
    org = np.concatenate([[[0, 0, 0]], org, [[n - 1] * 3]]).astype(np.int32) * 8
    vals = np.random.default_rng(levels).uniform(0.2, 0.6, (len(org), 512)).astype(np.float32)
    oc = build_octree(org, vals, 1.0 / (8 * n), 12)
    depth, node = 0, 0
    while oc.nodes["volx"][node].min() == 0xFFFFFFFF:
        node = int(oc.nodes["chn"][node].max())
        depth += 1
    assert depth == levels
    return oc


def _cfg(**more):
    """A camera close enough that the cluster fills the frame."""
    cfg = dict(c0_cfg(24, 24), **{"sigma_s": 600.0, "sigma_a": 6.0, "scattevs": 6, **more})
    viewi = np.array(cfg["viewi"], np.float32).reshape(4, 4)
    viewi[3, :3] = 0.5 + 0.25 * (viewi[3, :3] - 0.5)
    cfg["viewi"] = viewi.reshape(-1)
    return cfg


def _render(r, spp=16, seed=3):
    return r.render_tile(0, 0, 24, 24, spp, seed=seed, sample_base=0)


def _close(got, ref):
    assert ref[0][..., 3].sum() > 0
    for g, p in zip(got, ref):
        assert np.allclose(g, p, rtol=2e-5, atol=1e-6 * np.abs(p).max() + 1e-30)


def test_two_threads_with_different_depths():
    """The exact sampler's 256 entries need 49,424 bytes at depth 4 and 52,496 at depth 6."""
    from droplet_b200.renderer import Renderer

    rs, refs, failed = [], [], []
    for levels in (4, 6):
        r = Renderer(0)
        r.upload(_scene(levels))
        r.set_params(settings_from_cfg(_cfg(phase_mode=N.DR_PHASE_MIE_EXACT)))
        r.set_tuning(1)  # one thread per path
        refs.append(_render(r))
        r.set_tuning()
        rs.append(r)

    def work(r, ref):
        import torch

        try:
            sun, sky = (torch.zeros((24, 24, 4), device="cuda") for _ in range(2))
            torch.cuda.synchronize()
            for _ in range(4000):  # launches only: the calls of both threads interleave
                r.render_tile_async(0, 0, 24, 24, 16, 3, 0, sun.data_ptr(), sky.data_ptr())
            r.synchronize()
            _close((sun.cpu().numpy(), sky.cpu().numpy()), ref)
        except BaseException as e:  # noqa: BLE001 (reported by the main thread)
            failed.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(rs, refs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in rs:
        r.close()
    assert not failed, failed


def test_split_batch_of_both_depths():
    """Views with kernels of their own, captured deep first."""
    from droplet_b200.renderer import Batch, BatchView, Renderer

    s = settings_from_cfg(_cfg(phase_mode=N.DR_PHASE_MIE_EXACT))
    with Renderer(0) as r:
        scenes = [_scene(6), _scene(4)]
        b = Batch(r, scenes, [BatchView(0, s, 16, 3), BatchView(1, s, 16, 3)])
        try:
            b.set_split(1)
            assert b.get_split()[1] == 2
            b.launch()
            for v in range(2):
                r.upload(scenes[v])
                r.set_params(s)
                _close(b.read(v), _render(r))
        finally:
            b.close()


# the pipeline's dynamic part at depth 5 is 11,520 + 7,680 + 29,952 = 49,152 bytes with 576 entries (plain) and
# 8,960 + 7,680 + 32,512 = 49,152 with 448 (adjoint): exactly the default limit, which also holds the kernel's barrier
@pytest.mark.parametrize("entries,adjoint", [(572, False), (576, False), (580, False), (444, True), (448, True)])
def test_sizes_around_the_default_limit(entries, adjoint):
    """In a process of its own: a limit raised before would hide the fault."""
    subprocess.run([sys.executable, __file__, str(entries), str(int(adjoint))], check=True, timeout=300,
                   cwd=os.path.dirname(__file__))


def _at_the_limit(entries, adjoint):
    import torch

    from droplet_b200.renderer import Renderer

    pdf, cdf = mie_table()
    k = np.minimum(np.arange(entries) * len(pdf) // entries, len(pdf) - 1)
    with Renderer(0) as r:
        oc = _scene(5)
        r.upload(oc)
        r.set_params(settings_from_cfg(_cfg(mie_pdf=np.ascontiguousarray(pdf[k]), mie_cdf=np.ascontiguousarray(cdf[k]))))
        if adjoint:
            d = torch.ones((24, 24, 4), device="cuda")
            g = torch.zeros((oc.n_leaves, 512), device="cuda")
            a = torch.zeros(1, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            r.adjoint_tile_async(0, 0, 24, 24, 16, 3, 0, d.data_ptr(), d.data_ptr(), g.data_ptr(), a.data_ptr())
            r.synchronize()
            assert float(g.abs().sum()) > 0 and float(a) > 0
            return
        got = _render(r)
        r.set_tuning(1)  # one thread per path
        _close(got, _render(r))


if __name__ == "__main__":
    _at_the_limit(int(sys.argv[1]), bool(int(sys.argv[2])))
