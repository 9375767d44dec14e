"""The grid traversal (csrc/dr_device.cuh) against the octree traversal, and the
first-flight test against the flight in full, compiled for the host: the same
leaves, intervals (bit for bit) and node visits on every ray either accepts."""
import os
import subprocess

import numpy as np
import pytest

from droplet_b200 import workloads as W
from droplet_b200.scene import build_octree

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "droplet-render_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("grid")
    exe = str(d / "grid_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", f"-I{CUDA}/include", "-o", exe,
                    os.path.join(HERE, "host", "grid_check.cpp"), "-x", "c++", os.path.join(CSRC, "dr_host.cu"),
                    f"-L{CUDA}/lib64", "-lcudart", "-lpthread"], check=True)

    def run(*args):
        p = subprocess.run([exe, *map(str, args)], capture_output=True, text=True)
        assert p.returncode == 0, (args, p.returncode, p.stdout, p.stderr)
        return p.stdout

    run.dir = d
    return run


def _save(oc, path):
    with open(path, "wb") as f:
        np.array([len(oc.nodes), len(oc.bricks)], np.uint32).tofile(f)
        oc.nodes.tofile(f)
    return path


def _scene(name):
    if name == "slab":  # a deep sparse tree, some of whose inner nodes have no children
        rec = W.slab_recipe(1024)
        org = np.unique(np.concatenate([W.puff_blocks(rec, p) for p in rec.puffs]), axis=0)
        org = org[np.random.default_rng(0).random(len(org)) < 0.3]
        return build_octree(org.astype(np.int32), np.ones((len(org), 512), np.float32), rec.voxel_size, 12)
    n = int(name)
    rec = W.config0_recipe(64) if n == 64 else W.cumulus_recipe(n)
    org, vals = W.sparse_field(rec)
    return build_octree(org, vals, rec.voxel_size, 12)


@pytest.mark.parametrize("name,levels", [("64", 2), ("96", 3), ("slab", 6)])
def test_grid_traversal_equals_octree(check, name, levels):
    out = check(_save(_scene(name), str(check.dir / f"{name}.bin")), 300000, 7)
    assert f"levels {levels} " in out


def test_first_flight_test_is_safe(check):
    check("flights", 20000000, 3)


def test_leaf_list_pool_beyond_32_bits(check):
    """Lists that do not fit are counted as well: the ranges stay apart when more than 2^32 entries are asked for."""
    check("pool", 500000, 5)


def test_storage_takes_the_largest_size_that_fits(check):
    """List and pipeline storage where memory is short: smaller, before the kernels without it; asked for once."""
    check("storage", 200000, 11)


def test_cheaper_operations_give_the_same_bits(check):
    """Uniform draws, their logarithm, the brick lookup and the collision test without
    conversions and divisions, against the operations they replace."""
    check("exact", 20000000, 13)
