"""Meshes whose nodes sit at the edge between the GPU tree builder's block and
warp passes (64 references, two a lane) and at its rounds of 32: the trees
equal the host builder's node for node.  Triangles overlap heavily, so spatial
splits are taken and references straddle their planes; some triangles lie in a
bin plane or have a corner on one."""
import numpy as np
import pytest

from test_gpu_gbuild import assert_same_trees, custom_scene
from vulkanexp_gb300 import scenes

pytestmark = pytest.mark.gpu


def soup(rng, n, kind):
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    t = c + rng.uniform(-0.7, 0.7, (n, 3, 3)) * rng.uniform(0.05, 1.5, (n, 1, 3))
    if kind == "grid":  # corners on the planes of a 32-bin grid
        t = np.round(t * 16) / 16
    if kind == "slab":  # flat along y, a few standing up
        t[: n - n // 8, :, 1] = np.round(t[: n - n // 8, :1, 1] * 2) / 2
    return t.reshape(-1, 3), np.arange(3 * n).reshape(n, 3)


@pytest.mark.parametrize("kind", ["free", "grid", "slab"])
@pytest.mark.parametrize("leaf,alpha", [(2, 1e-3), (1, 1e-5), (8, 0.0)])
def test_trees_at_the_small_node_limit(gpu_lib, kind, leaf, alpha):
    rng = np.random.default_rng(len(kind) + leaf)
    counts = [2, 3, 31, 32, 33, 63, 64, 65, 66, 127, 129, 1023, 1025]
    meshes = [soup(rng, n, kind) for n in counts]
    eye = np.concatenate([np.eye(3), np.zeros((3, 1))], 1)
    instances = []
    for m in range(len(meshes)):
        t = eye.copy()
        t[:, 3] = (4.0 * (m % 4), 0.0, 4.0 * (m // 4))
        instances.append((m, t.reshape(12)))
    sc = custom_scene(meshes, instances)
    sc.bounds = (np.full(3, -2.0), np.full(3, 16.0))
    w = scenes.Workload("small nodes", sc, scenes.fit_grid(sc, (2, 2, 2), 8), scenes.default_light(), 1, 3)
    assert_same_trees(w, leaf, alpha)
