"""A top-level rebuild that is refused because the trees together are too deep
for the traversal stack: the moved scene's two traversals still agree.  The
rebuild has replaced the top level's nodes and the instances' leaf order by
then, so the walkers' copies of the nodes have to be the new ones too."""
import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context, DDGIError
from test_gpu_walk_nodes import boxes

pytestmark = pytest.mark.gpu

BOXES = 15


def deep_mesh(levels):
    """One triangle a level: each is more than 32 bins further out than the next
    smaller one along its axis, so that every split takes one off."""
    pos = []
    for i in range(levels):
        axis, m = i % 3, 2.0 ** (50.0 - 5.25 * (i // 3))
        p = np.zeros((3, 3))
        p[:, axis] = m
        p[1, (axis + 1) % 3] = p[2, (axis + 2) % 3] = 1e-6 * m
        pos.append(p)
    return np.concatenate(pos).astype(np.float32)


def scene(levels):
    """boxes() on a row of their own with the one-triangle mesh in place of the
    deep one, which no ray's mask meets."""
    sc = boxes(3, BOXES, 1.0, 1.0, (0, 0, 0))
    v = np.zeros(3 * levels, abi.VERTEX_DTYPE)
    v["pos"] = deep_mesh(levels)
    v["normal"] = (0, 1, 0)
    meshes, inst = sc.meshes.copy(), sc.instances.copy()
    meshes[0] = (len(sc.vertices), 3 * levels, sc.indices.size, 3 * levels)
    inst[0]["transform"] = scenes.affine_3x4(np.eye(3) * 2.0 ** -32, (0, 0, 0))
    inst[0]["mask"] = 0
    for i in range(BOXES):
        inst[1 + i]["transform"] = scenes.affine_3x4(np.eye(3), (3.0 * (i % 4) - 4, 0.0, 3.0 * (i // 4) - 4))
    idx = np.concatenate([sc.indices, np.arange(3 * levels, dtype=np.uint32)])
    return scenes.Scene(np.concatenate([sc.vertices, v]), idx, meshes, inst, sc.offsets, sc.materials)


@pytest.mark.parametrize("mode", ["fast_trace", "fast_trace_host"])
def test_traversals_agree_after_a_refused_rebuild(gpu_lib, mode):
    sc = scene(87)
    g = abi.make_grid((-30, -30, -30), (30, 30, 30), (4, 4, 4), 1024)
    ctx = Context(g)
    ctx.set_build_mode(mode)
    ctx.set_leaf_size(1)
    ctx.build_scene(sc)
    ctx.set_light(scenes.default_light())
    ctx.record_hits(True)
    assert 78 <= ctx.scene_info()["depth_blas"] <= 87
    # boxes five times as far and as large as the one before: a level each
    t = np.stack([scenes.affine_3x4(np.eye(3) * 0.3 * 0.5 * 5.0 ** i, [0.5 * 5.0 ** i] * 3) for i in range(BOXES)])
    with pytest.raises(DDGIError, match="too deep"):
        ctx.update_instances(t, ids=np.arange(1, BOXES + 1, dtype=np.uint32), rebuild=True)
    ctx.update(scenes.random_orientation(5, 2))
    got = ctx.get_hits(g.probe_count()).reshape(-1)
    step = np.float32(20.0)
    i = np.arange(64)
    origins = np.stack([i % 4, i % 16 // 4, i // 16], -1).astype(np.float32) * step + np.float32(-30.0)
    dirs = np.tile(ctx.get_ray_directions()[:, :3], (64, 1))
    tmax = float(np.sqrt(np.float32(3 * 3600.0)))
    want, _ = ctx.trace_rays(np.repeat(origins, 1024, 0), dirs, float(np.float32(0.01)), tmax, mask=0x3)
    ctx.close()
    hit = want["instance"] != abi.MISS
    assert len(np.unique(want["instance"][hit])) >= 4
    assert (got["instance"] == want["instance"]).all()
    assert (got["primitive"][hit] == want["primitive"][hit]).all()
    assert (got["t"][hit].view(np.uint32) == want["t"][hit].view(np.uint32)).all()
