"""The persistent walkers' box tests at the ends of their range: boxes of planes
far from the ray with a direction component that is zero (the product of the
centre's distance and the component's reciprocal passes the largest float), and
boxes ten thousand box sizes away."""
import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context
from test_gpu_walk_nodes import boxes

pytestmark = pytest.mark.gpu

AXES = [np.array(m, np.float32) for m in (
    [[1, 0, 0], [0, 1, 0], [0, 0, 1]], [[-1, 0, 0], [0, 1, 0], [0, 0, 1]],
    [[0, 1, 0], [1, 0, 0], [0, 0, 1]], [[0, 1, 0], [-1, 0, 0], [0, 0, 1]],
    [[0, 1, 0], [0, 0, 1], [1, 0, 0]], [[0, 1, 0], [0, 0, 1], [-1, 0, 0]])]


def plates(reach, scale):
    """Six plates around the origin at distance 2, each from -reach to 0.2 reach
    along its axes, a mesh and an instance each: vertices divided by `scale`,
    which the instance multiplies back."""
    base = scenes.room_with_boxes(1, 5)
    pos, nrm = [], []
    for k in range(6):
        axis, sign = k // 2, 1.0 if k % 2 else -1.0
        u, v = (axis + 1) % 3, (axis + 2) % 3
        p = np.zeros((4, 3))
        p[:, axis] = 2.0 * sign
        p[:, u] = reach * np.array([-1.0, 0.2, 0.2, -1.0])
        p[:, v] = reach * np.array([-0.3, -0.3, 0.7, 0.7])
        pos.append(p / scale)
        n = np.zeros((4, 3))
        n[:, axis] = -sign
        nrm.append(n)
    facing = np.array([0, 1, 2, 0, 2, 3], np.uint32)  # along +axis; the plates face the origin
    quads = np.concatenate([facing if k % 2 == 0 else facing[::-1] for k in range(6)])
    meshes = np.zeros(6, base.meshes.dtype)
    inst, off = base.instances.copy(), base.offsets.copy()
    for k in range(6):
        meshes[k] = (4 * k, 4, 6 * k, 6)
        inst[k]["transform"] = scenes.affine_3x4(np.eye(3) * scale, (0, 0, 0))
        inst[k]["mesh_index"] = inst[k]["custom_index"] = k
        off[k] = (0, 4 * k, 6 * k)
    return scenes.Scene(scenes.make_vertices(np.concatenate(pos), np.concatenate(nrm)), quads, meshes, inst,
                        off, base.materials)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -20])
@pytest.mark.parametrize("reach", [1e6, 1e9, 1e12, 5e12])
def test_plates_with_far_edges(gpu_lib, reach, scale):
    g = abi.make_grid((-1, -1, -1), (1, 1, 1), (4, 3, 5), 1)
    ctx = Context(g)
    ctx.build_scene(plates(reach, scale))
    ctx.set_light(scenes.make_light((0.0, 1.0, 0.0), (3.0, 2.0, 1.0), (0.5, 0.6, 0.7)))
    ctx.record_hits(True)
    n = g.probe_count()
    i = np.arange(n)
    f = np.float32
    origins = np.stack([i % 4, i % 12 // 4, i // 12], -1).astype(f) * (f(2.0) / f([3, 2, 4])) - f(1.0)
    for m in AXES:
        ctx.update(m.reshape(9))
        d = ctx.get_ray_directions()[:, :3]
        assert d.shape == (1, 3) and np.count_nonzero(d) == 1
        got = ctx.get_hits(n).reshape(-1)
        tmax = float(np.sqrt(f(12.0)))
        want, _ = ctx.trace_rays(origins, np.tile(d, (n, 1)), float(f(0.01)), tmax, mask=0x3)
        assert (want["instance"] != abi.MISS).all() and not want["backface"].any()
        for k in ("instance", "primitive", "backface"):
            assert (got[k] == want[k]).all()
        assert (got["t"].view(np.uint32) == want["t"].view(np.uint32)).all()
    # any hit: under a sun straight above, the plate above shades every other one
    ctx.update(AXES[3].reshape(9))  # straight down
    below = ctx.get_ray_records(n).reshape(-1, 4)
    ctx.set_pipeline(abi.PIPELINE_FUSED)
    ctx.update(AXES[3].reshape(9))
    plain = ctx.get_ray_records(n).reshape(-1, 4)
    ctx.close()
    # the atlas both read differs by one update's hysteresis; a sun term is of order one
    assert np.abs(below[:, :3] - plain[:, :3]).max() < 0.1


def test_boxes_ten_thousand_sizes_away(gpu_lib):
    rays, size, far = 256, 0.05, 500.0
    g = abi.make_grid((-500, -500, -500), (500, 500, 500), (2, 2, 2), rays)
    o9 = scenes.random_orientation(5, 1)
    ctx = Context(g)
    ctx.set_light(scenes.default_light())
    ctx.record_hits(True)
    sc = boxes(5, 8 * rays, 1.0, 1.0, (0, 0, 0))
    ctx.build_scene(sc)
    ctx.update(o9)
    d = ctx.get_ray_directions()[:, :3]
    i = np.arange(8)
    origins = np.repeat(np.stack([i % 2, i % 4 // 2, i // 4], -1).astype(np.float32) * 1000 - 500, rays, 0)
    dirs = np.tile(d, (8, 1))
    rng = np.random.default_rng(1)
    inst = sc.instances.copy()
    for k in range(8 * rays):  # a box in the way of every ray
        lin = scenes.yaw_matrix(rng.uniform(0, 6.28)) * size
        inst[k + 1]["transform"] = scenes.affine_3x4(lin, origins[k] + far * rng.uniform(0.5, 1.0) * dirs[k].astype(float))
    ctx.build_scene(scenes.Scene(sc.vertices, sc.indices, sc.meshes, inst, sc.offsets, sc.materials))
    ctx.update(o9)
    got = ctx.get_hits(8).reshape(-1)
    tmax = float(np.sqrt(np.float32(3e6)))
    want, _ = ctx.trace_rays(origins, dirs, float(np.float32(0.01)), tmax, mask=0x3)
    ctx.close()
    assert (want["instance"] != abi.MISS).all()
    for k in ("instance", "primitive", "backface"):
        assert (got[k] == want[k]).all()
    assert (got["t"].view(np.uint32) == want["t"].view(np.uint32)).all()
