"""The persistent walkers (nodes as centre and half extent, packed tests,
leaves held by kind) against the plain traversal over lower and upper planes
(ddgi_trace_rays): the same closest hits bit for bit, on the rays of an update.

Where box tests can go wrong: rays along the axes (a zero direction
component), a grid far larger than the boxes in it (an origin many box sizes
away, in object space too), boxes far from the world's origin, a mesh of one
triangle (a node with a box that is never hit), flat boxes, and ray counts
that leave warps and their leaf phases nearly empty."""
import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context

pytestmark = pytest.mark.gpu


def boxes(seed, n, spread, side, centre, flat=False):
    """n boxes of about `side` within `spread` of `centre`, and one triangle mesh."""
    sc = scenes.room_with_boxes(seed, n)
    rng = np.random.default_rng(seed)
    v = np.zeros(3, abi.VERTEX_DTYPE)
    v["pos"] = [(-1, 0, -1), (1, 0.2, -1), (0, 0.1, 1)]
    v["normal"] = (0, 1, 0)
    meshes = sc.meshes.copy()
    meshes[0] = (len(sc.vertices), 3, sc.indices.size, 3)  # in place of the room
    inst = sc.instances.copy()
    for i in range(len(inst)):
        s = side * rng.uniform(0.2, 1.0, 3)
        if flat and i % 3 == 0:
            s[i % 2] = 0.0 if i == 0 else 1e-6 * side
        if i == 0:
            s = np.full(3, side * 20)
        lin = scenes.yaw_matrix(rng.uniform(0, 6.28) if i % 4 else 0.0) @ np.diag(s)
        inst[i]["transform"] = scenes.affine_3x4(lin, np.asarray(centre) + rng.uniform(-spread, spread, 3))
    return scenes.Scene(np.concatenate([sc.vertices, v]), np.concatenate([sc.indices, np.arange(3, dtype=np.uint32)]),
                        meshes, inst, sc.offsets, sc.materials)


@pytest.mark.parametrize("n,spread,side,centre,extent,rays,mode", [
    (300, 4.0, 1.0, (0, 0, 0), 5.0, 64, "fast_trace"),
    (300, 4.0, 1.0, (0, 0, 0), 5.0, 64, "fast_build"),
    (200, 3.0, 0.05, (0, 0, 0), 500.0, 256, "fast_trace"),  # no ray finds these boxes
    (300, 30.0, 4.0, (0, 0, 0), 500.0, 1024, "fast_trace"),
    (200, 30.0, 2.0, (9000.0, -4000.0, 20000.0), 60.0, 33, "fast_trace"),
    (40, 0.02, 0.01, (1.0, 1.0, 1.0), 3.0, 1024, "fast_trace"),
    (1, 0.5, 1.0, (0, 0, 0), 3.0, 7, "fast_trace"),
])
@pytest.mark.parametrize("axes", [True, False])
def test_walkers_equal_plain_traversal(gpu_lib, n, spread, side, centre, extent, rays, mode, axes):
    sc = boxes(11, n, spread, side, centre, flat=mode == "fast_trace")
    inv = [abs(np.linalg.det(t.reshape(3, 4)[:, :3].astype(np.float64))) for t in sc.instances["transform"]]
    assert min(inv) > 1e-30
    lo = np.asarray(centre, np.float32) - np.float32(extent)
    hi = np.asarray(centre, np.float32) + np.float32(extent)
    g = abi.make_grid(lo, hi, (5, 4, 3), rays)
    ctx = Context(g)
    ctx.set_build_mode(mode)
    ctx.build_scene(sc)
    ctx.set_light(scenes.default_light())
    ctx.record_hits(True)
    # the identity keeps the table's axis-aligned directions as they are
    o9 = np.eye(3, dtype=np.float32).reshape(9) if axes else scenes.random_orientation(5, n)
    ctx.update(o9)
    got = ctx.get_hits(g.probe_count()).reshape(-1)
    f = np.float32
    lo32, hi32 = np.array(list(g.extent_min), f), np.array(list(g.extent_max), f)
    cell = (hi32 - lo32) / np.array([r - 1 for r in g.resolution], f)
    i = np.arange(g.probe_count())
    ijk = np.stack([i % 5, i % 20 // 5, i // 20], -1).astype(f)
    origins = np.repeat(ijk * cell + lo32, rays, 0)
    dirs = np.tile(ctx.get_ray_directions()[:, :3], (g.probe_count(), 1))
    e = hi32 - lo32
    tmax = float(np.sqrt(f(f(e[0] * e[0] + f(e[1] * e[1])) + f(e[2] * e[2]))))
    want, _ = ctx.trace_rays(origins, dirs, float(f(0.01)), tmax, mask=0x3)
    ctx.close()
    hit = want["instance"] != abi.MISS
    assert (got["instance"] == want["instance"]).all()
    assert n < 2 or side < 1e-3 * extent or hit.any()
    for k in ("primitive", "backface"):
        assert (got[k][hit] == want[k][hit]).all()
    assert (got["t"][hit].view(np.uint32) == want["t"][hit].view(np.uint32)).all()
