"""The reverse pass through the border copy, the blend and the hysteresis at
the smallest, odd and largest tile sides, against its closed form: with no
geometry every ray returns the sky, so after K updates from a zero atlas every
texel, border texels included, holds (1 - h^K) sky and dL/dsky is
(1 - h^K) times the sum of dL/datlas over all texels.  (Colour tiles of more
than 2,048 interior texels need more shared memory than the blend's reverse
pass asks for: refused with an error, as before.)

Sums of positive float32 terms in a few stages (texels of a tile into rays,
rays into float64): at most 62 x 62 + 1024 roundings of 2^-24 in a row, 3e-4;
they are unbiased, so 1e-4 holds with room."""
import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context, DDGIError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("color_res,depth_res,rays,K", [(3, 3, 33, 1), (4, 5, 64, 3), (7, 9, 100, 2), (8, 16, 256, 3),
                                                        (64, 3, 1024, 1)])
def test_sky_gradient_through_borders(gpu_lib, color_res, depth_res, rays, K):
    full = scenes.room_with_boxes(3, 1)
    empty = scenes.Scene(full.vertices, full.indices, full.meshes, full.instances[:0], full.offsets, full.materials)
    h = 0.75
    g = abi.make_grid((0, 0, 0), (4, 3, 2), (3, 2, 2), rays, color_res, depth_res, hysteresis=h)
    ctx = Context(g)
    ctx.build_scene(empty)
    ctx.set_light(scenes.default_light())
    ctx.forward_record(np.stack([scenes.random_orientation(9, k) for k in range(K)]), 2)
    G = np.random.default_rng(color_res).uniform(0.1, 1.0, ctx.atlas_shape(abi.ATLAS_COLOR)).astype(np.float32)
    if (color_res - 2) ** 2 > 2048:
        with pytest.raises(DDGIError):
            ctx.backward(G, len(empty.materials))
        ctx.close()
        return
    albedo, sun, sky = ctx.backward(G, len(empty.materials))
    ctx.close()
    want = (1.0 - h ** K) * G[..., :3].astype(np.float64).sum((0, 1))
    assert np.abs(sky - want).max() <= 1e-4 * want.max()
    assert not albedo.any() and not sun.any()
