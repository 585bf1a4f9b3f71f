"""The atlas lookup at the ends of the floats, against the oracle: an atlas of
radiances below the smallest normal number gives radiances of that size, as the
rounded square root and square of the reference do, and the visibility of
probes whose squared distance is near the largest float."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-120, -127, -132, -137])
def test_faint_atlas(gpu_lib, exponent):
    import torch

    g = abi.make_grid((0, 0, 0), (8, 4, 6), (5, 3, 4), 32, 8, 16)
    rng = np.random.default_rng(-exponent)
    ctx = Context(g)
    light = scenes.default_light()
    ctx.set_light(light)
    color = rng.uniform(0.3, 0.9, ctx.atlas_shape(abi.ATLAS_COLOR)).astype(np.float32) * np.float32(2.0 ** exponent)
    depth = rng.uniform(0.9, 2.7, ctx.atlas_shape(abi.ATLAS_DEPTH)).astype(np.float32)
    depth[..., 1] = depth[..., 0] ** 2 * np.float32(1.3)
    ctx.set_atlas(abi.ATLAS_COLOR, color)
    ctx.set_atlas(abi.ATLAS_DEPTH, depth)
    states = np.ones(g.probe_count(), np.uint32)
    ctx.set_probe_states(states)
    n = 4096
    d = rng.normal(size=(n, 3))
    gb = {"position_depth": np.column_stack([rng.uniform(0, (8, 4, 6), (n, 3)), np.ones(n)]),
          "normal_metalness": np.column_stack([d, np.zeros(n)]),
          "albedo_roughness": np.column_stack([np.full((n, 3), 0.7), np.full(n, 0.8)]),
          "emissive": np.zeros((n, 4)), "direct_light": np.zeros(n), "reflection": None}
    gb = {k: None if v is None else v.astype(np.float32) for k, v in gb.items()}
    origin = np.array([3.3, 9.1, -2.7], np.float32)
    dev = {k: None if v is None else torch.from_numpy(v.reshape(1, n, 4) if v.ndim == 2 else v.reshape(1, n)).cuda()
           for k, v in gb.items()}
    out = torch.empty((1, n, 4), dtype=torch.float32, device="cuda")
    ctx.final_gather(dev, origin, out)
    got = out.cpu().numpy().reshape(-1, 4)[:, :3].astype(np.float64)
    ctx.close()
    want = Oracle.final_gather(g, light, states, color, depth, gb, origin)[:, :3].astype(np.float64)
    assert (want > 0).all()
    # the gather's bar, and the spacing of the subnormal numbers: four roundings
    # of the bilinear sum, those of the square, the blend and the two products
    assert (np.abs(got - want) <= 1e-4 * want + 16 * 2.0 ** -149).all()


def test_grid_of_the_largest_cells(gpu_lib):
    # squared distances in a cell above 2^126, below the largest float
    import torch

    e = np.float32(1e19)
    g = abi.make_grid((0, 0, 0), (e, e, e), (2, 2, 2), 32, 8, 16, shadow_bias=0.0)
    rng = np.random.default_rng(4)
    ctx = Context(g)
    light = scenes.default_light()
    ctx.set_light(light)
    color = rng.uniform(0.3, 0.9, ctx.atlas_shape(abi.ATLAS_COLOR)).astype(np.float32)
    depth = np.zeros(ctx.atlas_shape(abi.ATLAS_DEPTH), np.float32)
    depth[..., 0] = rng.uniform(0.05, 0.4, depth.shape[:2]).astype(np.float32) * e
    depth[..., 1] = depth[..., 0] ** 2 + (np.float32(0.8) * e) ** 2 * rng.uniform(0.5, 1, depth.shape[:2])
    ctx.set_atlas(abi.ATLAS_COLOR, color)
    ctx.set_atlas(abi.ATLAS_DEPTH, depth)
    states = np.ones(8, np.uint32)
    ctx.set_probe_states(states)
    n = 4096
    gb = {"position_depth": np.column_stack([rng.uniform(0.1, 0.9, (n, 3)) * e, np.ones(n)]),
          "normal_metalness": np.column_stack([rng.normal(size=(n, 3)), np.zeros(n)]),
          "albedo_roughness": np.column_stack([np.full((n, 3), 0.7), np.full(n, 0.8)]),
          "emissive": np.zeros((n, 4)), "direct_light": np.zeros(n), "reflection": None}
    gb = {k: None if v is None else v.astype(np.float32) for k, v in gb.items()}
    origin = np.array([0.5, 0.5, 0.5], np.float32) * e
    dev = {k: None if v is None else torch.from_numpy(v.reshape(1, n, 4) if v.ndim == 2 else v.reshape(1, n)).cuda()
           for k, v in gb.items()}
    out = torch.empty((1, n, 4), dtype=torch.float32, device="cuda")
    ctx.final_gather(dev, origin, out)
    got = out.cpu().numpy().reshape(-1, 4)[:, :3].astype(np.float64)
    ctx.close()
    want = Oracle.final_gather(g, light, states, color, depth, gb, origin)[:, :3].astype(np.float64)
    assert np.isfinite(want).all() and (want > 0).all()
    assert (np.abs(got - want) <= 1e-4 * np.maximum(want, 1e-2)).all()
