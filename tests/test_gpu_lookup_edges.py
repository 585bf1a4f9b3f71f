"""The atlas lookup (final gather) where its coordinates can go wrong, against
the oracle: directions along the axes and in their planes (where the
octahedral fold meets a zero component), positions on probes, on cell faces
and on and past the grid's limits, probes that are off, tiles whose side is
not a power of two, one-cell grids.  Bar of the gather tests: 1e-4 relative
(floor 1e-2)."""
import itertools

import numpy as np
import pytest

from conftest import rel_err
from oracle.oracle import Oracle
from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_FP32, abi.PRECISION_BF16])
@pytest.mark.parametrize("res,tiles", [((2, 2, 2), (8, 16)), ((5, 3, 4), (6, 14)), ((4, 4, 4), (3, 3)), ((3, 2, 7), (7, 9))])
def test_lookup_edges(gpu_lib, precision, res, tiles):
    import torch

    g = abi.make_grid((0, 0, 0), (8, 4, 6), res, 32, *tiles, precision=precision)
    rng = np.random.default_rng(sum(res))
    ctx = Context(g)
    light = scenes.default_light()
    ctx.set_light(light)
    for kind in (abi.ATLAS_COLOR, abi.ATLAS_DEPTH):
        a = rng.uniform(0.3, 0.9, ctx.atlas_shape(kind)).astype(np.float16).astype(np.float32)
        if kind == abi.ATLAS_DEPTH:  # mean, and a mean square with some variance
            a[..., 0] *= 3.0
            a[..., 1] = a[..., 0] ** 2 * 1.3
            a = a.astype(np.float16).astype(np.float32)
        ctx.set_atlas(kind, a)
    states = rng.choice(np.array([0, 1, 8], np.uint32), size=g.probe_count(), p=[0.2, 0.4, 0.4]).astype(np.uint32)
    ctx.set_probe_states(states)
    ext = np.array([8.0, 4.0, 6.0])
    steps = [np.unique(np.concatenate([np.linspace(0, e, r), [e / 3, e + 0.5, -0.25]])) for e, r in zip(ext, res)]
    pos = np.array(list(itertools.product(*steps)), np.float64)
    dirs = np.array([d for d in itertools.product((-1, 0, 1), repeat=3) if any(d)], np.float64)
    n = len(pos) * len(dirs)
    P, D = np.repeat(pos, len(dirs), 0), np.tile(dirs, (len(pos), 1))
    z, one = np.zeros(n), np.ones(n)
    gb = {"position_depth": np.column_stack([P, one]), "normal_metalness": np.column_stack([D, z]),
          "albedo_roughness": np.column_stack([np.full((n, 3), 0.7), 0.8 * one]),
          "emissive": np.zeros((n, 4)), "direct_light": z, "reflection": None}
    gb = {k: None if v is None else v.astype(np.float32) for k, v in gb.items()}
    origin = np.array([3.3, 9.1, -2.7], np.float32)
    dev = {k: None if v is None else torch.from_numpy(v.reshape(1, n, 4) if v.ndim == 2 else v.reshape(1, n)).cuda()
           for k, v in gb.items()}
    out = torch.empty((1, n, 4), dtype=torch.float32, device="cuda")
    ctx.final_gather(dev, origin, out)
    got = out.cpu().numpy().reshape(-1, 4)
    want = Oracle.final_gather(g, light, states, ctx.get_atlas(abi.ATLAS_COLOR), ctx.get_atlas(abi.ATLAS_DEPTH), gb,
                               origin)
    ctx.close()
    assert np.isfinite(got).all()
    err = rel_err(got[:, :3], want[:, :3], 1e-2)
    assert err.max() <= 1e-4, "max rel err %.3g" % err.max()
