"""Front-hit shading with four, two and one lanes per hit, chosen by the number
of records: the first n probes updated by themselves must equal the same probes
of an update of all 8,000 (one lane per hit) from the same atlas.

Numbers of records on both sides of the choice's lines (97,280 resident threads
on 152 multiprocessors: a third of them, three quarters with a 16-bit atlas,
sixteen times them with a 32-bit one).  The lookups' sums are the same bit for
bit; what is left are the few multiply-adds that the compiler may contract
differently in two kernels, each within 2^-24 of values of order one, blended
over 256 rays: 1e-5 relative (floor 1e-2), one unit in the last place of the
published 16-bit atlas (2^-10 relative)."""
import numpy as np
import pytest

from vulkanexp_gb300 import abi, scenes
from vulkanexp_gb300.ddgi import Context
from test_gpu_blend_tile import RES, by_probe

pytestmark = pytest.mark.gpu

RAYS = 256


def updates(precision, n):
    w = scenes.workload(0)
    g = abi.make_grid(w.grid.extent_min, w.grid.extent_max, RES, RAYS, 8, 16, hysteresis=0.5, depth_sharpness=50.0,
                      precision=precision)
    ctx = Context(g)
    ctx.build_scene(w.scene)
    ctx.set_light(w.light)
    ctx.update(w.orientation(0))
    ctx.update(w.orientation(1), None if n is None else np.arange(n, dtype=np.uint32))
    out = (by_probe(ctx.get_atlas(abi.ATLAS_COLOR), 8), by_probe(ctx.get_atlas(abi.ATLAS_DEPTH), 16),
           ctx.get_probe_states())
    ctx.close()
    return out


@pytest.fixture(scope="module")
def whole(gpu_lib):
    return {p: updates(p, None) for p in (abi.PRECISION_FP32, abi.PRECISION_BF16)}


@pytest.mark.parametrize("precision,n", [(abi.PRECISION_FP32, n) for n in (1, 126, 127, 6080, 6081)] +
                         [(abi.PRECISION_BF16, n) for n in (1, 126, 127, 285, 286)])
def test_lanes_per_hit_agree(whole, precision, n):
    tol = 1e-5 if precision == abi.PRECISION_FP32 else 2.0 ** -10
    got, want = updates(precision, n), whole[precision]
    for a, b in zip(got[:2], want[:2]):
        assert (np.abs(a[:n] - b[:n]) <= tol * np.maximum(np.abs(b[:n]), 1e-2)).all()
    assert np.array_equal(got[2][:n], want[2][:n])
