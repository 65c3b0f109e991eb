"""The direct pass and its wide retry against the oracle, bit for bit, over the forms of the
retry's taps: copied (one and two targets; an odd step, which has no tap lattice; the largest
patch) and read from the lattice (three targets and more), on planes on either side of the size
from which correlations take the f32 sample positions."""
import numpy as np
import pytest

from chiaro_b200 import scenes
from chiaro_b200.depth import DepthOptions, output_shape, refine_multiview_depth

pytestmark = pytest.mark.gpu

CASES = {
    "one target": dict(width=322, height=251, sources=1, step=8, radius=4),
    "two targets": dict(width=842, height=331, sources=2, step=8, radius=4),
    "three targets": dict(width=331, height=250, sources=3, step=8, radius=4),
    "three targets, f32 positions": dict(width=842, height=331, sources=3, step=8, radius=3),
    "four targets, wide patch": dict(width=830, height=300, sources=4, step=12, radius=6),
    "four targets, odd step": dict(width=333, height=420, sources=4, step=9, radius=4),
    "five targets, fine grid": dict(width=402, height=300, sources=5, step=4, radius=2),
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("seed", [3, 4])
def test_direct_pass_is_the_oracles(gpu_ctx, name, seed):
    from oracle import oracle
    c = CASES[name]
    support = 1 if c["sources"] == 1 else 2
    opt = DepthOptions(grid_step=c["step"], planes=24, patch_radius=c["radius"], near_depth=400.0, far_depth=25000.0,
                       minimum_support=support, best_view_count=max(support, 3))
    sc = scenes.make_scene("wide", c["width"], c["height"], c["sources"], 5, 1, (500.0, 8000.0), (20.0, 60.0), 0.4, opt,
                           seed, distortion=True, focal_px=None)
    (columns, rows, _), (cc, cr, _) = output_shape(sc.width, sc.height, opt)
    buffers = [oracle.debug_buffers(len(sc.cameras), cc * cr, opt.planes + 1, columns * rows) for _ in range(2)]
    oracle.refine_multiview_depth(sc.inputs(), 0, sc.alignments(), opt, threads=8, debug=buffers[0])
    refine_multiview_depth(sc.inputs(), 0, sc.alignments(), opt, context=gpu_ctx, debug=buffers[1])
    has = buffers[0]["direct_has"] == 1
    assert has.any()
    for key in ("direct_has", "direct_tested", "direct_guidance"):
        assert np.array_equal(buffers[1][key].view(np.uint8), buffers[0][key].view(np.uint8)), key
    for key in ("direct_depth", "direct_confidence", "direct_improvement"):
        assert np.array_equal(buffers[1][key][has].view(np.uint8), buffers[0][key][has].view(np.uint8)), key
