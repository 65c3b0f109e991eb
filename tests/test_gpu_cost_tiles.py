"""The cost volume's node tiles against the oracle, bit for bit, where they can go wrong:
grids that no tile divides, one node column or row, few and many labels (every tile size and
labels scored in several parts), epipolar lines near either axis (samples stored by rows or by
columns), an odd step (no tap lattice), a patch larger than the default, and planes so small
that they take the form without tiles."""
import numpy as np
import pytest

from chiaro_b200 import scenes
from chiaro_b200.depth import DepthOptions, output_shape, refine_multiview_depth

pytestmark = pytest.mark.gpu

CASES = {
    "odd grid, one target": dict(width=322, height=251, sources=1, planes=24, step=8, radius=4, focal=None),
    # narrower than its patches: no node can be tested
    "narrow": dict(width=18, height=420, sources=2, planes=16, step=8, radius=2, focal=None, tested=False),
    "tall": dict(width=90, height=420, sources=2, planes=16, step=8, radius=2, focal=600.0),
    "odd step": dict(width=331, height=220, sources=3, planes=70, step=9, radius=3, focal=None),
    "long reach": dict(width=560, height=430, sources=4, planes=128, step=8, radius=4, focal=2400.0),
    "large patch": dict(width=400, height=300, sources=2, planes=20, step=12, radius=9, focal=1500.0),
    # planes of at least 320 pixels and 600,000 hypotheses: node tiles
    "tiles, one target": dict(width=851, height=662, sources=1, planes=80, step=8, radius=4, focal=None),
    "tiles, odd step": dict(width=433, height=845, sources=3, planes=70, step=9, radius=3, focal=None),
    "tiles, long reach": dict(width=700, height=500, sources=4, planes=128, step=8, radius=4, focal=2400.0),
    "tiles, fine grid": dict(width=642, height=480, sources=2, planes=30, step=4, radius=2, focal=1500.0),
    "tiles, large patch": dict(width=640, height=400, sources=3, planes=110, step=12, radius=9, focal=1500.0),
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("seed", [3, 4])
def test_cost_volume_of_tiles_is_the_oracles(gpu_ctx, name, seed):
    from oracle import oracle
    c = CASES[name]
    support = 1 if c["sources"] == 1 else 2
    opt = DepthOptions(grid_step=c["step"], planes=c["planes"], patch_radius=c["radius"], near_depth=400.0,
                       far_depth=25000.0, minimum_support=support, best_view_count=max(support, 3))
    sc = scenes.make_scene("tiles", c["width"], c["height"], c["sources"], 5, 1, (500.0, 8000.0), (20.0, 60.0), 0.4, opt,
                           seed, distortion=True, focal_px=c["focal"])
    (columns, rows, _), (cc, cr, _) = output_shape(sc.width, sc.height, opt)
    expected = oracle.debug_buffers(len(sc.cameras), cc * cr, opt.planes + 1, columns * rows)
    oracle.refine_multiview_depth(sc.inputs(), 0, sc.alignments(), opt, threads=8, debug=expected)
    got = oracle.debug_buffers(len(sc.cameras), cc * cr, opt.planes + 1, columns * rows)
    refine_multiview_depth(sc.inputs(), 0, sc.alignments(), opt, context=gpu_ctx, debug=got)
    assert expected["coarse_tested"].any() == c.get("tested", True)
    for key in ("coarse_scores", "coarse_costs", "coarse_guidance", "coarse_tested"):
        assert np.array_equal(got[key].view(np.uint8), expected[key].view(np.uint8)), key
