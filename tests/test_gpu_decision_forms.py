"""The decisions' forms against the oracle, bit for bit: pooled (one and two targets) or a warp a
node, four or nine taps in flight, on either side of the slot size and patch from which nine are
taken (target_decision_kernel)."""
import numpy as np
import pytest

from chiaro_b200 import scenes
from chiaro_b200.depth import DepthOptions, output_shape, refine_multiview_depth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sources,radius", [(1, 4), (1, 8), (2, 4), (2, 6), (3, 4), (3, 5), (4, 3), (4, 4), (9, 2), (9, 4)])
def test_decisions_are_the_oracles(gpu_ctx, sources, radius):
    from oracle import oracle
    support = 1 if sources == 1 else 2
    opt = DepthOptions(grid_step=8, planes=24, patch_radius=radius, near_depth=400.0, far_depth=25000.0,
                       minimum_support=support, best_view_count=max(support, 3))
    sc = scenes.make_scene("decisions", 331, 250, sources, 5, 1, (500.0, 8000.0), (20.0, 60.0), 0.4, opt, 3,
                           distortion=True)
    (columns, rows, _), (cc, cr, _) = output_shape(sc.width, sc.height, opt)
    got, expected = (oracle.debug_buffers(sources + 1, cc * cr, opt.planes + 1, columns * rows) for _ in range(2))
    al_got, al_expected = sc.alignments(), sc.alignments()
    assert refine_multiview_depth(sc.inputs(), 0, al_got, opt, context=gpu_ctx, debug=got) is not None
    ref = oracle.refine_multiview_depth(sc.inputs(), 0, al_expected, opt, threads=8, debug=expected)
    assert np.array_equal(got["decision_kind"], expected["decision_kind"])
    assert len(set(expected["decision_kind"].tolist())) >= 3
    for t in range(1, sources + 1):
        assert np.array_equal(al_got[t].warp.points.reshape(-1).view(np.uint32), ref["points"][t].view(np.uint32))
        assert np.array_equal(al_got[t].warp.confidence.view(np.uint32), ref["warp_confidence"][t].view(np.uint32))
