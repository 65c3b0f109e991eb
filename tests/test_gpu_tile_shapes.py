"""Every CTA size of the cost volume's tile form gives the oracle's bits: with the targets in turn in
a CTA and side by side, and with five to eight targets to aggregate (test_gpu_cost_forms.py has more)."""
import numpy as np
import pytest

from chiaro_b200 import scenes
from chiaro_b200.depth import DepthOptions, output_shape, refine_multiview_depth

pytestmark = pytest.mark.gpu

KEYS = ("coarse_scores", "coarse_costs", "coarse_guidance", "coarse_tested")


def make(width, height, sources, planes):
    from oracle import oracle
    opt = DepthOptions(grid_step=8, planes=planes, patch_radius=3, near_depth=400.0, far_depth=25000.0,
                       minimum_support=2, best_view_count=3)
    sc = scenes.make_scene("shapes", width, height, sources, 5, 1, (500.0, 8000.0), (20.0, 60.0), 0.4, opt, 3,
                           distortion=True, focal_px=1200.0)
    (columns, rows, _), (cc, cr, _) = output_shape(width, height, opt)
    assert cc * cr * sources * (planes + 1) >= 600_000  # hypotheses from which tiles pay
    expected = oracle.debug_buffers(sources + 1, cc * cr, planes + 1, columns * rows)
    oracle.refine_multiview_depth(sc.inputs(), 0, sc.alignments(), opt, threads=8, debug=expected)
    return sc, expected


def check(context, case):
    from oracle import oracle
    sc, expected = case
    (columns, rows, _), (cc, cr, _) = output_shape(sc.width, sc.height, sc.options)
    got = oracle.debug_buffers(len(sc.cameras), cc * cr, sc.options.planes + 1, columns * rows)
    refine_multiview_depth(sc.inputs(), 0, sc.alignments(), sc.options, context=context, debug=got)
    assert expected["coarse_tested"].any()
    for key in KEYS:
        assert np.array_equal(got[key].view(np.uint8), expected[key].view(np.uint8)), key


@pytest.fixture(scope="module", params=[(700, 520, 3, 64), (1010, 650, 2, 40)], ids=["side by side", "in turn"])
def case(request):
    return make(*request.param)


@pytest.mark.parametrize("threads", [64, 96, 128, 160, 192])
def test_every_shape_of_the_tiles(case, threads):
    from chiaro_b200.runtime import DepthContext
    context = DepthContext(0)
    try:
        context.set_autotune(threads)
        check(context, case)
    finally:
        context.close()


@pytest.mark.parametrize("sources", [5, 6, 8])
def test_targets_to_aggregate(gpu_ctx, sources):
    check(gpu_ctx, make(690, 470, sources, 30))
