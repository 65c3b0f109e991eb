"""The cost volume's forms side by side (GPU): node by node on small planes and grids, in node
tiles on the others, with the targets in turn or side by side (launch_cost). Each is tuned by
itself."""
import numpy as np
import pytest

from chiaro_b200 import scenes
from chiaro_b200.depth import DepthOptions, output_shape, refine_multiview_depth

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from chiaro_b200.runtime import DepthContext
    c = DepthContext(0)
    yield c
    c.close()


def make_case(width, height, sources, planes, seed=3, step=8, radius=4, focal=None, support=None):
    support = support or (1 if sources == 1 else 2)
    opt = DepthOptions(grid_step=step, planes=planes, patch_radius=radius, near_depth=400.0, far_depth=25000.0,
                       minimum_support=support, best_view_count=max(support, 3))
    return scenes.make_scene("forms", width, height, sources, 5, 1, (500.0, 8000.0), (20.0, 60.0), 0.4, opt, seed,
                             distortion=True, focal_px=focal)


def run(ctx, scene, debug=None):
    alignments = scene.alignments()
    dmap = refine_multiview_depth(scene.inputs(), 0, alignments, scene.options, context=ctx, debug=debug)
    assert dmap is not None
    return dmap, alignments


def compare_with_the_oracle(ctx, scene, direct=False):
    """Runs the stage and compares its cost volume (and its direct pass) with the oracle's, bit
    for bit; returns the oracle's flags of the nodes that scored."""
    from oracle import oracle
    (columns, rows, _), (cc, cr, _) = output_shape(scene.width, scene.height, scene.options)
    views = len(scene.cameras)
    got, expected = (oracle.debug_buffers(views, cc * cr, scene.options.planes + 1, columns * rows) for _ in range(2))
    run(ctx, scene, got)
    oracle.refine_multiview_depth(scene.inputs(), 0, scene.alignments(), scene.options, threads=8, debug=expected)
    keys = ["coarse_scores", "coarse_costs", "coarse_guidance", "coarse_tested"]
    if direct:
        keys += ["direct_has", "direct_tested", "direct_guidance"]
        has = expected["direct_has"] == 1
        for key in ("direct_depth", "direct_confidence", "direct_improvement"):
            assert np.array_equal(got[key][has].view(np.uint8), expected[key][has].view(np.uint8)), key
    for key in keys:
        assert np.array_equal(got[key].view(np.uint8), expected[key].view(np.uint8)), key
    return expected["coarse_tested"]


# (both of at least 4096 nodes, with one target and 65 labels)
@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
def test_the_forms_of_a_bucket_are_tuned_apart(ctx, order):
    rasters = [(723, 531), (1000, 700)]  # below and above the 600,000 hypotheses from which tiles pay
    for n, i in enumerate(order):
        width, height = rasters[i]
        run(ctx, make_case(width, height, 1, 64))
        assert int(ctx.lib.chiaro_depth_tuning(ctx.handle, None, None, 0)) == n + 1
        assert list(ctx.tuning()) == [(1, 65, 4)]  # the reported key is the bucket's


# The segments' sum in samples is some 470 and 6200 here.
def test_segments_far_beyond_the_reach_go_node_by_node(ctx):
    """Two lenses, one bucket and raster: the long lens spreads the labels far beyond a
    hypothesis's reach and takes the other form, which is timed by itself. Both are the oracle's."""
    for n, focal in enumerate((2500.0, 15000.0)):
        scene = make_case(700, 520, 4, 96, focal=focal)
        assert compare_with_the_oracle(ctx, scene).any()
        assert int(ctx.lib.chiaro_depth_tuning(ctx.handle, None, None, 0)) == n + 1


# No sample position is taken in f32 beyond a luminance side of 8192. With three targets the grid of
# 164,000 fine nodes is large enough for the wide retry to read its taps from the lattice.
@pytest.mark.parametrize("width,sources", [(16384, 1), (16384, 3), (16400, 3)])
def test_planes_beyond_the_f32_positions(ctx, width, sources):
    scene = make_case(width, 150, sources, 16, radius=3, focal=3000.0)
    assert compare_with_the_oracle(ctx, scene, direct=True).any()


@pytest.mark.parametrize("width,height,sources,planes", [(700, 520, 2, 96), (700, 520, 4, 96), (700, 520, 12, 30),
                                                        (1000, 700, 9, 33)])
def test_tiles_hold_no_scratch_of_their_own(width, height, sources, planes):
    """The same call with a lens that takes the tiles and with one that does not: the tiles add the
    nodes' reference patches (24 bytes each) and at most a copy of the targets' planes, and go in
    several launches from eight targets on, side by side (700x520) or in turn."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from chiaro_b200.runtime import DepthContext
    from oracle import oracle
    held = []
    for focal in (1200.0, 15000.0):
        scene = make_case(width, height, sources, planes, focal=focal)
        context = DepthContext(0)
        try:
            if not held:
                assert compare_with_the_oracle(context, scene).any()
            else:  # with the same debug outputs
                (columns, rows, _), (cc, cr, _) = output_shape(width, height, scene.options)
                run(context, scene, oracle.debug_buffers(sources + 1, cc * cr, planes + 1, columns * rows))
            held.append(context.memory_held())
        finally:
            context.close()
    _, (cc, cr, _) = output_shape(width, height, scene.options)
    assert 0 < held[0] - held[1] <= 24 * cc * cr + sources * 4 * (width // 2 + 3) * (height // 2 + 3)


@pytest.mark.parametrize("sources", [2, 9])
def test_a_limit_that_holds_the_other_form_is_enough(sources):
    """A context whose memory limit holds the call node by node answers it, with the same bits, first
    and again, after a call of another size took the tiles, and in tiles when the limit is lifted."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from chiaro_b200.runtime import DepthContext
    tiled, nodewise = (make_case(1000, 700, sources, 40, focal=focal) for focal in (1200.0, 15000.0))
    smaller = make_case(900, 640, sources, 40, focal=1200.0)
    results, held = [], []
    for scene, limit in ((nodewise, False), (tiled, False), (tiled, True)):
        context = DepthContext(0)
        try:
            if limit:
                context.set_memory_limit(held[0])
                run(context, smaller)
            for _ in range(2 if limit else 1):
                results.append(run(context, scene)[0])
            held.append(context.memory_held())
            if limit:
                assert held[-1] <= held[0]
                context.set_memory_limit(0)
                results.append(run(context, scene)[0])
                assert context.memory_held() > held[0]
        finally:
            context.close()
    assert held[1] > held[0]
    for other in results[2:]:
        assert np.array_equal(other.depth.view(np.uint64), results[1].depth.view(np.uint64))
        assert np.array_equal(other.confidence.view(np.uint32), results[1].confidence.view(np.uint32))


# 700x520: a CTA per target and a kernel that joins them
@pytest.mark.parametrize("width,height,sources,planes", [(700, 520, 2, 96), (331, 250, 2, 24)])
def test_a_replay_reports_the_launches_it_holds(ctx, width, height, sources, planes):
    from chiaro_b200.depth import DeviceStage
    scene = make_case(width, height, sources, planes)
    stage = DeviceStage(scene.inputs(), 0, scene.alignments(), scene.options, context=ctx)
    stage.graph = True
    launches = []
    for state in (0, 1, 2):  # launched, captured, replayed
        assert stage() and stage.graph_state == state
        launches.append(ctx.launches())
    assert len(set(launches)) == 1
