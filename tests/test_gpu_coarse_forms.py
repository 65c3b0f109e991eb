"""The coarse search on grids large enough for the cost volume's node tiles, against the oracle bit
for bit: the plain search, and the fallback windows of the banded one, in tiles over the windows'
node list or, where the windows are small, node by node."""
import numpy as np
import pytest

from chiaro_b200 import scenes
from chiaro_b200.band import centred_offsets, tiles_of
from chiaro_b200.coarse import BandOptions, coarse_depth, sample_labels
from chiaro_b200.depth import DepthOptions, DeviceStage, output_shape

pytestmark = pytest.mark.gpu

TILE_ITEMS = 600_000  # hypotheses from which a cost volume runs in tiles


@pytest.fixture(scope="module", params=[(700, 520, 3, 8), (699, 521, 5, 9)])
def case(request):
    """Step 9 has no tap lattice."""
    from oracle import oracle
    width, height, sources, step = request.param
    opt = DepthOptions(grid_step=step, planes=56, patch_radius=4, near_depth=400.0, far_depth=25000.0,
                       minimum_support=2, best_view_count=3)
    sc = scenes.make_scene("coarse", width, height, sources, 5, 1, (500.0, 8000.0), (20.0, 60.0), 0.4, opt, 3,
                           distortion=True, focal_px=1200.0)
    (columns, rows, _), (cc, cr, _) = output_shape(width, height, opt)
    dbg = oracle.debug_buffers(len(sc.cameras), cc * cr, opt.planes + 1, columns * rows)
    oracle.refine_multiview_depth(sc.inputs(), 0, sc.alignments(), opt, threads=8, debug=dbg)
    return sc, dbg, cc, cr, opt.planes + 1, sources


def test_plain_search_in_tiles(gpu_ctx, case):
    sc, dbg, cc, cr, d, sources = case
    assert cc * cr * d * sources >= TILE_ITEMS
    r = coarse_depth(DeviceStage(sc.inputs(), 0, sc.alignments(), sc.options, context=gpu_ctx))
    reg = dbg["regularised"].reshape(cc * cr, d)
    assert np.array_equal(r.winner.cpu().numpy(), 1 + np.argmin(reg[:, 1:], axis=1))
    assert np.array_equal(r.tested.cpu().numpy(), dbg["coarse_tested"])


@pytest.mark.parametrize("tile,band,margin,tiled", [(4, 12, 8, True), (4, 12, 60, True), (2, 32, 1, False)])
def test_fallback_windows_in_either_form(gpu_ctx, case, tile, band, margin, tiled):
    from test_gpu_coarse import _oracle_banded
    sc, dbg, cc, cr, d, sources = case
    stage = DeviceStage(sc.inputs(), 0, sc.alignments(), sc.options, context=gpu_ctx)
    r = coarse_depth(stage, BandOptions(None, tile, band, margin, 1.0))
    sampled = np.array(sample_labels(d))
    lowest = sampled[np.argmin(dbg["coarse_costs"].reshape(cc * cr, d)[:, sampled], axis=1)].reshape(cr, cc)
    tx, ty = tiles_of(cc, cr, tile)
    centres = np.array([np.median(lowest[y * tile:(y + 1) * tile, x * tile:(x + 1) * tile])
                        for y in range(ty) for x in range(tx)])
    offsets = centred_offsets(centres, d, band)
    assert np.array_equal(r.offsets.cpu().numpy(), offsets)
    winner, fallback = _oracle_banded(dbg, cc, cr, d, offsets, tile, band, margin)
    assert np.array_equal(r.fallback.cpu().numpy(), fallback)
    assert np.array_equal(r.winner.cpu().numpy(), winner)
    items = r.report["window_nodes"] * d * sources
    assert (items >= TILE_ITEMS) == tiled and items > 0


def test_small_windows_make_no_tile_buffers(case):
    """A few windows of a large grid go node by node: the plain search that follows on the context
    makes the tiles' patches and planes beside its own volumes and paths."""
    from chiaro_b200.runtime import DepthContext
    sc, _, cc, cr, d, sources = case
    context = DepthContext(0)
    try:
        stage = DeviceStage(sc.inputs(), 0, sc.alignments(), sc.options, context=context)
        assert 0 < coarse_depth(stage, BandOptions(None, 2, 32, 1, 1.0)).report["window_nodes"] * d * sources < TILE_ITEMS
        before = context.memory_held()
        coarse_depth(stage)
        own = 4 * (3 * cc * cr * d + 8 * ((cc * cr * d + 63) // 64 * 64))
        planes = sources * 4 * (sc.width // 2) * (sc.height // 2)
        assert context.memory_held() - before >= own + 24 * cc * cr + planes
    finally:
        context.close()
