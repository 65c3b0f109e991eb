"""The work that users of this package have it do, as cases that can be timed.

Every case is a call (or the few calls a program makes in a row) of the package's public
entry points, at sizes of the synthetic workloads in ``chiaro_b200.scenes`` or between
them. ``listed()`` names the standing cases, ``draw(rng)`` gives further ones of the same
ranges, ``prepare(case, seed)`` makes what a program holds before the call, ``run(state)``
is one pass, ``work(case)`` the bytes and operations a pass cannot do without, and
``exact(case, seed)`` the pass's results in 64 bits where they are plain arithmetic (the
depth stage's results are decisions between scores, which have no such value).

The kinds of case:

* ``stage``  - the depth stage on planes that live in device memory (``DeviceStage``): a
  service that keeps its frames there. With ``graph`` the stage replays its CUDA graph.
* ``call``   - ``refine_multiview_depth`` on host arrays: the drop-in call of a program
  that has its planes in host memory, copies both ways included.
* ``coarse`` - the coarse search alone (``coarse_depth``), plain or with the trained band
  network, as the band's training and a preview use it.
* ``sgm``    - the semi-global matching of one capture's groupings as a batch.
* ``module`` - what a capture does per module around the stage: the log-luminance of both
  mosaics, the global alignment and the resolution-domain refinement.
* ``train``  - loss and gradient of the band network over a batch of images (its forward
  and backward pass).
"""
import ctypes as C
import math
from pathlib import Path

import numpy as np
import torch

from chiaro_b200 import abi, scenes
from chiaro_b200.align import AlignInput, AlignOptions, align_module
from chiaro_b200.bandnet import CH, LAYERS, TAPS, BandNet, Sample
from chiaro_b200.coarse import BandOptions, coarse_depth, sample_labels
from chiaro_b200.depth import DepthOptions, DeviceStage, output_shape, refine_multiview_depth
from chiaro_b200.image import Mosaic, VignettingMesh
from chiaro_b200.resolution import refine_resolution_warp
from chiaro_b200.runtime import DepthContext, default_context

WEIGHTS = Path(scenes.__file__).resolve().parent / "weights" / "bandnet.bin"
DEVICE = "cuda:0"


def _stage(name, width, height, sources, planes, kind="stage", mirrored=False, tele=False, grid_step=8, radius=4,
           graph=False, band=False):
    """A depth case. ``tele``: modules resampled to the wide modules' angular pixel size (a
    narrow field of view at full focal length); ``mirrored``: modules behind fold mirrors."""
    case = dict(kind=kind, width=width, height=height, sources=sources, planes=planes, mirrored=mirrored, tele=tele,
                grid_step=grid_step, radius=radius)
    if kind == "stage":
        case["graph"] = graph
    if kind == "coarse":
        case["band"] = band
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the five wide modules of a 16-module capture at full size: the headline workload
        _stage("stage_five_view", 4160, 3120, 4, 128),
        # one stereo pair: the reference's CPU-sized configuration
        _stage("stage_two_view", 1040, 780, 1, 64),
        # tele grouping behind mirrors with an odd raster and many planes
        _stage("stage_tele_odd", 1567, 1173, 3, 192, mirrored=True, tele=True),
        # mid grouping searched on the direct pass's own grid, with a small patch
        _stage("stage_fine_grid", 2080, 1560, 2, 64, tele=True, grid_step=4, radius=3),
        # a small grouping of a stream, replayed from the stage's CUDA graph
        _stage("stage_graph_small", 1040, 780, 2, 64, mirrored=True, tele=True, graph=True),
        # the smallest calls: a thumbnail-sized preview from host memory
        _stage("call_small", 320, 240, 2, 24, kind="call"),
        # a mid grouping from host memory, copies included
        _stage("call_mid", 3120, 2340, 3, 64, kind="call", mirrored=True, tele=True),
        # the coarse search alone, all labels
        _stage("coarse_plain", 2080, 1560, 3, 192, kind="coarse", mirrored=True, tele=True),
        # the coarse search with the trained band network, at the size it was trained for
        _stage("coarse_band", 1040, 780, 4, 192, kind="coarse", band=True),
        # the semi-global matching of one capture's ten groupings
        dict(name="sgm_capture", kind="sgm", scale=1.0, instances=10),
        # luminance, alignment and refinement of one full-size module
        dict(name="module_chain", kind="module", width=4160, height=3120, mesh=True),
        # one gradient of the band network over a training batch
        dict(name="band_gradient", kind="train", columns=131, rows=99, labels=193, images=16),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["stage"] * 5 + ["call", "call", "coarse", "coarse", "sgm", "module", "train"])
    if kind == "sgm":
        return dict(kind=kind, scale=round(math.exp(rng.uniform(math.log(0.1), 0.0)), 4), instances=rng.randint(1, 10))
    if kind == "module":
        width = spread(320, 4160)
        return dict(kind=kind, width=width, height=int(width * rng.uniform(0.6, 0.8)), mesh=rng.random() < 0.5)
    if kind == "train":
        return dict(kind=kind, columns=spread(24, 160), rows=spread(24, 120), labels=rng.randint(33, 193),
                    images=rng.randint(1, 16))
    width = spread(240, 2600)
    height = int(width * rng.uniform(0.6, 0.85))
    fine = width < 1300 and rng.random() < 0.25
    case = _stage(None, width, height, rng.choice([1, 2, 2, 3, 3, 4, 4, 5]), rng.choice([24, 48, 64, 96, 128, 192])
                  + rng.choice([0, 0, 1, 5]), kind=kind, mirrored=rng.random() < 0.4, tele=rng.random() < 0.5,
                  grid_step=rng.choice([4, 6]) if fine else rng.choice([8, 8, 8, 9, 12]), radius=rng.choice([4, 4, 4, 3, 2]))
    if kind == "stage":
        case["graph"] = rng.random() < 0.2
    if kind == "coarse":
        case["band"] = case["planes"] >= 64 and rng.random() < 0.5
    return case


# ---- inputs ---------------------------------------------------------------------------
def _options(case):
    single = case["sources"] == 1  # one source never reaches the default support of two
    return DepthOptions(grid_step=case["grid_step"], planes=case["planes"], patch_radius=case["radius"],
                        near_depth=400.0, far_depth=25000.0 if single else 50000.0,
                        minimum_support=1 if single else 2, best_view_count=1 if single else 3)


def _scene(case, seed):
    """A rendered capture: slanted textured planes and spheres seen by every module, with
    distortion, small rotations, 20-60 mm baselines and sensor noise."""
    n = case["sources"]
    mirrors = {i: (i + seed) % 2 == 0 for i in range(n + 1)} if case["mirrored"] else {}
    focal = scenes.FOCAL_MM / scenes.PIXEL_PITCH_MM if case["tele"] else None
    return scenes.make_scene("perf", case["width"], case["height"], n, 12, 3, (500.0, 20000.0), (20.0, 60.0), 0.5,
                             _options(case), seed, distortion=True, mirrors=mirrors, render_device=DEVICE,
                             focal_px=focal)


def _sgm_shapes(case):
    """The coarse grids of a capture's groupings, their rasters scaled."""
    groupings = scenes.CAPTURE_GROUPINGS[10 - case["instances"]:]
    return [(-(-int(w * case["scale"]) // 8) + 1, -(-int(h * case["scale"]) // 8) + 1, planes + 1)
            for w, h, planes, _, _ in groupings]


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _volume(gen, columns, rows, labels):
    """A cost volume like the stage's: a valley around each node's label over a smooth
    surface, noise, and missing costs (2.25) at some nodes' labels; log-luminance guidance."""
    y = torch.linspace(0, 6.0, rows, device=DEVICE)[:, None]
    x = torch.linspace(0, 9.0, columns, device=DEVICE)[None, :]
    phase = torch.rand(4, generator=gen, device=DEVICE) * 6.28
    centre = (0.5 + 0.2 * torch.sin(x + phase[0]) + 0.2 * torch.cos(y + phase[1])) * labels
    at = torch.arange(labels, device=DEVICE, dtype=torch.float32)
    costs = (at[None, None, :] - centre[:, :, None]).abs().mul_(1.0 / 24.0).clamp_(max=1.0)
    costs.add_(torch.rand(costs.shape, generator=gen, device=DEVICE), alpha=0.4)
    costs[torch.rand(costs.shape, generator=gen, device=DEVICE) < 0.05] = 2.25
    guidance = 3.5 + 2.0 * torch.sin(2.0 * x + phase[2]) * torch.cos(3.0 * y + phase[3])
    guidance = guidance + 0.3 * torch.randn(guidance.shape, generator=gen, device=DEVICE)
    return costs.reshape(-1).contiguous(), guidance.clamp(0.0, 7.0).reshape(-1).contiguous()


def _mosaics(case, seed):
    """Two modules' raw Q6 mosaics (the second shifted and noisy), and their calibrated cameras."""
    scene_case = _stage(None, case["width"], case["height"], 1, 64)
    rng = np.random.default_rng(seed)
    tiles = [scenes._noise_tile(np.random.default_rng(seed * 7919 + i)) for i in range(4)]
    w, h = case["width"], case["height"]
    k = scenes._intrinsics(w, h)
    ref = scenes._camera(w, h, k, np.eye(3), np.zeros(3))
    tgt = scenes._camera(w, h, k, scenes._random_rotation(rng, 0.3), np.array([25.0, 0.0, 0.0]))
    surfaces = [scenes._background(rng, ref, 20000.0, 3.0, 0)]
    for i in range(5):
        surfaces.append(scenes._random_plane(rng, ref, 1.0 / rng.uniform(1 / 20000.0, 1 / 3000.0), (0.2, 0.6), 30.0,
                                             3.0, (i + 1) % 4))
    on_device = [torch.as_tensor(t, device=DEVICE) for t in tiles]
    mesh = None
    if case["mesh"]:
        gy, gx = np.meshgrid(np.linspace(-1, 1, 13), np.linspace(-1, 1, 17), indexing="ij")
        mesh = VignettingMesh(17, 13, (1.0 + 0.5 * (gx * gx + gy * gy)).astype(np.float32))
    mosaics = []
    for i, cam in enumerate((ref, tgt)):
        raw = scenes.render_module_gpu(cam, surfaces, on_device, seed * 104729 + i, DEVICE)
        mosaics.append(Mosaic(w, h, ((raw >> 2) << 6).cpu().numpy().astype(np.uint16), float(16 << 6),
                              float(1023 << 6), mesh))
    return mosaics, (ref, tgt), _options(scene_case)


def _train_batch(case, seed):
    gen = _generator(seed)
    c, r, d = case["columns"], case["rows"], case["labels"]
    bins = torch.tensor([0] + sample_labels(d), device=DEVICE)
    samples = []
    for _ in range(case["images"]):
        costs, guidance = _volume(gen, c, r, d)
        costs = costs.reshape(r * c, d)
        winners = 1 + costs[:, 1:].argmin(1)
        mask = (torch.rand(r * c, generator=gen, device=DEVICE) < 0.95).to(torch.uint8)
        samples.append(Sample(costs[:, bins].contiguous().reshape(-1), guidance, winners.to(torch.int32), mask, c, r, d,
                              len(bins)))
    return samples


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("stage", "call", "coarse"):
        scene = _scene(case, seed)
        if kind == "call":
            return dict(kind=kind, scene=scene, inputs=scene.inputs())
        # a graph belongs to one stage's buffers, so its program keeps a context for it
        ctx = DepthContext(0) if case.get("graph") else default_context()
        stage = DeviceStage(scene.inputs(), 0, scene.alignments(), scene.options, context=ctx,
                            graph=case.get("graph", False))
        band = None
        if case.get("band"):
            net = BandNet(ctx)
            net.load(WEIGHTS)
            band = BandOptions(params=net.params)
        return dict(kind=kind, stage=stage, band=band)
    if kind == "sgm":
        gen = _generator(seed)
        shapes = _sgm_shapes(case)
        volumes = [_volume(gen, *s) for s in shapes]
        outs = [torch.empty_like(costs) for costs, _ in volumes]
        batch = (abi.SgmInstanceC * len(shapes))()
        for i, ((costs, guidance), out, (c, r, d)) in enumerate(zip(volumes, outs, shapes)):
            batch[i] = abi.SgmInstanceC(costs.data_ptr(), guidance.data_ptr(), out.data_ptr(), c, r, d)
        return dict(kind=kind, ctx=default_context(), volumes=volumes, outs=outs, batch=batch)
    if kind == "module":
        mosaics, cameras, _ = _mosaics(case, seed)
        return dict(kind=kind, mosaics=mosaics, cameras=cameras, size=(case["width"], case["height"]))
    net = BandNet(default_context())
    net.load(WEIGHTS)
    return dict(kind=kind, net=net, samples=_train_batch(case, seed))


# ---- one pass -------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "stage":
        stage = state["stage"]
        if not stage():
            raise RuntimeError("the stage refused its inputs")
        reports = [stage.report(t) for t in stage.targets]
        return dict(depth=stage.depth, confidence=stage.confidence, provenance=stage.provenance,
                    points=[stage.points[t] for t in stage.targets],
                    weights=[stage.point_confidence[t] for t in stage.targets],
                    refined=[r.refined_nodes for r in reports], improvement=[r.median_score_improvement for r in reports])
    if kind == "call":
        alignments = state["scene"].alignments()
        depth = refine_multiview_depth(state["inputs"], 0, alignments, state["scene"].options)
        return dict(depth=depth.depth, confidence=depth.confidence, provenance=depth.provenance,
                    points=[a.warp.points for a in alignments[1:]], weights=[a.warp.confidence for a in alignments[1:]],
                    refined=[a.report.depth.refined_nodes for a in alignments[1:]])
    if kind == "coarse":
        result = coarse_depth(state["stage"], state["band"])
        return dict(winner=result.winner, tested=result.tested,
                    bands=result.offsets if result.offsets is not None else [],
                    fallback=result.fallback if result.fallback is not None else [])
    if kind == "sgm":
        ctx, batch = state["ctx"], state["batch"]
        ctx.check(ctx.lib.chiaro_sgm_aggregate_batch_device(ctx.handle, batch, len(batch), 0, 0))
        return state["outs"]
    if kind == "module":
        (ref_mosaic, tgt_mosaic), (ref_cam, tgt_cam) = state["mosaics"], state["cameras"]
        w, h = state["size"]
        planes = [ref_mosaic.luminance_half(), tgt_mosaic.luminance_half()]
        inputs = [AlignInput(name=n, luminance=p, width=w, height=h, camera=c, nominal_focal_px=c.focal_px)
                  for n, p, c in zip(("A1", "A2"), planes, (ref_cam, tgt_cam))]
        aligned = align_module(inputs[0], inputs[1], AlignOptions())
        refined = refine_resolution_warp(planes[0], planes[1], aligned.warp, w, h)
        return dict(luminance=[p.data for p in planes], warp=aligned.warp.points, weights=aligned.warp.confidence,
                    gain=aligned.gain, refined=refined.warp.points, refined_weights=refined.warp.confidence)
    gradient, loss = state["net"].gradient(state["samples"])
    return dict(gradient=gradient, loss=loss)


# ---- what a pass cannot do without -------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("stage", "call", "coarse"):
        (cols, rows, _), (cc, cr, _) = output_shape(case["width"], case["height"], _options(case))
        v, d = case["sources"], case["planes"] + 1
        m, n = cols * rows, cc * cr
        taps = (2 * case["radius"] + 1) ** 2
        planes = 4 * (1 + v) * (case["width"] // 2) * (case["height"] // 2)
        cost = n * (25 if case.get("band") else d) * v * taps * 16.0
        if kind == "coarse":
            return {"bytes": planes + 5 * n, "flops": cost + n * d * 8 * 6.0}
        # 16 operations a tap: 14 hypotheses a node in the direct pass, 14 in the decisions
        return {"bytes": planes + m * (13 + 12 * v), "flops": cost + n * d * 8 * 6.0 + 28.0 * m * v * taps * 16.0}
    if kind == "sgm":
        cells = sum(c * r * d for c, r, d in _sgm_shapes(case))
        return {"bytes": 8 * cells, "flops": 8 * 6.0 * cells}
    if kind == "module":
        n = (case["width"] // 2) * (case["height"] // 2)
        # mosaics in, planes out and in again; the pyramid's patch searches are most of the operations
        return {"bytes": 2 * n * (8 + 4 + 4 + 4), "flops": 2 * n * 20.0 + n * 120.0}
    pixels = case["columns"] * case["rows"] * case["images"]
    return {"bytes": pixels * (17 * 4 + 4 + 4 + 1), "flops": pixels * 6.0 * LAYERS * TAPS * CH * CH}


# ---- 64-bit results ---------------------------------------------------------------------
def _sgm_exact(costs, guidance, columns, rows, labels):
    """Eight-path aggregation in 64 bits: for each direction, every path advanced together, one
    node of each path at a step."""
    cost = costs.double().reshape(rows, columns, labels)
    guide = guidance.double().reshape(rows, columns)
    total = torch.zeros_like(cost)
    for dr, dc in ((0, 1), (0, -1), (1, 0), (-1, 0), (1, 1), (-1, -1), (1, -1), (-1, 1)):
        steps = columns if dr == 0 else rows
        previous = None
        for s in range(steps):
            if dr == 0:
                i = s if dc > 0 else columns - 1 - s
                current, g = cost[:, i], guide[:, i]
            else:
                i = s if dr > 0 else rows - 1 - s
                current, g = cost[i], guide[i]
            if previous is None:
                value = current.clone()
            else:
                last, g_last = previous
                if dr != 0 and dc != 0:  # the node before sits one column back along the path
                    last, g_last = torch.roll(last, dc, 0), torch.roll(g_last, dc, 0)
                edge = 1.0 / (1.0 + 4.0 * (g - g_last).abs())
                p1, p2 = 0.06 * edge.clamp(min=0.35), 0.45 * edge.clamp(min=0.12)
                low = last.min(1).values
                best = torch.minimum(last, (low + p2)[:, None])
                best[:, 1:] = torch.minimum(best[:, 1:], last[:, :-1] + p1[:, None])
                best[:, :-1] = torch.minimum(best[:, :-1], last[:, 1:] + p1[:, None])
                value = current + best - low[:, None]
                if dr != 0 and dc != 0:  # a path that enters at the side starts there
                    side = 0 if dc > 0 else columns - 1
                    value[side] = current[side]
            if dr == 0:
                total[:, i] += value
            else:
                total[i] += value
            previous = (value, g)
    return total.reshape(-1)


def _gradient_exact(case, seed):
    samples = _train_batch(case, seed)
    net = BandNet(default_context())
    net.load(WEIGHTS)
    params = net.params.double().requires_grad_(True)
    c, r, d = case["columns"], case["rows"], case["labels"]
    labels = torch.tensor(sample_labels(d), device=DEVICE)
    features, targets, masks = [], [], []
    for s in samples:
        bins = s.costs.double().reshape(r * c, -1)[:, 1:]
        low, at = bins.min(1)
        f = torch.zeros(r * c, CH, dtype=torch.float64, device=DEVICE)
        f[:, 0] = s.guidance.double() / 8.0
        f[:, 1:17] = bins - low[:, None]
        f[:, 17] = (labels[at] - 1).double() / (d - 2)
        f[:, 18] = low
        features.append(f.reshape(r, c, CH).permute(2, 0, 1))
        targets.append((s.winners.double() - 1.0) / (d - 2))
        masks.append(s.mask.double())
    x = torch.stack(features)
    layer = TAPS * CH * CH
    for k in range(LAYERS):
        p = params[k * (layer + CH):(k + 1) * (layer + CH)]
        weight = p[:layer].reshape(3, 3, CH, CH).permute(2, 3, 0, 1)
        x = torch.nn.functional.conv2d(x, weight, p[layer:], padding=1)
        if k + 1 < LAYERS:
            x = torch.relu(x)
    mask = torch.cat(masks)
    error = x[:, 0].reshape(-1) - torch.cat(targets)
    loss = (torch.nn.functional.huber_loss(error, torch.zeros_like(error), reduction="none", delta=0.02) * mask).sum()
    loss = loss / mask.sum()
    (gradient,) = torch.autograd.grad(loss, params)
    return dict(gradient=gradient.cpu().numpy(), loss=float(loss))


def _luminance_exact(mosaic):
    h, w = mosaic.height // 2, mosaic.width // 2
    s = torch.from_numpy(mosaic.samples.astype(np.int32)).to(DEVICE).double()[:2 * h, :2 * w]
    mean = (s[0::2, 0::2] + s[0::2, 1::2] + s[1::2, 0::2] + s[1::2, 1::2]) * 0.25
    linear = (mean - mosaic.black_q6) / max(mosaic.white_q6 - mosaic.black_q6, 1.0)
    if mosaic.vignetting is not None:
        return None  # the mesh lookup's own rounding decides its cell
    return torch.log(1.0 + 1000.0 * linear.clamp(min=0.0)).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "sgm":
        gen = _generator(seed)
        return [_sgm_exact(*_volume(gen, *s), *s).cpu().numpy() for s in _sgm_shapes(case)]
    if kind == "train":
        return _gradient_exact(case, seed)
    if kind == "module" and not case["mesh"]:
        mosaics, _, _ = _mosaics(case, seed)
        return dict(luminance=[_luminance_exact(m) for m in mosaics], warp=None, weights=None, gain=None, refined=None,
                    refined_weights=None)
    return None
