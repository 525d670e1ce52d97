"""Performance cases of the lidar backbone library, as plain data and functions.

Each case is one call sequence a program makes through the public Python front-end
(``engine.Engine``, ``ops``, ``centerpoint_post``) on inputs of the sizes such programs meet:

* ``backbone``  one ``Engine.forward`` / ``forward_dds`` on voxel features and coordinates that are
                on the GPU already, and the dense BEV tensor the detection network reads.  int8
                CenterPoint and fp16 BEVFusion; one frame (a vehicle, latency) or a batch of frames
                (offline, throughput).  The reference's log of nuScenes frames runs from 10.8 k to
                135 k voxels (mean 82.5 k), its benchmark configurations from 60 k to 200 k.
* ``sweep``     raw points to BEV: the voxelizer, then the backbone with the row count it left on
                the device.
* ``voxelize``  the voxelizer alone (fp32 drivers, fp16 recordings).
* ``segment``   an encoder-decoder block: SubM, stride 2, SubM, inverse convolution, skip sum; two
                sparse outputs.
* ``layer``     one SubM layer through the kernel-level calls: hash table, neighbour map, conv.
* ``detect``    CenterPoint head decode and rotated NMS of six tasks, up to the list of boxes.

Scenes: ``law`` draws voxels by the spatial law of the benchmark configurations; ``sample`` takes the
voxel coordinates of a real frame (the two sample frames in tests/golden), turned and mirrored by the
seed and cut to a sector when fewer voxels are asked for.
"""
import functools
import math
import os

import numpy as np
import torch

from lidar_ai_solution_b200 import centerpoint_post, engine, models, ops, scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GRID = scenes.CENTERPOINT_GRID_ZYX           # 41 x 1440 x 1440 cells
VOXELIZER_GRID = (1440, 1440, 40)            # x, y, z
MAX_VOXELS = 160000                          # rows the voxelizer's output buffers hold
SAMPLE = {"centerpoint": "centerpoint_zyx", "bevfusion": "bevfusion_zyx"}

# Tensor ranges of the seed-0 CenterPoint backbone: absmax over one 120 k-voxel ``law`` frame run in
# fp16 (engine.calibrate), three digits, for the tensors "0" .. "37" in execution order.
RANGES = dict((str(i), v) for i, v in enumerate((
    54.0, 104.0, 132.0, 115.0, 164.0, 164.0, 221.0, 177.0, 239.0, 239.0, 372.0, 158.0, 159.0, 371.0,
    371.0, 221.0, 160.0, 442.0, 442.0, 234.0, 105.0, 86.6, 248.0, 248.0, 138.0, 122.0, 258.0, 258.0,
    166.0, 74.0, 49.1, 158.0, 158.0, 87.8, 62.5, 149.0, 149.0, 126.0)))


# ------------------------------------------------------------------------------- the cases
def _backbone(kind, precision, scene, voxels, batch, count, **name):
    return dict(name, what="backbone", kind=kind, precision=precision, scene=scene, voxels=voxels,
                batch=batch, count=count)


def listed():
    return [
        # the sparsest frame of the reference's log: launches and latency
        _backbone("centerpoint", "int8", "law", 10800, 1, "host", name="cp_int8_10k8_b1"),
        # one benchmark frame at a time: a vehicle's latency
        _backbone("centerpoint", "int8", "law", 120000, 1, "host", name="cp_int8_120k_b1"),
        # the throughput benchmark: eight frames in one call
        _backbone("centerpoint", "int8", "law", 120000, 8, "host", name="cp_int8_120k_b8"),
        # a real frame, its row count known to the device only (as after the voxelizer)
        _backbone("centerpoint", "int8", "sample", 79745, 1, "device", name="cp_int8_real_79k_b1"),
        # the other backbone in fp16: a small real frame and the largest configured one
        _backbone("bevfusion", "fp16", "sample", 17748, 1, "host", name="bev_fp16_real_17k_b1"),
        _backbone("bevfusion", "fp16", "law", 200000, 1, "host", name="bev_fp16_200k_b1"),
        # a vehicle's whole lidar path up to the detection network
        dict(name="sweep_fp32_140k", what="sweep", points=140000, dtype="fp32"),
        # the size of the reference's recorded ten-sweep cloud
        dict(name="voxelize_fp16_271k", what="voxelize", points=271156, dtype="fp16"),
        # a segmentation-style block on an odd row count
        dict(name="segment_fp16_c32_50k", what="segment", voxels=50001, channels=32),
        # the middle of the layer sweep of the benchmark configurations
        dict(name="layer_int8_c64_120k", what="layer", voxels=120000, channels=64, precision="int8"),
        # a few hundred candidate boxes per task, and a crowded frame that fills the ranking
        dict(name="detect_typical", what="detect", mean_logit=-6.0),
        dict(name="detect_crowded", what="detect", mean_logit=-3.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["backbone"] * 5 + ["sweep", "voxelize", "segment", "layer", "detect"])
    if what == "backbone":
        kind, precision = rng.choice([("centerpoint", "int8"), ("centerpoint", "int8"),
                                      ("bevfusion", "fp16")])
        scene = rng.choice(["law", "law", "sample"])
        most = 200000 if scene == "law" else {"centerpoint": 79745, "bevfusion": 17748}[kind]
        voxels = _log_int(rng, 10800, most)
        # a real frame has a fifth of the work of a drawn one of equal size, fp16 twice int8's
        room = {"int8": 960000, "fp16": 360000}[precision] // voxels
        batch = rng.choice([b for b in (1, 1, 2, 3, 4, 8) if b <= max(1, room)])
        count = "device" if batch == 1 and voxels <= MAX_VOXELS and rng.random() < 0.4 else "host"
        return _backbone(kind, precision, scene, voxels, batch, count)
    if what in ("sweep", "voxelize"):
        return dict(what=what, points=_log_int(rng, 30000, 300000 if what == "voxelize" else 200000),
                    dtype=rng.choice(["fp32", "fp16"]))
    if what == "segment":
        return dict(what=what, voxels=_log_int(rng, 10000, 120000), channels=rng.choice([16, 32, 64]))
    if what == "layer":
        return dict(what=what, voxels=_log_int(rng, 10000, 200000),
                    channels=rng.choice([16, 32, 64, 128]), precision=rng.choice(["int8", "fp16"]))
    return dict(what=what, mean_logit=round(rng.uniform(-8.0, -3.0), 2))


# ----------------------------------------------------------------------------- the inputs
def _coords(scene, kind, n, seed):
    """One frame's coordinates, int32 [n, 4] = (0, z, y, x), in the order a voxelizer gives them."""
    if scene == "law":
        return scenes.make_coords(n, GRID, seed)
    rng = np.random.default_rng(seed)
    zyx = np.load(os.path.join(ROOT, "tests", "golden", "fixture_coords.npz"))[SAMPLE[kind]]
    zyx = zyx.astype(np.int32)
    y, x = zyx[:, 1], zyx[:, 2]
    if rng.random() < 0.5:
        y, x = x, y
    if rng.random() < 0.5:
        y = GRID[1] - 1 - y
    if rng.random() < 0.5:
        x = GRID[2] - 1 - x
    out = np.stack([np.zeros_like(y), zyx[:, 0], y, x], 1)
    if n < len(out):  # a sector of the sweep
        turn = (np.arctan2(y - GRID[1] / 2, x - GRID[2] / 2) + rng.uniform(0, 2 * np.pi)) % (2 * np.pi)
        out = out[np.sort(np.argsort(turn, kind="stable")[:n])]
    return np.ascontiguousarray(out)


def _bound(scene, n):
    """output_bound of the model: the exporters' 200 000 rows where they suffice; a drawn scene
    grows to three times its voxels after the first stride-2 layers."""
    if scene == "sample" or n <= 60000:
        return 200000
    return 300000 if n <= 120000 else 520000


@functools.lru_cache(maxsize=None)
def _model(kind, precision, bound):
    model = models.scn_backbone(kind, seed=0, grid_zyx=GRID, output_bound=bound)
    return models.quantize(model, RANGES) if precision == "int8" else model


@functools.lru_cache(maxsize=None)
def _engine(kind, precision, bound, batch):
    """A program loads its model once and runs every frame on that engine, whose output buffers
    live as long as it does."""
    e = engine.Engine.from_model(_model(kind, precision, bound), engine.PRECISION_INT8
                                 if precision == "int8" else engine.PRECISION_FP16)
    e.prepare(GRID, batch)
    return e


@functools.lru_cache(maxsize=None)
def _segment_engine(channels, bound):
    e = engine.Engine.from_model(models.encoder_decoder(channels, 0, 5, bound),
                                 engine.PRECISION_FP16)
    e.prepare(GRID)
    return e


def _points(case, seed):
    pts = scenes.make_points(case["points"], seed)
    return torch.from_numpy(pts.astype(np.float16) if case["dtype"] == "fp16" else pts).cuda()


def _voxel_params(case):
    return ops.voxel_params(scenes.CENTERPOINT_RANGE, scenes.CENTERPOINT_VOXEL, VOXELIZER_GRID, 5,
                            1 if case["dtype"] == "fp16" else 0, 10, MAX_VOXELS, 0)


def _down_cells(coords, grid, k, s, p):
    """Linear output cells (sorted) and pair count of a strided convolution."""
    og = [(g + 2 * b - a) // c + 1 for g, a, c, b in zip(grid, k, s, p)]
    cells, pairs = [], 0
    for k0 in range(k[0]):
        for k1 in range(k[1]):
            for k2 in range(k[2]):
                o, ok = [], True
                for a, kk in enumerate((k0, k1, k2)):
                    v = coords[:, 1 + a] + p[a] - kk
                    ok = ok & (v >= 0) & (v % s[a] == 0) & (v // s[a] < og[a])
                    o.append(v // s[a])
                cell = (o[0].astype(np.int64) * og[1] + o[1]) * og[2] + o[2]
                cells.append(cell[ok])
                pairs += int(ok.sum())
    return np.unique(np.concatenate(cells)), pairs, og


def _cells_to_coords(cells, grid):
    out = np.zeros((len(cells), 4), np.int32)
    out[:, 3] = cells % grid[2]
    out[:, 2] = cells // grid[2] % grid[1]
    out[:, 1] = cells // (grid[2] * grid[1])
    return out


def prepare(case, seed):
    what = case["what"]
    if what == "backbone":
        feats, coords = [], []
        for b in range(case["batch"]):
            c = _coords(case["scene"], case["kind"], case["voxels"], 64 * seed + b)
            feats.append(scenes.make_point_features(c, 64 * seed + b))
            c[:, 0] = b
            coords.append(c)
        f = torch.from_numpy(np.concatenate(feats)).cuda()
        c = torch.from_numpy(np.concatenate(coords)).cuda()
        state = {"n": None}
        if case["count"] == "device":  # buffers of the voxelizer's size, the count beside them
            state["n"] = ops.device_count(len(f))
            f = torch.cat([f, f.new_zeros((MAX_VOXELS - len(f), 5))])
            c = torch.cat([c, c.new_zeros((MAX_VOXELS - len(c), 4))])
        state.update(run=_run_backbone, features=f, indices=c, batch=case["batch"],
                     engine=_engine(case["kind"], case["precision"],
                                    _bound(case["scene"], case["voxels"]), case["batch"]))
        return state
    if what == "sweep":
        return {"run": _run_sweep, "points": _points(case, seed), "params": _voxel_params(case),
                "engine": _engine("centerpoint", "int8", 520000, 1)}
    if what == "voxelize":
        return {"run": _run_voxelize, "points": _points(case, seed), "params": _voxel_params(case)}
    if what == "segment":
        c = scenes.make_coords(case["voxels"], GRID, seed)
        f = scenes.make_point_features(c, seed)
        e = _segment_engine(case["channels"], _bound("law", case["voxels"]))
        coarse, _, _ = _down_cells(c, GRID, (3, 3, 3), (2, 2, 2), (1, 1, 1))
        keep = torch.zeros((3 * case["voxels"], 2 * case["channels"]), dtype=torch.float16, device="cuda")
        return {"run": _run_segment, "engine": e, "features": torch.from_numpy(f).cuda(),
                "indices": torch.from_numpy(c).cuda(), "coarse_rows": len(coarse), "coarse": keep}
    if what == "layer":
        ch, n = case["channels"], case["voxels"]
        rng = np.random.default_rng(seed)
        w = (rng.standard_normal((ch, 27, ch)) * np.sqrt(2.0 / (27 * ch))).astype(np.float32)
        bias = (rng.standard_normal(ch) * 0.1).astype(np.float32)
        x = np.clip(rng.standard_normal((n, ch), np.float32), -4, 4)
        if case["precision"] == "int8":
            amax = np.abs(w).reshape(ch, -1).max(1)
            wq = np.clip(np.rint(w * (127.0 / amax)[:, None, None]), -127, 127).astype(np.int8)
            x = np.rint(x * (127.0 / 4)).astype(np.int8)
            weights = ops.ConvWeights(wq, ops.I8, amax / 127 * np.float32(4 / 127), bias)
        else:
            x = x.astype(np.float16)
            weights = ops.ConvWeights(w.astype(np.float16), ops.F16, None, bias)
        return {"run": _run_layer, "x": torch.from_numpy(x).cuda(), "weights": weights,
                "indices": torch.from_numpy(scenes.make_coords(n, GRID, seed)).cuda(),
                "n": ops.device_count(n), "kind": ops.I8 if case["precision"] == "int8" else ops.F16}
    heads = scenes.make_centerpoint_heads(seed, mean_logit=case["mean_logit"])
    return {"run": _run_detect, "post": centerpoint_post.PostProcess(),
            "heads": [{k: torch.from_numpy(v).cuda() for k, v in h.items()} for h in heads]}


# ------------------------------------------------------------------------------ the calls
def _run_backbone(s):
    if s["n"] is None:
        s["engine"].forward(s["features"], s["indices"], GRID, batch=s["batch"])
    else:
        s["engine"].forward_dds(s["features"], s["indices"], s["n"], GRID, batch=s["batch"])
    return s["engine"].output(0)


def _run_sweep(s):
    features, indices, n = ops.voxelize(s["points"], s["params"])
    s["engine"].forward_dds(features, indices, n, GRID)
    return s["engine"].output(0)


def _run_voxelize(s):
    return ops.voxelize(s["points"], s["params"])


def _run_segment(s):
    s["engine"].forward(s["features"], s["indices"], GRID)
    # the coarse features move to a buffer of the program's own, one size for all frames
    s["coarse"][:s["coarse_rows"]].copy_(s["engine"].output(1)[:s["coarse_rows"]])
    return s["engine"].output(0)[:len(s["features"])], s["coarse"]


def _run_layer(s):
    table = ops.hash_build(s["indices"], s["n"], GRID)
    neighbours = ops.subm_map(s["indices"], s["n"], GRID, table)
    return neighbours, ops.conv_forward(s["x"], neighbours, s["n"], s["weights"], act=ops.ACT_RELU,
                                        out_kind=s["kind"], inv_out_scale=127.0 / 4)


def _run_detect(s):
    s["post"].run(s["heads"])
    kept = s["post"].result()  # the tracker waits for the number of boxes
    return s["post"].boxes, len(kept)


def run(state):
    return state["run"](state)


# ------------------------------------------------------------------- work and tolerances
def _subm_pairs(coords, grid):
    """(row, tap) pairs of a 3x3x3 SubM map; the 13 taps before the centre mirror those after."""
    key = (coords[:, 1].astype(np.int64) * grid[1] + coords[:, 2]) * grid[2] + coords[:, 3]
    key.sort()
    z, y, x = key // (grid[1] * grid[2]), key // grid[2] % grid[1], key % grid[2]
    pairs = len(key)
    for t in range(13):
        dz, dy, dx = t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1
        ok = (z + dz >= 0) & (y + dy >= 0) & (y + dy < grid[1]) & (x + dx >= 0) & (x + dx < grid[2])
        want = (key + (dz * grid[1] + dy) * grid[2] + dx)[ok]
        at = np.minimum(np.searchsorted(key, want), len(key) - 1)
        pairs += 2 * int((key[at] == want).sum())
    return pairs


@functools.lru_cache(maxsize=None)
def _backbone_ops(scene, kind, n):
    """Multiply-adds x 2 of one frame through the backbone (present neighbours only)."""
    coords, grid, total, cin = _coords(scene, kind, n, 0), GRID, 0, 16
    for stage, (c, pad) in enumerate(((16, None), (32, (1, 1, 1)), (64, (1, 1, 1)), (128, (0, 1, 1)))):
        if pad is not None:
            cells, pairs, grid = _down_cells(coords, grid, (3, 3, 3), (2, 2, 2), pad)
            coords = _cells_to_coords(cells, grid)
            total += 2 * pairs * cin * c
        pairs = _subm_pairs(coords, grid)
        total += 4 * 2 * pairs * c * c + (2 * pairs * 5 * c if stage == 0 else 0)
        cin = c
    _, pairs, _ = _down_cells(coords, grid, (3, 1, 1), (2, 1, 1), (0, 0, 0))
    return total + 2 * pairs * 128 * 128


@functools.lru_cache(maxsize=None)
def _law_pairs(n):
    c = scenes.make_coords(n, GRID, 0)
    cells, down, og = _down_cells(c, GRID, (3, 3, 3), (2, 2, 2), (1, 1, 1))
    return _subm_pairs(c, GRID), down, len(cells), _subm_pairs(_cells_to_coords(cells, og), og)


BEV_BYTES = 256 * 180 * 180 * 2
BACKBONE_WEIGHTS = 27 * (5 * 16 + 4 * (16 * 16 + 32 * 32 + 64 * 64 + 128 * 128)
                         + 16 * 32 + 32 * 64 + 64 * 128) + 3 * 128 * 128


def work(case):
    """Inputs, weights and results once each; the multiply-adds of neighbours that exist."""
    what = case["what"]
    if what == "backbone":
        b = case["batch"]
        return {"bytes": b * (case["voxels"] * (5 * 2 + 16) + BEV_BYTES)
                + BACKBONE_WEIGHTS * (1 if case["precision"] == "int8" else 2),
                "flops": b * _backbone_ops(case["scene"], case["kind"], case["voxels"])}
    if what in ("sweep", "voxelize"):
        size = 4 if case["dtype"] == "fp32" else 2
        points = case["points"] * 5 * size
        if what == "voxelize":
            return {"bytes": points + MAX_VOXELS * (5 * 2 + 16), "flops": case["points"] * 5}
        # about nine voxels for ten points
        return {"bytes": points + BEV_BYTES + BACKBONE_WEIGHTS,
                "flops": _backbone_ops("law", "centerpoint", int(0.89 * min(case["points"], 180000)))}
    if what == "segment":
        c, n = case["channels"], case["voxels"]
        fine, down, rows, coarse = _law_pairs(n)
        return {"bytes": n * (5 * 2 + 16 + 2 * c) + rows * 2 * 2 * c + 27 * 2 * (5 * c + 8 * c * c),
                "flops": 2 * (fine * 5 * c + down * 2 * c * c * 2 + coarse * 4 * c * c)}
    if what == "layer":
        c, n, size = case["channels"], case["voxels"], 1 if case["precision"] == "int8" else 2
        return {"bytes": n * (16 + 2 * c * size + 4 * 27) + 27 * c * c * size,
                "flops": 2 * _law_pairs(n)[0] * c * c}
    channels = sum(centerpoint_post.HEAD_CHANNELS.values()) * 6 + sum(centerpoint_post.TASK_NUM_CLASSES)
    return {"bytes": channels * 180 * 180 * 2 + 500 * 44, "flops": 180 * 180 * 10 * 4}


def tolerance(case):
    what = case["what"]
    if what == "sweep" or (what == "backbone" and case["precision"] == "int8"):
        # int8 rows behind fp16 layers: an fp16 sum formed in another order flips int8 roundings,
        # whose steps are coarse with absmax ranges (1/127 of a range that is many times the rms)
        return {"rel": 0.03, "max": 0.99}
    if what == "backbone":
        # 21 fp16 layers; a flip of the last bit early on shows most in small values
        return {"rel": 3e-3, "max": 0.2}
    if what == "segment":
        return {"rel": 1e-3, "max": 2e-2}
    if what == "voxelize":
        return {"rel": 5e-4, "max": 2e-3, "differ": 0.0}  # means rounded to fp16, whole coordinates
    if what == "layer":
        return {"rel": 1e-3, "max": 2e-2, "differ": 0.0}  # whole maps and int8 rows, fp16 rows
    return {"rel": 1e-5, "max": 1e-4}
