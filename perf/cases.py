"""Workloads whose speed is tracked: what a program that uses this library has it do.

Every case is a call (or the few calls of one layer) through the public entry points on inputs made
from a seed on the GPU.  Three kinds of voxel scenes stand for point clouds:

* ``uniform`` -- voxels drawn uniformly in the grid, as ``cumm_b200.workloads`` and the benchmark
  draw them: about one neighbour per voxel in the big grid, so the calls move rows and do little
  arithmetic;
* ``surface`` -- voxels on a rolling ground sheet and on upright walls, what a scanner sees: four to
  six neighbours per voxel, in many different neighbour patterns;
* ``crop`` -- a small grid, uniformly filled to almost a half: few rows with many neighbours.

``listed`` is the fixed set, ``draw`` gives further cases of the same ranges."""
import functools
import math

import torch

from cumm_b200.conv.main import ConvMainUnitTest
from cumm_b200.gemm.main import GemmMainUnitTest
from cumm_b200.layer import SparseConvLayer, make_desp
from cumm_b200.pairgen import build_tables_gpu
from cumm_b200.sequence import prepare_gemm_sequence
from cumm_b200.tensorview import float16, float32
from cumm_b200.tensorview.gemm import (Activation, ConvOpType, ConvParams, GemmAlgoDesp, GemmParams,
                                       ShuffleStrideType)
from cumm_b200.workloads import GRID

SMALL_GRID = (8, 24, 24)
MARGIN = 64  # cells of the grid's y and x extents that a strided layer's scene leaves free


def _conv(kind, scene, n, C, K, **more):
    case = {"kind": kind, "scene": scene, "n": n, "scenes": 1, "C": C, "K": K, "ksize": 3, "stride": 1,
            "api": "prepared"}
    case.update(more)
    return case


def listed():
    def named(name, case):
        return dict(case, name=name)

    return [
        # The last stage of a network or a cropped object: so few rows that launches and host work are the time.
        # The calls go through the drop-in entry point, an argument record filled for each.
        named("train small", _conv("train", "crop", 2000, 64, 64, api="params")),
        # One training step of a submanifold layer on one scene: the benchmark's single-scene configuration.
        named("train scene", _conv("train", "uniform", 150000, 128, 128)),
        # The same layer on a batch of eight scenes, with fp32 weight gradients for an exchange between GPUs.
        named("train batch", _conv("train", "uniform", 120000, 128, 128, scenes=8, dw="f32")),
        # A layer in the middle of a network on a scanned scene: many neighbours, an odd row count.
        named("train surface", _conv("train", "surface", 100003, 64, 64)),
        # A downsampling layer that widens the channels; output rows differ from input rows.
        named("train down", _conv("train", "surface", 40009, 32, 64, stride=2)),
        # A large receptive field, 125 filter offsets (several mask words per row), narrow channels.
        named("train wide", _conv("train", "surface", 30011, 32, 32, ksize=5, api="params")),
        # Inference with bias and ReLU at large channels: the tensor cores have the work.
        named("infer f16", _conv("infer", "surface", 60000, 256, 256, api="params")),
        # Quantised inference, the benchmark's configuration: stride 2, every output row once.
        named("infer int8", _conv("infer8", "uniform", 150000, 128, 128, stride=2)),
        # The tables that a new scene needs before its first layer, both directions.
        named("tables scene", _conv("tables", "uniform", 150000, 0, 0)),
        # The same for a downsampling layer, which has to find its output voxels first.
        named("tables down", _conv("tables", "uniform", 150000, 0, 0, stride=2)),
        # A layer as one gather-GEMM-scatter call per filter offset, each adding into the output.
        named("gather gemm", _conv("pairs", "uniform", 150000, 64, 64, api="calls")),
        # A 2-D convolution over a bird's-eye grid behind the sparse layers: every row has every neighbour.
        named("dense 2d", {"kind": "dense", "batch": 2, "height": 200, "width": 176, "C": 128, "K": 128, "ksize": 3,
                           "stride": 1}),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: rows over three decades, odd counts among them, channel
    counts in steps of the access width."""
    kind = rng.choice(["train", "train", "train", "infer", "infer8", "tables", "pairs", "dense"])
    if kind == "dense":
        return {"kind": kind, "batch": rng.randint(1, 3), "height": _log_int(rng, 12, 200),
                "width": _log_int(rng, 12, 200), "C": 8 * rng.randint(2, 16), "K": 8 * rng.randint(2, 16),
                "ksize": 3, "stride": rng.choice([1, 1, 2])}
    scene = rng.choice(["uniform", "surface", "surface"])
    n = _log_int(rng, 1500, 150000)
    step = 16 if kind == "infer8" else 8
    if rng.random() < 0.5:
        C, K = rng.choice([32, 64, 128]), rng.choice([32, 64, 128])
    else:
        C, K = step * rng.randint(2, 128 // step), step * rng.randint(2, 128 // step)
    more = {}
    if kind in ("train", "infer", "infer8", "tables"):
        more["stride"] = rng.choice([1, 1, 1, 2])
    if kind == "train":
        more["api"] = rng.choice(["prepared", "prepared", "params"])
        more["dw"] = rng.choice(["f16", "f32"])
        if rng.random() < 0.2:
            more.update(ksize=5, api="params", stride=1)
            n, C, K = min(n, 30000), min(C, 64), min(K, 64)
    elif kind == "infer":
        more["api"] = "params"
        if rng.random() < 0.3:
            n, C, K = min(n, 60000), 8 * rng.randint(17, 32), 8 * rng.randint(17, 32)
    elif kind == "infer8":
        more["add"] = rng.random() < 0.5 and more["stride"] == 1
    elif kind == "tables":
        C = K = 0
        more["scenes"] = rng.choice([1, 1, 4])
        if rng.random() < 0.2:
            more.update(ksize=5, stride=1)
    elif kind == "pairs":
        more["api"] = rng.choice(["calls", "calls", "sequence"])
    return _conv(kind, scene, n, C, K, **more)


# ---------------------------------------------------------------- scenes
def _grid(case):
    return SMALL_GRID if case["scene"] == "crop" else GRID


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _sample(case, gen, scene):
    """``n`` unique voxels of one scene, in random order: int32 [n, 4] (batch, z, y, x)."""
    n, (gz, gy, gx) = case["n"], _grid(case)
    if case["stride"] > 1:
        gy, gx = gy - MARGIN, gx - MARGIN

    def ints(hi, count):
        return torch.randint(0, hi, (count,), generator=gen, device="cuda")

    if case["scene"] == "surface":
        m = 3 * n
        side = min(int(math.sqrt(0.9 * n)) + 8, gx)
        y, x = ints(side, m), ints(side, m)
        ground = 10 + 4 * torch.sin(y * (2 * math.pi / 180)) + 4 * torch.cos(x * (2 * math.pi / 230))
        wall = ints(10, m) < 3
        along_y = ints(2, m) == 0
        y = torch.where(wall & ~along_y, y // 64 * 64, y)
        x = torch.where(wall & along_y, x // 64 * 64, x)
        z = torch.where(wall, ints(gz, m), ground.long())
        lin = (z * gy + y) * gx + x
    elif gz * gy * gx < 16 * n:
        lin = torch.randperm(gz * gy * gx, generator=gen, device="cuda")
    else:
        lin = ints(gz * gy * gx, n + n // 50 + 64)
    lin = torch.unique(lin)
    lin = lin[torch.randperm(lin.numel(), generator=gen, device="cuda")[:n]]
    if lin.numel() != n:
        raise RuntimeError(f"scene of {n} voxels has only {lin.numel()} distinct ones")
    return torch.stack([torch.full_like(lin, scene), lin // (gy * gx), lin // gx % gy, lin % gx], 1).int()


def _coords(case, seed):
    """The rows of all scenes.  A strided layer has as many output rows as its scene makes, so there the
    seed moves one scene by whole strides, mirrors its layers and shuffles its rows: the row counts of
    every seed are the same, the coordinates, their order and their neighbours' row numbers are not."""
    gen = _generator(seed)
    if case["stride"] == 1:
        return torch.cat([_sample(case, gen, s) for s in range(case["scenes"])])
    same = _generator(case["n"])
    coords = torch.cat([_sample(case, same, s) for s in range(case["scenes"])])
    steps = MARGIN // case["stride"]
    move = 1 + torch.randint(0, steps - 1, (2,), generator=gen, device="cuda", dtype=torch.int32)
    coords[:, 2:] += case["stride"] * move
    if seed % 2:
        coords[:, 1] = _grid(case)[0] - 1 - coords[:, 1]
    return coords[torch.randperm(len(coords), generator=gen, device="cuda")].contiguous()


def _table_args(case):
    k, s = case["ksize"], case["stride"]
    return dict(batch_size=case["scenes"], grid=_grid(case), ksize=(k, k, k), stride=(s, s, s), subm=s == 1,
                backward=True)


@functools.lru_cache(maxsize=64)
def _counts(items):
    """(rows in, rows out, pairs) of a case's scene, for ``work``."""
    case = dict(items)
    t = build_tables_gpu(_coords(case, 0), **_table_args(case))
    return t.n_in, t.n_out, int((t.indices >= 0).sum())


# ---------------------------------------------------------------- inputs
def prepare(case, seed):
    if case["kind"] == "dense":
        return _prepare_dense(case, seed)
    coords = _coords(case, seed)
    if case["kind"] == "tables":
        return {"case": case, "coords": coords, "args": _table_args(case)}
    gen = _generator(seed + 1)
    C, K, kv = case["C"], case["K"], case["ksize"] ** 3
    t = build_tables_gpu(coords, **_table_args(case))
    state = {"case": case, "tables": t}

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    if case["kind"] == "infer8":
        def bytes_(*shape):
            return torch.randint(-127, 128, shape, generator=gen, device="cuda").to(torch.int8)

        scale = torch.empty(K, device="cuda").uniform_(1e-3, 1e-2, generator=gen)
        state.update(x=bytes_(t.n_in, C), w=bytes_(K, kv, C), out=torch.zeros((t.n_out, K), dtype=torch.int8, device="cuda"),
                     scale=scale, bias=normal(K))
        layer = SparseConvLayer(t, state["w"], state["x"], state["out"])
        if case.get("add"):  # a residual branch and a ReLU in the same call
            state["residual"] = bytes_(t.n_out, K)
            layer.fwd_params.output_add, layer.fwd_params.beta = state["residual"], 0.5
            layer.fwd_params.act_type = Activation.ReLU
        layer.prepare_int8(scale, state["bias"])
        state["layer"] = layer
        return state
    x, w, extra = _values(case, seed, t.n_in, t.n_out)
    if case["kind"] == "pairs":
        out = torch.zeros((t.n_out, K), dtype=torch.float16, device="cuda")
        state.update(x=x, w=w, out=out, calls=[])
        for f in range(kv):
            rows = torch.nonzero(t.indices[f] >= 0).flatten()
            if rows.numel():
                state["calls"].append((f, t.indices[f, rows].contiguous(), rows.int()))
        if case["api"] == "sequence":
            state["sequence"] = prepare_gemm_sequence([_gemm_params(state, *c) for c in state["calls"]])
        return state
    state.update(x=x, w=w, out=torch.zeros((t.n_out, K), dtype=torch.float16, device="cuda"))
    if case["kind"] == "infer":
        state["bias"] = extra
        return state
    state["dout"] = extra
    state["din"] = torch.zeros((t.n_in, C), dtype=torch.float16, device="cuda")
    state["dw"] = torch.zeros((K, kv, C), dtype=torch.float32 if case.get("dw") == "f32" else torch.float16, device="cuda")
    if case["api"] == "prepared":
        state["layer"] = SparseConvLayer(t, w, x, state["out"], state["dout"], state["din"], state["dw"])
    return state


def _values(case, seed, n_in, n_out):
    """fp16 rows, weights and the third operand (bias, or the output's gradient) of a sparse case."""
    gen = _generator(seed + 1)
    C, K, kv = case["C"], case["K"], case["ksize"] ** 3

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    x = normal(n_in, C).half()
    w = (normal(*((kv, C, K) if case["kind"] == "pairs" else (K, kv, C))) / math.sqrt(kv * C)).half()
    if case["kind"] == "pairs":
        return x, w, None
    return x, w, (normal(K) if case["kind"] == "infer" else normal(n_out, K)).half()


def _dense_values(case, seed):
    gen = _generator(seed)
    B, H, W, C, K, k, s = (case[q] for q in ("batch", "height", "width", "C", "K", "ksize", "stride"))

    def half(*shape, scale=1.0):
        return (torch.randn(shape, generator=gen, device="cuda") * scale).half()

    x, w = half(B, H, W, C), half(K, k, k, C, scale=1 / math.sqrt(k * k * C))
    dout = half(B, (H + 2 * (k // 2) - k) // s + 1, (W + 2 * (k // 2) - k) // s + 1, K)
    return x, w, dout


def _prepare_dense(case, seed):
    x, w, dout = _dense_values(case, seed)
    return {"case": case, "x": x, "w": w, "dout": dout, "out": torch.zeros_like(dout), "din": torch.zeros_like(x),
            "dw": torch.zeros_like(w)}


# ---------------------------------------------------------------- one pass
def _gemm_params(state, f, a_inds, c_inds):
    case = state["case"]
    d = GemmAlgoDesp()
    d.dtype_a = d.dtype_b = d.dtype_c = float16
    d.dacc = d.dcomp = float32
    d.trans_a, d.trans_b, d.trans_c = False, False, False
    d.tile_shape = [128, 64 if case["K"] <= 64 else 128, 64 if case["C"] <= 64 else 128]
    d.warp_tile_shape = list(d.tile_shape)
    d.tensorop = [128, d.tile_shape[1], 16]
    d.num_stage = 3
    d.algo = "Blackwell"
    d.shuffle_type = ShuffleStrideType.ShuffleAC
    d.element_per_access_a = d.element_per_access_b = d.element_per_access_c = 8
    p = GemmParams()
    p.algo_desp = d
    p.a, p.b, p.c = state["x"], state["w"][f], state["out"]
    p.a_inds, p.c_inds = a_inds, c_inds
    p.beta = 1.0
    return p


def _conv_params(op, x, weight, out, ndim=3, dynamic=False):
    p = ConvParams(ndim, op)
    p.conv_algo_desp = make_desp(op, False, int(x.shape[-1]), int(out.shape[-1]))
    p.conv_algo_desp.ndim, p.conv_algo_desp.dynamic_mask = ndim, dynamic
    p.input, p.weight, p.output = x, weight, out
    if op == ConvOpType.BackwardWeight:
        p.mask_width, p.split_k_slices = 128, 32
    return p


def _implicit_gemm(op, t, x, weight, out, bias=None):
    p = _conv_params(op, x, weight, out, dynamic=t.kv > 32)
    if op == ConvOpType.BackwardInput:
        p.indices, p.mask, p.mask_argsort = t.indices_bwd, t.mask_bwd, t.mask_argsort_bwd
    else:
        p.indices, p.mask_argsort = t.indices, t.mask_argsort
        p.mask = t.mask_output if op == ConvOpType.BackwardWeight else t.mask
        if op == ConvOpType.Forward:
            p.mask_output = t.mask_output
    if bias is not None:
        p.bias, p.beta, p.act_type = bias, 1.0, Activation.ReLU
    ConvMainUnitTest.implicit_gemm2(p)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "tables":
        t, coords = build_tables_gpu(state["coords"], return_out_coords=True, **state["args"])
        return {"out_coords": coords, "indices": t.indices, "mask": t.mask, "argsort": t.mask_argsort,
                "indices_bwd": t.indices_bwd, "mask_bwd": t.mask_bwd, "argsort_bwd": t.mask_argsort_bwd,
                "tile_masks": t.mask_output}
    if kind == "infer8":
        state["layer"].fwd.launch()
        return state["out"]
    if kind == "infer":
        _implicit_gemm(ConvOpType.Forward, state["tables"], state["x"], state["w"], state["out"], state["bias"])
        return state["out"]
    if kind == "pairs":
        state["out"].zero_()
        if case["api"] == "sequence":
            state["sequence"].launch()
        else:
            for call in state["calls"]:
                GemmMainUnitTest.matmul2(_gemm_params(state, *call))
        return state["out"]
    if kind == "dense":
        for op, x, w, out in ((ConvOpType.Forward, state["x"], state["w"], state["out"]),
                              (ConvOpType.BackwardInput, state["din"], state["w"], state["dout"]),
                              (ConvOpType.BackwardWeight, state["x"], state["dw"], state["dout"])):
            p = _conv_params(op, x, w, out, ndim=2)
            p.conv_algo_desp.mask_sparse = False
            p.padding, p.stride, p.dilation = [case["ksize"] // 2] * 2, [case["stride"]] * 2, [1, 1]
            ConvMainUnitTest.implicit_gemm2(p)
    elif case["api"] == "prepared":
        state["layer"].fwd.launch()
        state["layer"].dgrad.launch()
        state["layer"].wgrad.launch()
    else:
        t = state["tables"]
        _implicit_gemm(ConvOpType.Forward, t, state["x"], state["w"], state["out"])
        _implicit_gemm(ConvOpType.BackwardInput, t, state["din"], state["w"], state["dout"])
        _implicit_gemm(ConvOpType.BackwardWeight, t, state["x"], state["dw"], state["dout"])
    return {"out": state["out"], "din": state["din"], "dw": state["dw"]}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Rows and weights once in and once out per operator, one 4-byte row number per pair, and the
    rows' masks and sort order."""
    if case["kind"] == "dense":
        rows_in = case["batch"] * case["height"] * case["width"]
        rows_out = case["batch"] * (-(-case["height"] // case["stride"])) * (-(-case["width"] // case["stride"]))
        weight = case["ksize"] ** 2 * case["C"] * case["K"]
        data = rows_in * case["C"] + rows_out * case["K"] + weight
        return {"bytes": 3 * 2 * data, "flops": 3 * 2 * rows_out * weight}
    n_in, n_out, pairs = _counts(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    C, K, kv = case["C"], case["K"], case["ksize"] ** 3
    words = -(-kv // 32)
    if case["kind"] == "tables":
        tables = (n_in + n_out) * (4 * kv + 4 * words + 4)
        return {"bytes": 16 * n_in + 16 * n_out * (case["stride"] != 1) + tables, "flops": 0}
    if case["kind"] == "pairs":
        return {"bytes": 2 * (n_in * C + n_out * K + kv * C * K) + 8 * pairs, "flops": 2 * pairs * C * K}
    size = 1 if case["kind"] == "infer8" else 2
    rows = size * (n_in * C + n_out * K + kv * C * K)
    order = 4 * pairs + n_out * (4 * words + 4)
    if case["kind"] == "train":
        order_bwd = 4 * pairs + n_in * (4 * words + 4)
        return {"bytes": 3 * rows + 2 * order + order_bwd, "flops": 3 * 2 * pairs * C * K}
    if case.get("add"):
        rows += n_out * K
    return {"bytes": rows + order, "flops": 2 * pairs * C * K}


def tolerance(case):
    """int8 rows and tables are whole numbers and have one right value.  fp16 rows are fp32 sums
    rounded once: against sums in 64 bits they measure 2.1e-4 (2-norm) and 4.9e-4 (largest), and
    up to 3.8e-4 and 3.6e-3 where every filter offset's call rounds; four times that."""
    if case["kind"] in ("tables", "infer8"):
        return "exact"
    if case["kind"] == "pairs":
        return {"rel": 1.6e-3, "max": 1.5e-2}
    return {"rel": 8.4e-4, "max": 2e-3}


# ---------------------------------------------------------------- the same in 64 bits
def _keys(c, grid):
    return ((c[:, 0] * grid[0] + c[:, 1]) * grid[1] + c[:, 2]) * grid[2] + c[:, 3]


def _neighbours(case, coords):
    """(number of output rows, [(input rows, output rows) per filter offset])."""
    k, s, grid = case["ksize"], case["stride"], _grid(case)
    offsets = [(z, y, x) for z in range(k) for y in range(k) for x in range(k)]
    coords = coords.long()
    shift = lambda r: torch.tensor((0,) + r, device="cuda") - torch.tensor([0] + 3 * [k // 2], device="cuda")
    out = coords
    if s != 1:  # every position that reads some input row, in row-major order
        ogrid = [(g + 2 * (k // 2) - k) // s + 1 for g in grid]
        limit = torch.tensor(ogrid, device="cuda")
        found = []
        for r in offsets:
            at = (coords - shift(r))[:, 1:]
            ok = ((at >= 0) & (at % s == 0) & (at // s < limit)).all(1)
            found.append(_keys(torch.cat([coords[ok, :1], at[ok] // s], 1), ogrid))
        key = torch.unique(torch.cat(found))
        out = torch.stack([key // (ogrid[0] * ogrid[1] * ogrid[2]), key // (ogrid[1] * ogrid[2]) % ogrid[0],
                           key // ogrid[2] % ogrid[1], key % ogrid[2]], 1)
    keys, order = torch.sort(_keys(coords, grid))
    limit = torch.tensor(grid, device="cuda")
    pairs = []
    for r in offsets:
        at = torch.cat([out[:, :1], out[:, 1:] * s], 1) + shift(r)
        inside = ((at[:, 1:] >= 0) & (at[:, 1:] < limit)).all(1)
        want = _keys(at, grid)
        place = torch.searchsorted(keys, want).clamp(max=len(keys) - 1)
        rows = torch.nonzero(inside & (keys[place] == want)).flatten()
        pairs.append((order[place[rows]], rows))
    return len(out), pairs


def exact(case, seed):
    """Results of floating point in 64 bits; tables and int8 rows are compared bit for bit instead."""
    if case["kind"] in ("tables", "infer8"):
        return None
    if case["kind"] == "dense":
        x, w, dout = (v.double() for v in _dense_values(case, seed))
        k, s, half = case["ksize"], case["stride"], case["ksize"] // 2
        H, W = dout.shape[1:3]
        x = torch.nn.functional.pad(x, (0, 0, half, half, half, half))
        out, din, dw = torch.zeros_like(dout), torch.zeros_like(x), torch.zeros_like(w)
        for y in range(k):
            for z in range(k):
                rows = (slice(None), slice(y, y + s * (H - 1) + 1, s), slice(z, z + s * (W - 1) + 1, s))
                out += x[rows] @ w[:, y, z].T
                din[rows] += dout @ w[:, y, z]
                dw[:, y, z] = dout.flatten(0, 2).T @ x[rows].flatten(0, 2)
        return {"out": out, "din": din[:, half:-half, half:-half], "dw": dw}
    coords = _coords(case, seed)
    n_out, pairs = _neighbours(case, coords)
    x, w, extra = _values(case, seed, len(coords), n_out)
    x, w = x.double(), w.double()
    if case["kind"] == "pairs":
        w = w.permute(2, 0, 1)
    out = torch.zeros((n_out, case["K"]), dtype=torch.float64, device="cuda")
    for f, (i, o) in enumerate(pairs):
        out[o] += x[i] @ w[:, f].T
    if case["kind"] == "pairs":
        return out
    if case["kind"] == "infer":
        return (out + extra.double()).clamp(min=0)
    dout, din, dw = extra.double(), torch.zeros_like(x), torch.zeros_like(w)
    for f, (i, o) in enumerate(pairs):
        din[i] += dout[o] @ w[:, f]
        dw[:, f] = dout[o].T @ x[i]
    return {"out": out, "din": din, "dw": dw}
