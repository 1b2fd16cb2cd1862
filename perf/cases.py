"""The work that a user of this framework has it do, as cases that can be timed.

Every case goes through the public entry points only: ``build_pair_table``,
``run_forward``, ``ConvMainUnitTest.implicit_gemm2``, ``GemmMainUnitTest.matmul2``,
``GatherAll`` / ``ScatterAll`` and ``SparseEncoder.forward``.  Clouds have the
statistics of the benchmark's LiDAR-like clouds (planar patches and Gaussian
clusters in a 41 x 1600 x 1408 grid, ``cumm.voxelgen.lidar_voxels``), made here
with torch on the GPU because the large ones take seconds in numpy.

``exact`` restates each path in float64 with plain torch.
"""
import math
import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "cumm-rocm_b200"))

GRID = (41, 1600, 1408)  # (z, y, x)
PAIRS_PER_VOXEL = 12.7   # submanifold 3x3x3 on these clouds, 5k to 300k voxels
BF16, F16, F32 = torch.bfloat16, torch.float16, torch.float32
DTYPES = {"bf16": BF16, "f16": F16, "f32": F32}

# serving encoder: (kind, C, K) per layer, as cumm.serve.LAYERS
ENCODER = (("subm", 16, 16), ("subm", 16, 16), ("down", 16, 32), ("subm", 32, 32), ("down", 32, 64),
           ("subm", 64, 64), ("subm", 64, 64), ("down", 64, 128), ("subm", 128, 128), ("subm", 128, 128))


def listed():
    return [
        # one small cloud (an indoor scan, a cropped object) through one layer whose
        # pair table is at hand: launches and host time count
        {"name": "fwd_small", "kind": "conv", "n": 4000, "c": 64, "k": 64, "dtype": "bf16", "ops": "f",
         "table": "sorted", "order": "scan"},
        # the benchmark's training step: one 200k-voxel LiDAR cloud, forward, input
        # gradient and weight gradient of one layer over a kept pair table
        {"name": "train_200k_c64", "kind": "conv", "n": 200_000, "c": 64, "k": 64, "dtype": "bf16", "ops": "fdw",
         "table": "sorted", "order": "scan"},
        # a caller of the reference's API: no sorted table, no tile order, voxels in
        # the order a hash voxeliser leaves them, an odd voxel count, fp16
        {"name": "train_ragged_c32", "kind": "conv", "n": 37_421, "c": 32, "k": 32, "dtype": "f16", "ops": "fd",
         "table": "plain", "order": "hash"},
        # the encoder's widest layers in training
        {"name": "train_60k_c128", "kind": "conv", "n": 60_000, "c": 128, "k": 128, "dtype": "bf16", "ops": "fdw",
         "table": "sorted", "order": "scan"},
        # the full-precision path (correctness workload: 20k voxels, C = K = 32)
        {"name": "train_20k_c32_f32", "kind": "conv", "n": 20_000, "c": 32, "k": 32, "dtype": "f32", "ops": "fdw",
         "table": "plain", "order": "scan"},
        # stride-2 downsample 64 -> 128 on the 200k cloud, E4M3 inference
        {"name": "down_200k_fp8", "kind": "down", "n": 200_000, "c": 64, "k": 128, "dtype": "e4m3", "order": "scan"},
        # what every new cloud needs before its first layer
        {"name": "pairs_subm_200k", "kind": "pairs", "n": 200_000, "stride": 1, "order": "scan"},
        {"name": "pairs_down_60k", "kind": "pairs", "n": 60_000, "stride": 2, "order": "scan"},
        # 64 clouds batched: pair build and one layer, the largest pass
        {"name": "batch64_layer", "kind": "batch", "n": 2_600_000, "clouds": 64, "c": 64, "k": 64, "order": "scan"},
        # one served request through the whole encoder (pair builds included)
        {"name": "encoder_60k", "kind": "encoder", "n": 60_000, "order": "scan"},
        # dense matmul2: the benchmark's square GEMM
        {"name": "gemm_8192", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "ta": False, "tb": False,
         "dtype": "bf16", "out": "bf16"},
        # standalone row movement (pooling, scatter to a dense grid): 1M rows of 128 bytes
        {"name": "gather_scatter_1m", "kind": "rows", "n": 1_000_000, "c": 64, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["conv", "conv", "conv", "conv", "down", "pairs", "batch", "encoder", "gemm", "rows"])
    order = rng.choice(["scan", "scan", "hash"])
    if kind == "conv":
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        n = _log(rng, 3000, 40_000 if dtype == "f32" else 300_000)
        c, k = rng.choice([16, 32, 64, 128]), rng.choice([16, 32, 64, 128])
        if dtype == "f32":
            c, k = min(c, 64), min(k, 64)
        # the desps serve weight gradients of bf16 and f32
        ops = rng.choice(["f", "fd"]) if dtype == "f16" else rng.choice(["f", "fd", "fdw", "fdw"])
        return {"kind": kind, "n": n, "c": c, "k": k, "dtype": dtype, "ops": ops,
                "table": rng.choice(["sorted", "plain"]), "order": order}
    if kind == "down":
        c, k = rng.choice([(16, 32), (32, 64), (64, 128), (64, 64), (128, 128)])
        return {"kind": kind, "n": _log(rng, 5000, 300_000), "c": c, "k": k,
                "dtype": rng.choice(["bf16", "f16", "e4m3"]), "order": order}
    if kind == "pairs":
        return {"kind": kind, "n": _log(rng, 2000, 400_000), "stride": rng.choice([1, 1, 2]), "order": order}
    if kind == "batch":
        clouds = rng.choice([2, 5, 16, 33])
        return {"kind": kind, "n": clouds * _log(rng, 5000, 60_000), "clouds": clouds,
                "c": rng.choice([16, 32, 64]), "k": rng.choice([16, 32, 64]), "order": order}
    if kind == "encoder":
        return {"kind": kind, "n": _log(rng, 10_000, 200_000), "order": order}
    if kind == "gemm":
        # square-ish GEMMs and the tall ones of 1x1x1 convolutions over voxels
        if rng.random() < 0.5:
            m, n, k = (8 * _log(rng, 32, 768) for _ in range(3))
        else:
            m, n, k = _log(rng, 4000, 400_000), rng.choice([32, 64, 96, 128, 256]), rng.choice([32, 64, 128, 256])
        dtype = rng.choice(["bf16", "f16"])
        # a transposed A has m as its contiguous dimension, which 16-byte rows need a multiple of 8
        return {"kind": kind, "m": m, "n": n, "k": k, "ta": m % 8 == 0 and rng.random() < 0.3,
                "tb": rng.random() < 0.5, "dtype": dtype, "out": rng.choice([dtype, "f32"])}
    return {"kind": "rows", "n": _log(rng, 5000, 2_000_000), "c": rng.choice([16, 24, 32, 64, 100, 128]),
            "dtype": rng.choice(["bf16", "f16", "f32"])}


# ------------------------------------------------------------------ inputs
def _planes(n, gen, dev):
    """Points on `n`-voxel clouds' planar patches and clusters, [m, 3] (z, y, x)
    in the order they are sampled."""
    dims = torch.tensor(GRID, dtype=F32, device=dev)
    per = max(1, min(4000, (2 * n) // 400 * 20))
    centers = torch.rand(20, 1, 3, generator=gen, device=dev) * dims
    yield (centers + 2.0 * torch.randn(20, per, 3, generator=gen, device=dev)).reshape(-1, 3)
    side = max(8.0, math.sqrt(n / 8) * 0.75)
    m = int(4 * side * side)
    while True:
        center = torch.rand(3, generator=gen, device=dev) * dims
        nrm = torch.randn(3, generator=gen, device=dev)
        nrm[0] *= 3.0  # mostly ground-like
        nrm = nrm / nrm.norm()
        u = torch.linalg.cross(nrm, torch.tensor([0.0, 0.0, 1.0], device=dev))
        u = u / u.norm().clamp_min(1e-3)
        v = torch.linalg.cross(nrm, u)
        ab = (torch.rand(m, 2, generator=gen, device=dev) - 0.5) * side
        yield center + ab[:, :1] * u + ab[:, 1:] * v


def _keys(n, gen, dev, margin=0):
    """n distinct linearised voxels, ascending, `margin` voxels inside the grid
    in y and x."""
    keys = torch.empty(0, dtype=torch.int64, device=dev)
    low = torch.tensor((0, margin, margin), device=dev)
    lim = torch.tensor(GRID, device=dev) - low
    for i, p in enumerate(_planes(n, gen, dev)):
        v = torch.floor(p).long()
        v = v[((v >= low) & (v < lim)).all(1)]
        keys = torch.cat([keys, (v[:, 0] * GRID[1] + v[:, 1]) * GRID[2] + v[:, 2]])
        if i and keys.numel() >= n:
            keys = torch.unique(keys)
            if keys.numel() >= n:
                return keys[:n]


def _coords(n, gen, dev, order, clouds=1, strided=False):
    """int32 [n, 4] (batch, z, y, x).  "scan": ascending, as the repository's
    generator and a sorted voxeliser leave them; "hash": in no order.

    Where strided layers follow, the number of their outputs depends on the
    cloud's shape: there the scene goes with n alone and the seed moves it
    through the grid by multiples of 8 voxels (the encoder's total stride), so
    that every seed's outputs have the same sizes."""
    shape_gen, shift = gen, 0
    if strided:
        shape_gen = torch.Generator(device=dev)
        shape_gen.manual_seed(n)
        dy, dx = (8 * torch.randint(-8, 9, (2,), generator=gen, device=dev)).tolist()
        shift = dy * GRID[2] + dx
    # cloud sizes differ by up to a factor of ten, as a batch of real scans'
    w = torch.exp(0.8 * torch.randn(clouds, generator=gen, device=dev)).clamp(0.3, 4.0)
    sizes = (w / w.sum() * n).long().tolist()
    sizes[0] += n - sum(sizes)
    parts = []
    for b, s in enumerate(sizes):
        lin = _keys(s, shape_gen, dev, 64 if strided else 0) + shift
        parts.append(torch.stack([torch.full_like(lin, b), lin // (GRID[1] * GRID[2]),
                                  lin // GRID[2] % GRID[1], lin % GRID[2]], 1).int())
        if order == "hash":
            parts[-1] = parts[-1][torch.randperm(s, generator=gen, device=dev)]
    return torch.cat(parts).contiguous()


def _weight(k, c, gen, dev):
    b = math.sqrt(6.0 / (27 * c))
    return (torch.rand(k, 27, c, generator=gen, device=dev) * 2 - 1) * b


def _inputs(case, seed):
    """The tensors of a case, made from the seed alone."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "gemm":
        dt = DTYPES[case["dtype"]]
        a = torch.randn((case["k"], case["m"]) if case["ta"] else (case["m"], case["k"]), generator=gen, device=dev)
        b = torch.randn((case["n"], case["k"]) if case["tb"] else (case["k"], case["n"]), generator=gen, device=dev)
        return {"a": a.to(dt), "b": b.to(dt)}
    if kind == "rows":
        dt = DTYPES[case["dtype"]]
        src = torch.randn(case["n"], case["c"], generator=gen, device=dev).to(dt)
        return {"src": src, "idx": torch.randperm(case["n"], generator=gen, device=dev).int()}
    strided = kind in ("down", "encoder") or case.get("stride", 1) != 1
    d = {"coords": _coords(case["n"], gen, dev, case["order"], case.get("clouds", 1), strided)}
    if kind == "pairs":
        return d
    if kind == "encoder":
        d["x"] = torch.randn(case["n"], 16, generator=gen, device=dev).to(BF16)
        d["w"] = [_weight(k, c, gen, dev) for _, c, k in ENCODER]
        return d
    c, k, dt = case["c"], case["k"], case.get("dtype", "bf16")
    x, w = torch.randn(case["n"], c, generator=gen, device=dev), _weight(k, c, gen, dev)
    if dt == "e4m3":
        # activations over one scale, weights over one per output channel, folded together
        sx, sw = x.abs().amax() / 448.0, w.abs().amax((1, 2)) / 448.0
        d["x"], d["w"] = (x / sx).to(torch.float8_e4m3fn), (w / sw[:, None, None]).to(torch.float8_e4m3fn)
        d["scale"] = (sx * sw).float().contiguous()
    else:
        d["x"], d["w"] = x.to(DTYPES[dt]), w.to(DTYPES[dt])
    if "d" in case.get("ops", "") or "w" in case.get("ops", ""):
        d["dy"] = torch.randn(case["n"], k, generator=gen, device=dev).to(DTYPES[dt])
    return d


# ------------------------------------------------------------------ the framework's calls
def _table(coords, stride, clouds=1):
    from cumm.spconv_ops import build_pair_table
    if stride == 1:
        return build_pair_table(coords, GRID)
    return build_pair_table(coords, GRID, stride=(2, 2, 2), padding=(1, 1, 1), subm=False, batch_size=clouds)


def _desp(op, x, w, y):
    from cumm.conv.main import get_all_conv_algo_desp
    for d in get_all_conv_algo_desp():
        if (d.op_type == op and d.dtype_input == x and d.dtype_weight == w and d.dtype_output == y):
            return d
    raise KeyError((op, x, w, y))


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind in ("conv", "down"):
        from cumm.conv.main import ConvMainUnitTest
        s["op"] = ConvMainUnitTest()
        pt = s["pt"] = _table(s["coords"], 2 if kind == "down" else 1)
        if kind == "down" or case["table"] == "sorted":
            pt.sorted_indices("fwd")
            pt.tile_order("fwd")
            if "d" in case.get("ops", ""):
                pt.sorted_indices("bwd")
    elif kind == "encoder":
        from cumm.serve import SparseEncoder
        enc = s["enc"] = SparseEncoder(GRID)
        enc.w = s["w"]
        enc.wb = [w.bfloat16() for w in s["w"]]
    elif kind == "gemm":
        from cumm import tensorview as tv
        from cumm.gemm.main import GemmMainUnitTest, get_all_algo_desp
        from cumm.tensorview.gemm import ShuffleStrideType
        code = {"bf16": tv.bfloat16, "f16": tv.float16, "f32": tv.float32}
        s["op"] = GemmMainUnitTest()
        s["desp"] = next(d for d in get_all_algo_desp()
                         if d.dtype_a == code[case["dtype"]] and d.dtype_c == code[case["out"]]
                         and d.trans_a == case["ta"] and d.trans_b == case["tb"]
                         and d.shuffle_type == ShuffleStrideType.kNoShuffle)
    torch.cuda.synchronize()
    return s


def _conv_step(s):
    """Forward, and the gradients the case asks for, of one submanifold layer."""
    from cumm import tensorview as tv
    from cumm.tensorview.gemm import ConvOpType, ConvParams
    case, pt, x, w = s["case"], s["pt"], s["x"], s["w"]
    n, c, k = case["n"], case["c"], case["k"]
    dt = {"bf16": tv.bfloat16, "f16": tv.float16, "f32": tv.float32}[case["dtype"]]
    sort = case["table"] == "sorted"
    stream = torch.cuda.current_stream().cuda_stream
    res = {}

    def params(op, dt_w, inp, weight, out, indices, which):
        p = ConvParams(3, op)
        p.conv_algo_desp = _desp(op, dt, dt_w, dt)
        p.input, p.weight, p.output = tv.Tensor(inp), tv.Tensor(weight), tv.Tensor(out)
        p.indices = tv.Tensor(indices)
        p.mask = tv.Tensor(pt.masks_fwd[0], tv.uint32)
        p.mask_argsort = tv.Tensor(pt.argsorts_fwd[0])
        if sort:
            p.indices_sorted = tv.Tensor(pt.sorted_indices(which))
            if op != ConvOpType.kBackwardWeight:
                p.tile_order = tv.Tensor(pt.tile_order(which))
        p.stream = stream
        return p

    out = res["out"] = torch.empty((n, k), dtype=x.dtype, device=x.device)
    p = params(ConvOpType.kForward, dt, x, w, out, pt.pairs_fwd, "fwd")
    tile = p.conv_algo_desp.tile_shape[0]
    mask_out = torch.empty(((n + tile - 1) // tile,), dtype=torch.int32, device=x.device)
    p.mask_output = tv.Tensor(mask_out, tv.uint32)
    s["op"].implicit_gemm2(p)
    if "d" in case["ops"]:
        din = res["din"] = torch.empty((n, c), dtype=x.dtype, device=x.device)
        p = params(ConvOpType.kBackwardInput, dt, din, w, s["dy"], pt.pairs_bwd, "bwd")
        p.reverse_mask = True
        s["op"].implicit_gemm2(p)
    if "w" in case["ops"]:
        dw = res["dw"] = torch.empty((k, 27, c), dtype=F32, device=x.device)
        p = params(ConvOpType.kBackwardWeight, tv.float32, x, dw, s["dy"], pt.pairs_fwd, "fwd")
        p.mask = tv.Tensor(mask_out, tv.uint32)
        p.mask_width = tile
        s["op"].implicit_gemm2(p)
    return res


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "conv":
        return _conv_step(s)
    if kind == "pairs":
        pt = _table(s["coords"], case["stride"])
        res = {"fwd": pt.pairs_fwd, "bwd": pt.pairs_bwd, "mask": pt.masks_fwd[0], "argsort": pt.argsorts_fwd[0],
               "sorted": pt.sorted_indices("fwd"), "coords": pt.out_inds}
        if case["stride"] != 1:
            res["mask_bwd"], res["argsort_bwd"] = pt.masks_bwd[0], pt.argsorts_bwd[0]
        return res
    if kind == "encoder":
        return s["enc"].forward(s["coords"], s["x"])
    from cumm import tensorview as tv
    if kind in ("batch", "down"):
        from cumm.autotune import FwdConfig, run_forward
        dt = {"bf16": tv.bfloat16, "f16": tv.float16, "e4m3": tv.float_e4m3}[case.get("dtype", "bf16")]
        dt_out = tv.bfloat16 if dt == tv.float_e4m3 else dt
        pt = _table(s["coords"], 1) if kind == "batch" else s["pt"]
        out = torch.empty((pt.n_out, case["k"]), dtype=F16 if dt_out == tv.float16 else BF16, device=s["x"].device)
        run_forward(FwdConfig(1, 0), s["x"], s["w"], out, {1: pt}, dt, dt_out, scale=s.get("scale"))
        return out
    if kind == "gemm":
        from cumm.tensorview.gemm import GemmParams
        c = torch.empty((case["m"], case["n"]), dtype=DTYPES[case["out"]], device=s["a"].device)
        p = GemmParams()
        p.algo_desp = s["desp"]
        p.a, p.b, p.c = tv.Tensor(s["a"]), tv.Tensor(s["b"]), tv.Tensor(c)
        p.stream = torch.cuda.current_stream().cuda_stream
        s["op"].matmul2(p)
        return c
    # rows: the gathered rows, and their sum with the source scattered by the same indices
    from cumm.gemm.gather import GatherAll, ScatterAll
    stream = torch.cuda.current_stream().cuda_stream
    got = torch.empty_like(s["src"])
    GatherAll().gather(tv.Tensor(got), tv.Tensor(s["src"]), tv.Tensor(s["idx"]), stream=stream)
    acc = torch.zeros_like(s["src"])
    ScatterAll().scatter(tv.Tensor(acc), tv.Tensor(s["src"]), tv.Tensor(s["idx"]), stream=stream)
    return {"gathered": got, "scattered": acc}


# ------------------------------------------------------------------ work
def work(case):
    """Inputs read once, outputs written once; 2 * pairs * C * K per convolution."""
    kind, n = case["kind"], case.get("n", 0)
    if kind == "gemm":
        m, nn, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + k * nn) + m * nn * (4 if case["out"] == "f32" else 2), "flops": 2.0 * m * nn * k}
    if kind == "rows":
        row = n * case["c"] * (4 if case["dtype"] == "f32" else 2)
        return {"bytes": 4 * row + 4 * n, "flops": 0.0}
    # what a pair build reads and writes: coordinates; both tables, masks, argsort, sorted table
    build = n * 16 + n * (2 * 27 * 4 + 8 + 27 * 4)
    if kind == "pairs":
        return {"bytes": build if case["stride"] == 1 else n * 16 + n * (27 * 4 + 8) + n // 2 * (2 * 27 * 4 + 8 + 16),
                "flops": 0.0}
    if kind == "encoder":
        # 60k voxels: 1, 0.5, 0.25, 0.12 of them at the four resolutions
        flops = bytes_ = 0.0
        for (kd, c, k), (fi, fo, pv) in zip(ENCODER, ((1, 1, 12.7), (1, 1, 12.7), (1, .46, 3.4), (.46, .46, 14), (.46, .2, 3.4),
                                                     (.2, .2, 15), (.2, .2, 15), (.2, .08, 3.4), (.08, .08, 16), (.08, .08, 16))):
            flops += 2.0 * pv * fi * n * c * k
            bytes_ += 2 * n * (fi * c + fo * k) + 2 * 27 * c * k + fo * n * 27 * 4
        return {"bytes": bytes_, "flops": flops}
    c, k = case["c"], case["k"]
    e = {"f32": 4, "e4m3": 1}.get(case.get("dtype", "bf16"), 2)
    if kind == "down":
        no = int(0.46 * n)
        return {"bytes": n * c * e + 27 * c * k * e + no * k * 2 + no * (27 * 4 + 8), "flops": 2.0 * 3.4 * n * c * k}
    one = 2.0 * PAIRS_PER_VOXEL * n * c * k
    fwd = n * (c + k) * e + 27 * c * k * e + n * (27 * 4 + 8)
    if kind == "batch":
        return {"bytes": build + fwd, "flops": one}
    ops = case["ops"]
    return {"bytes": fwd * len(ops), "flops": one * len(ops)}


# ------------------------------------------------------------------ float64 restatement
def _lin(c, shape):
    return ((c[:, 0].long() * shape[0] + c[:, 1]) * shape[1] + c[:, 2]) * shape[2] + c[:, 3]


def _offsets(dev):
    r = torch.arange(3, device=dev)
    return torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).reshape(27, 3)


def _find(table_keys, perm, keys, ok):
    pos = torch.searchsorted(table_keys, keys).clamp_max(table_keys.numel() - 1)
    hit = ok & (table_keys[pos] == keys)
    return torch.where(hit, perm[pos], torch.full_like(pos, -1)).int()


def _exact_subm(coords, shape):
    """[27, n] input index of every output through every offset, -1 for none."""
    keys, perm = torch.sort(_lin(coords, shape))
    lim = torch.tensor(shape, device=coords.device)
    res = []
    for off in _offsets(coords.device) - 1:
        c = coords.clone()
        c[:, 1:] += off.int()
        ok = ((c[:, 1:] >= 0) & (c[:, 1:] < lim)).all(1)
        res.append(_find(keys, perm, _lin(c, shape), ok))
    return torch.stack(res)


def _exact_down(coords, shape):
    """(pairs [27, n_out], pairs_bwd [27, n], output coordinates, output shape) of
    a 3x3x3, stride-2, pad-1 convolution, outputs in ascending order."""
    oshape = [(d - 1) // 2 + 1 for d in shape]
    lim = torch.tensor(oshape, device=coords.device)
    outs = []
    for off in _offsets(coords.device):
        t = coords[:, 1:] + 1 - off.int()
        ok = ((t >= 0) & (t % 2 == 0) & (t // 2 < lim)).all(1)
        outs.append((torch.cat([coords[:, :1], t // 2], 1), ok))
    keys = torch.unique(torch.cat([_lin(c, oshape)[ok] for c, ok in outs]))
    ident = torch.arange(keys.numel(), device=keys.device)
    pb = torch.stack([_find(keys, ident, _lin(c, oshape), ok) for c, ok in outs])
    pf = torch.full((27, keys.numel()), -1, dtype=torch.int32, device=keys.device)
    for k in range(27):
        i = torch.nonzero(pb[k] >= 0).squeeze(1)
        pf[k, pb[k, i].long()] = i.int()
    z, r = keys // (oshape[1] * oshape[2]), keys % (oshape[1] * oshape[2])
    out = torch.stack([z // oshape[0], z % oshape[0], r // oshape[2], r % oshape[2]], 1).int()
    return pf, pb, out, oshape


def _exact_fwd(x, w, pf):
    y = torch.zeros(pf.shape[1], w.shape[0], dtype=torch.float64, device=x.device)
    xd, wd = x.double(), w.double()
    for k in range(27):
        o = torch.nonzero(pf[k] >= 0).squeeze(1)
        y[o] += xd[pf[k, o].long()] @ wd[:, k].t()
    return y


def _masks(pf):
    bits = (1 << torch.arange(27, device=pf.device))[:, None]
    return ((pf >= 0).long() * bits).sum(0)


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    if kind == "gemm":
        a, b = s["a"].double(), s["b"].double()
        return (a.t() if case["ta"] else a) @ (b.t() if case["tb"] else b)
    if kind == "rows":
        i = s["idx"].long()
        return {"gathered": s["src"].double()[i], "scattered": torch.zeros_like(s["src"]).double().index_copy_(0, i, s["src"].double())}
    if kind == "encoder":
        x, cur, shape, pf = s["x"], s["coords"], list(GRID), None
        for (kd, _, _), w in zip(ENCODER, s["w"]):
            w = w.to(BF16)  # the weights the layers are given
            if kd == "subm":
                pf = _exact_subm(cur, shape) if pf is None else pf
                x = _exact_fwd(x, w, pf).clamp_min(0.0)
            else:
                pd, _, cur, shape = _exact_down(cur, shape)
                x, pf = _exact_fwd(x, w, pd).clamp_min(0.0), None
        return x, cur
    if kind == "pairs" and case["stride"] == 1:
        pf = _exact_subm(s["coords"], GRID)
        m, order = torch.sort(_masks(pf), stable=True)
        return {"fwd": pf, "bwd": pf.flip(0), "mask": m.int(), "argsort": order.int(), "sorted": pf[:, order], "coords": s["coords"]}
    if kind == "pairs":
        pf, pb, out, _ = _exact_down(s["coords"], GRID)
        m, order = torch.sort(_masks(pf), stable=True)
        mb, order_b = torch.sort(_masks(pb), stable=True)
        return {"fwd": pf, "bwd": pb, "mask": m.int(), "argsort": order.int(), "sorted": pf[:, order], "coords": out,
                "mask_bwd": mb.int(), "argsort_bwd": order_b.int()}
    if kind == "down":
        pf = _exact_down(s["coords"], GRID)[0]
        y = _exact_fwd(s["x"].float(), s["w"].float(), pf)
        return y * s["scale"].double() if "scale" in s else y
    pf = _exact_subm(s["coords"], GRID)
    out = _exact_fwd(s["x"], s["w"], pf)
    if kind == "batch":
        return out
    res = {"out": out}
    dy = s["dy"].double() if "dy" in s else None
    if "d" in case["ops"]:
        # pairs seen from the inputs: offset k of one side is offset 26 - k of the other
        res["din"] = _exact_fwd(dy, s["w"].permute(2, 1, 0), pf.flip(0))
    if "w" in case["ops"]:
        dw = torch.zeros(case["k"], 27, case["c"], dtype=torch.float64, device=dy.device)
        xd = s["x"].double()
        for k in range(27):
            o = torch.nonzero(pf[k] >= 0).squeeze(1)
            dw[:, k] = dy[o].t() @ xd[pf[k, o].long()]
        res["dw"] = dw
    return res
