"""The workloads by which this library's speed is followed, through its public entry points.

A case is a dict of plain values.  ``kind`` says which entry point it calls:

  step         one ``FourBitAdamW.step()`` over a list of parameters in a warm state (moments of earlier steps, loaded
               through ``load_state_dict``); outputs: every parameter, code buffer and scale
  fused_4bit   the per-tensor call ``fused_4bit`` (both moments with block-128 scales)
  fused_fp32   the per-tensor call ``fused_single_tensor`` (float32 moments)
  codec_block  ``quantize_m``, ``dequantize_m``, ``quantize_v_block``, ``dequantize_v_block`` of one fp32 tensor
  codec_rank1  ``quantize_v``, ``dequantize_v`` of one fp32 matrix

``exact`` gives the same results in 64 bits from plain torch operations.
"""
from __future__ import annotations

import math

import torch

import quantfour_adamw_cuda_b200 as qf
from quantfour_adamw_cuda_b200 import functional as F

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}
BLOCK = 128
LR, B1, B2, EPS, WD = 1e-4, 0.9, 0.999, 1e-8, 0.1
CLIP = 0.999  # a clipping coefficient; g * CLIP rounds back to g in bf16, so a pass can be repeated on the same gradients

QM = [-0.8875, -0.6625, -0.4375, -0.2125, -0.0775, -0.0325, -0.0055, 0.0,
      0.0055, 0.0325, 0.0775, 0.2125, 0.4375, 0.6625, 0.8875, 1.0]
MM = [-0.775, -0.55, -0.325, -0.145, -0.055, -0.019, -0.00275, 0.00275,
      0.019, 0.055, 0.145, 0.325, 0.55, 0.775, 0.94375]
QV = [0.0625 * k for k in range(1, 17)]
MV = [0.09375 + 0.0625 * k for k in range(15)]


def listed():
    layer = "1024,1024,3072x1024,3072,1024x1024,1024,1024,1024,4096x1024,4096,1024x4096,1024"
    return [
        # the smallest step: a small multi-layer network, where launches and host time are all there is
        _step("small_mlp_bf16", "256x64,256,256x256,256,10x256,10", "bfloat16"),
        # one layer of the 355 M-parameter model of shapes.gpt2_medium: matrices, biases and norms in one call, gradients clipped
        _step("transformer_layer_bf16", layer, "bfloat16", clip=True),
        # the same layer trained in half precision
        _step("transformer_layer_fp16", layer, "float16"),
        # one fp32 4096 x 4096 matrix: the first configuration of the benchmark
        _step("matrix_fp32", "4096x4096", "float32"),
        # one decoder layer of the 7B shape of the benchmark
        _step("decoder_layer_bf16", "4096x4096,4096x4096,4096x4096,4096x4096,11008x4096,11008x4096,4096x11008,4096,4096", "bfloat16"),
        # one decoder layer of the 13B shape with its embedding and its head, late in a run: the largest
        _step("decoder_layer_head_bf16", "32000x5120,5120x5120,5120x5120,5120x5120,5120x5120,13824x5120,13824x5120,5120x13824,5120,5120,32000x5120",
              "bfloat16", step=20000),
        # matrices whose rows have no round length: projections, classifier heads, feature tables
        _step("ragged_matrices_bf16", "1000x1500,3000x600,4097x333,50257x300,300x77", "bfloat16"),
        # convolution weights (more than two dimensions: block scales) with their norms and a head
        _step("convolutions_fp32", "64x3x7x7,256x128x3x3,256x256x3x3,512x256x3x3,512x512x3x3,512x512x3x3,2048x512x1x1,512,512,1000x2048", "float32"),
        # an embedding in fine-tuning: many tokens of the vocabulary never occur, their rows have no gradient and no state
        _step("embedding_unseen_rows_bf16", "32000x1024", "bfloat16", unseen=0.4),
        # the per-tensor call of the extension module, odd element count
        {"name": "fused_4bit_bf16", "kind": "fused_4bit", "n": 4096 * 4096 + 77, "dtype": "bfloat16", "step": 100},
        # both moments of a tensor into 4 bits and back (a checkpoint, an optimizer of one's own)
        {"name": "codec_block", "kind": "codec_block", "n": 1 << 26},
        {"name": "codec_rank1", "kind": "codec_rank1", "rows": 4096, "cols": 11008},
    ]


def _step(name, shapes, dtype, step=100, clip=False, unseen=0.0, capturable=False, nd_rank1=False):
    return {"name": name, "kind": "step", "shapes": shapes, "dtype": dtype, "step": step, "clip": clip, "unseen": unseen,
            "capturable": capturable, "nd_rank1": nd_rank1}


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "step", "fused_4bit", "fused_fp32", "codec_block", "codec_rank1"])
    if kind == "codec_block":
        return {"kind": kind, "n": _log(rng, 1000, 1 << 26)}
    if kind == "codec_rank1":
        cols = rng.choice([256 * rng.randint(1, 43), _log(rng, 16, 11008)])
        return {"kind": kind, "rows": _log(rng, 16, min(65536, (1 << 26) // cols)), "cols": cols}
    if kind != "step":
        return {"kind": kind, "n": _log(rng, 1000, 1 << 25), "dtype": rng.choice(sorted(DTYPES)), "step": rng.choice([10, 100, 5000])}
    dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32", "float32", "float16"])
    shapes = []
    budget = _log(rng, 1 << 14, 1 << 28)
    while len(shapes) < 8 and (not shapes or rng.random() < 0.8):
        form = rng.choice(["matrix", "matrix", "ragged", "ragged", "conv", "vector"])
        if form == "vector":
            s = (_log(rng, 16, 20000),)
        elif form == "conv":
            k = rng.choice([1, 3, 3, 5, 7])
            s = (_log(rng, 16, 1024), _log(rng, 3, 1024), k, k)
        elif form == "ragged":
            s = (_log(rng, 8, 60000), _log(rng, 8, 9000))
        else:
            s = (_log(rng, 8, 32000), 256 * rng.choice([1, 2, 3, 4, 5, 8, 10, 16, 20, 32, 43]))
        if math.prod(s) <= budget:
            budget -= math.prod(s)
            shapes.append("x".join(map(str, s)))
        elif budget < 1 << 12:
            break
    option = rng.random()
    c = _step("", ",".join(shapes), dtype, step=rng.choice([3, 100, 5000, 20000]), clip=dtype == "bfloat16" and 0.2 < option < 0.4,
              capturable=option < 0.1, nd_rank1=0.1 <= option < 0.2)
    del c["name"]
    return c


# ---- inputs, with plain torch operations ------------------------------------------------------------------------------


def _shapes(case):
    return [tuple(int(d) for d in s.split("x")) for s in case["shapes"].split(",")]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _codes(x, mid):
    """Number of midpoints below x, packed two to a byte, the even element in the low nibble."""
    c = torch.bucketize(x.reshape(-1), torch.tensor(mid, device=x.device, dtype=x.dtype), out_int32=True).to(torch.uint8)
    if c.numel() % 2:
        c = torch.cat([c, c.new_zeros(1)])
    c = c.view(-1, 2)
    return (c[:, 0] | (c[:, 1] << 4)).contiguous().view(torch.int8)


def _values(codes, n, qmap):
    b = codes.view(torch.uint8)
    q = torch.tensor(qmap, device=codes.device, dtype=torch.float32)
    both = torch.stack([q[(b & 15).int()], q[(b >> 4).int()]], dim=1).reshape(-1)
    return both[:n]


def _blocks(x):
    """Flattened, zero-padded to whole blocks, [-1, 128]."""
    f = x.reshape(-1)
    pad = -f.numel() % BLOCK
    return (torch.cat([f, f.new_zeros(pad)]) if pad else f).view(-1, BLOCK)


def _quantize_block(x, mid):
    b = _blocks(x)
    s = b.abs().amax(dim=1)
    y = torch.where(s[:, None] > 0, b / s[:, None], torch.zeros_like(b)).reshape(-1)[:x.numel()]
    return _codes(y, mid), s


def _maxima(v):
    return [v.amax(dim=[d for d in range(v.dim()) if d != a], keepdim=True) for a in range(v.dim())]


def _smallest(maxima):
    s = maxima[0]
    for m in maxima[1:]:
        s = torch.minimum(s, m)
    return s


def _gradient(shape, gen):
    """About 1e-3, one value in a thousand a hundred times as large."""
    g = torch.randn(shape, device="cuda", generator=gen)
    g.mul_(1e-3)
    return torch.where(torch.rand(shape, device="cuda", generator=gen) < 1e-3, g * 100, g)


def _second_moment(shape, gen):
    """About 1e-6, with rows and columns of different size."""
    v = torch.rand(shape, device="cuda", generator=gen).add_(0.2).mul_(1e-6)
    for a, d in enumerate(shape if len(shape) > 1 else ()):
        v.mul_(torch.rand([d if k == a else 1 for k in range(len(shape))], device="cuda", generator=gen).mul_(2).exp_())
    return v


def _tensor(shape, dtype, gen, unseen=0.0, scheme="auto", nd_rank1=False):
    """Parameter, gradient and state of one tensor in a warm state."""
    n = math.prod(shape)
    p = torch.randn(shape, device="cuda", generator=gen).mul_(0.02).to(dtype)
    g = _gradient(shape, gen)
    m = _gradient(shape, gen).mul_(0.4)
    v = _second_moment(shape, gen)
    if unseen:
        gone = (torch.rand([shape[0]] + [1] * (len(shape) - 1), device="cuda", generator=gen) < unseen)
        for x in (g, m, v):
            x.masked_fill_(gone, 0.0)
    t = {"shape": shape, "p": p, "g": g.to(dtype), "n": n}
    if scheme == "auto":
        scheme = "fp32" if n <= 4096 else "rank1" if len(shape) == 2 or (nd_rank1 and len(shape) > 2) else "block"
    t["scheme"] = scheme
    if scheme == "fp32":
        return dict(t, m=m, v=v)
    t["m"], t["m_scale"] = _quantize_block(m, MM)
    if scheme == "rank1":
        t["maxima"] = _maxima(v)
        s = _smallest(t["maxima"])
        t["v"] = _codes(torch.where(s > 0, v / s, torch.zeros_like(v)), MV)
    else:
        t["v"], t["v_scale"] = _quantize_block(v, MV)
    return t


def _tensors(case, seed):
    gen, dtype = _generator(seed), DTYPES[case["dtype"]]
    if case["kind"] == "step":
        return [_tensor(s, dtype, gen, case["unseen"], nd_rank1=case["nd_rank1"]) for s in _shapes(case)]
    return [_tensor((case["n"],), dtype, gen, scheme="block" if case["kind"] == "fused_4bit" else "fp32")]


# ---- the passes ---------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "codec_block":
        return {"case": case, "m": _gradient((case["n"],), _generator(seed)), "v": _second_moment((case["n"],), _generator(seed + 1))}
    if kind == "codec_rank1":
        return {"case": case, "v": _second_moment((case["rows"], case["cols"]), _generator(seed))}
    ts = _tensors(case, seed)
    if kind != "step":
        return {"case": case, "t": ts[0]}
    params = [torch.nn.Parameter(t["p"]) for t in ts]
    options = {"capturable": True, "schedule_rows": 1024} if case["capturable"] else {"nd_rank1": True} if case["nd_rank1"] else {}
    opt = qf.FourBitAdamW(params, lr=LR, betas=(B1, B2), eps=EPS, weight_decay=WD, **options)
    state = {}
    for i, t in enumerate(ts):
        quantized = t["scheme"] != "fp32"
        momentum, variance = {}, {}
        if quantized:
            momentum["max1"] = t["m_scale"]
            variance.update({"max_dims": t["maxima"], "max1": None} if t["scheme"] == "rank1" else {"max1": t["v_scale"]}, dim=len(t["shape"]))
        state[i] = {"step": torch.tensor(float(case["step"])), "exp_avg": t["m"], "exp_avg_sq": t["v"],
                    "momentum_qstate": {"enable": quantized, "overhead": momentum, "qmap": None},
                    "variance_qstate": {"enable": quantized, "overhead": variance, "qmap": None}}
    opt.load_state_dict({"state": state, "param_groups": opt.state_dict()["param_groups"]})
    for p, t in zip(params, ts):
        p.grad = t["g"]
    return {"case": case, "opt": opt, "params": params, "scale": CLIP if case["clip"] else None}


def _state_tensors(opt, p):
    st = opt.state[p]
    momentum, variance = st["momentum_qstate"]["overhead"], st["variance_qstate"]["overhead"]
    out = [p.detach(), st["exp_avg"], st["exp_avg_sq"]]
    if "max1" in momentum:
        out.append(momentum["max1"])
        out += list(variance["max_dims"]) if variance.get("max_dims") is not None else [variance["max1"]]
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        opt = state["opt"]
        if state["scale"] is None:
            opt.step()
        else:
            opt.step(grad_scale=state["scale"])
        return [_state_tensors(opt, p) for p in state["params"]]
    if kind == "codec_block":
        mc, ms = F.quantize_m(state["m"])
        vc, vs = F.quantize_v_block(state["v"])
        return [mc, ms, F.dequantize_m(mc, ms, case["n"]), vc, vs, F.dequantize_v_block(vc, vs, case["n"])]
    if kind == "codec_rank1":
        c, row, col = F.quantize_v(state["v"])
        return [c, row, col, F.dequantize_v(c, row, col)]
    t = state["t"]
    if kind == "fused_4bit":
        F.fused_4bit(t["p"], t["g"], t["m"], t["v"], t["m_scale"], t["v_scale"], B1, B2, LR, WD, EPS, case["step"])
        return [t["p"], t["m"], t["v"], t["m_scale"], t["v_scale"]]
    F.fused_single_tensor(t["p"], t["g"], t["m"], t["v"], B1, B2, LR, WD, EPS, case["step"])
    return [t["p"], t["m"], t["v"]]


# ---- what a pass cannot do without, and how far another correct one may be ---------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "codec_block":   # fp32 in, 4 bits and one scale per block out, and back; twice
        n, blocks = case["n"], -(-case["n"] // BLOCK)
        return {"bytes": 2 * (8 * n + 2 * ((n + 1) // 2) + 8 * blocks), "flops": 6 * n}
    if kind == "codec_rank1":
        n = case["rows"] * case["cols"]
        return {"bytes": 8 * n + 2 * ((n + 1) // 2) + 8 * (case["rows"] + case["cols"]), "flops": 4 * n}
    size = 4 if case["dtype"] == "float32" else 2
    total = flops = 0
    for s in _shapes(case) if kind == "step" else [(case["n"],)]:
        n = math.prod(s)
        flops += 20 * n
        if kind == "fused_fp32" or (kind == "step" and n <= 4096):
            total += n * (3 * size + 16)
            continue
        blocks = -(-n // BLOCK)
        total += 3 * n * size + 4 * ((n + 1) // 2) + 8 * blocks
        rank1 = kind == "step" and (len(s) == 2 or (case["nd_rank1"] and len(s) > 2))
        total += 8 * sum(s) if rank1 else 8 * blocks
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Element-wise arithmetic in fp32: an implementation that rounds each operation differs from another in the last
    place at most.  A 16-bit parameter next to a rounding boundary may then move by one of its units (2^-8 or 2^-11 of its
    value; a few of a million do), a 4-bit code at a tie between two levels by one level (less than one in a million)."""
    half = case["kind"] in ("step", "fused_4bit", "fused_fp32") and case["dtype"] != "float32"
    return {"rel": 1e-5 if half else 1e-6, "max": 1e-2 if half else 1e-5, "differ": 1e-6}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------


def _exact_update(t, step, scale=None):
    n = t["n"]
    p, g = t["p"].double().reshape(-1), t["g"]
    g = (g.float() * scale).to(g.dtype) if scale is not None else g
    g = g.double().reshape(-1)
    if t["scheme"] == "fp32":
        m, v = t["m"].double().reshape(-1), t["v"].double().reshape(-1)
    else:
        m = (_blocks(_values(t["m"], n, QM)).double() * t["m_scale"].double()[:, None]).reshape(-1)[:n]
        if t["scheme"] == "rank1":
            v = (_values(t["v"], n, QV).view(t["shape"]).double() * _smallest(t["maxima"]).double()).reshape(-1)
        else:
            v = (_blocks(_values(t["v"], n, QV)).double() * t["v_scale"].double()[:, None]).reshape(-1)[:n]
    m = m + (1 - B1) * (g - m)
    v = B2 * v + (1 - B2) * g * g
    p = p * (1 - LR * WD) - LR / (1 - B1 ** step) * m / (v.sqrt() / math.sqrt(1 - B2 ** step) + EPS)
    if t["scheme"] == "fp32":
        return p.view(t["shape"]), m.view(t["shape"]), v.view(t["shape"])
    scales = [_blocks(m).abs().amax(dim=1)]
    scales += _maxima(v.view(t["shape"])) if t["scheme"] == "rank1" else [_blocks(v).amax(dim=1)]
    return p.view(t["shape"]), scales


def exact(case, seed):
    kind = case["kind"]
    if kind == "codec_block":
        out = []
        for x, mid, qmap in ((_gradient((case["n"],), _generator(seed)), MM, QM), (_second_moment((case["n"],), _generator(seed + 1)), MV, QV)):
            codes, scales = _quantize_block(x, mid)   # fp32: the codes are what the format defines
            y = (_blocks(_values(codes, case["n"], qmap)).double() * scales.double()[:, None]).reshape(-1)[:case["n"]]
            out += [None, scales.double(), y]
        return out
    if kind == "codec_rank1":
        v = _second_moment((case["rows"], case["cols"]), _generator(seed))
        row, col = _maxima(v)
        s = torch.minimum(row, col)
        y = _values(_codes(v / s, MV), v.numel(), QV).view(v.shape).double() * s.double()
        return [None, row.reshape(-1).double(), col.reshape(-1).double(), y]
    out = []
    for t in _tensors(case, seed):
        if kind == "step":
            r = _exact_update(t, case["step"] + 1, CLIP if case["clip"] else None)
        else:
            r = _exact_update(t, case["step"])
        out.append(list(r) if t["scheme"] == "fp32" else [r[0], None, None, *r[1]])
    return out if kind == "step" else out[0]
