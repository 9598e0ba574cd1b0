"""Performance cases: what a program that uses this package has it do, through the public entry points.

Seven kinds of work:

  encode    e8_encode_packed: values and scales -> packed codes (4 bytes per 8 values)
  decode    e8_decode_packed: packed codes and scales -> values
  roundtrip e8_encode_packed followed by e8_decode_packed in the same type (compressing a bf16 checkpoint
            or cache and reading it back)
  digits    e8_encode followed by e8_decode, the reference-shaped calls on float32 digit tensors
  host      HostCodec.encode followed by .decode on page-locked host arrays
  qat       one training step of an E8 layer: forward, then backward from the gradient of its output
  linear    inference with an E8CodeLinear: generation with few tokens, prefill with many
  exchange  the two device operations of the quantised gradient average on one of `ranks` GPUs: encode
            the own gradient, decode and average the gathered code streams

Sizes are those of the package's benchmarks and tests; `draw` spreads over the same ranges.
"""
import math

import torch

from coset_b200 import _lib
from coset_b200.core.base import LatticeConfig
from coset_b200.core.e8 import create_e8_hnlq_linear, e8_decode, e8_decode_packed, e8_encode, e8_encode_packed
from coset_b200.gradcomm import CudaCodec, bert_base_gradient_numel
from coset_b200.host import HostCodec
from coset_b200.vlut import E8CodeLinear

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}


def listed():
    return [
        # the bulk codec: a whole model's float32 weights at once, one scale per block of 8
        {"name": "encode_bulk", "kind": "encode", "n": 1 << 25, "dtype": "f32", "tile": 1},
        {"name": "decode_bulk", "kind": "decode", "n": 1 << 25, "dtype": "f32", "tile": 1},
        # one bf16 tensor of a checkpoint, one scale per row of 768 values, a length that is no multiple of anything
        {"name": "roundtrip_bf16_ragged", "kind": "roundtrip", "n": 1000003, "dtype": "bf16", "tile": 96},
        # the reference's own calls at its own test size: an ordinary small call
        {"name": "digits_64k", "kind": "digits", "n": 65536, "q": 4, "M": 2, "beta": 1.0},
        # arrays that live in host memory
        {"name": "host_4m", "kind": "host", "n": 1 << 22, "dtype": "f32", "tile": 1},
        # training: a feed-forward layer in bf16, and a small classifier head in float32 with a batch of 128
        {"name": "qat_ffn_bf16", "kind": "qat", "tokens": 4096, "n_in": 768, "n_out": 3072, "dtype": "bf16", "tiling": "row", "bias": True},
        {"name": "qat_head_f32", "kind": "qat", "tokens": 128, "n_in": 768, "n_out": 768, "dtype": "f32", "tiling": "block", "bias": True},
        # inference: one sequence and a batch of 16 sequences being generated, a short and a long prefill
        {"name": "linear_t1", "kind": "linear", "tokens": 1, "n_in": 4096, "n_out": 4096, "dtype": "bf16", "tiling": "row", "bias": True, "clip": 2.0},
        {"name": "linear_t16", "kind": "linear", "tokens": 16, "n_in": 4096, "n_out": 4096, "dtype": "bf16", "tiling": "block", "bias": False, "clip": 0.0},
        {"name": "linear_t256", "kind": "linear", "tokens": 256, "n_in": 4096, "n_out": 4096, "dtype": "bf16", "tiling": "row", "bias": True, "clip": 2.0},
        {"name": "linear_t4096", "kind": "linear", "tokens": 4096, "n_in": 4096, "n_out": 4096, "dtype": "bf16", "tiling": "block", "bias": False, "clip": 0.0},
        # data-parallel training: the whole gradient of a 109-million-parameter model, eight ranks
        {"name": "exchange_8", "kind": "exchange", "n": bert_base_gradient_numel() // 8, "ranks": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["encode", "decode", "roundtrip", "digits", "host", "qat", "qat", "linear", "linear", "linear", "exchange"])
    if kind in ("encode", "decode", "roundtrip"):
        # one scale per block, per row of 64 to 4096 values, or (tile 0) one for the whole tensor
        hi = 1 << 24 if kind == "roundtrip" else 1 << 25
        return {"kind": kind, "n": _log(rng, 1 << 12, hi), "dtype": rng.choice(["f32", "f32", "bf16"]), "tile": rng.choice([1, 1, 0, 8 * rng.randint(1, 64)])}
    if kind == "digits":
        q, M = rng.choice([(4, 2), (4, 2), (4, 2), (4, 1), (3, 2), (4, 3), (8, 2)])
        return {"kind": kind, "n": _log(rng, 1 << 8, 1 << 20), "q": q, "M": M, "beta": round(rng.uniform(0.5, 2.0), 3)}
    if kind == "host":
        return {"kind": kind, "n": _log(rng, 1 << 14, 1 << 22), "dtype": rng.choice(["f32", "bf16"]), "tile": rng.choice([1, 96, 0])}
    if kind == "exchange":
        return {"kind": kind, "n": _log(rng, 1 << 16, bert_base_gradient_numel() // 8), "ranks": rng.choice([2, 4, 8])}
    # feature counts: mostly multiples of 64, some only of 8; token counts of every size
    while True:
        step = rng.choice([64, 64, 64, 8])
        n_in = max(64, _log(rng, 128, 8192) // step * step)
        n_out = max(64, _log(rng, 128, 8192) // step * step)
        case = {"kind": kind, "n_in": n_in, "n_out": n_out, "dtype": rng.choice(["bf16", "bf16", "bf16", "f32"]),
                "tiling": rng.choice(["row", "block"]), "bias": rng.random() < 0.5}
        if kind == "qat":
            case["tokens"] = _log(rng, 32, 8192)
            if case["tokens"] * n_in * n_out <= 4096 ** 3 // 3:
                return case
        else:
            case["tokens"] = rng.choice([_log(rng, 1, 16), _log(rng, 16, 4096)])
            case["clip"] = rng.choice([0.0, 2.0])
            if case["tokens"] * n_in * n_out <= 4096 ** 3:
                return case


# ------------------------------------------------------------------ inputs
def _values(n, g, sigma=0.02):
    """n values of a trained weight tensor: N(0, sigma), 0.1 % outliers of 10 sigma, clipped to +-2."""
    x = torch.randn(n, device="cuda", generator=g) * sigma
    u = torch.rand(n, device="cuda", generator=g)
    x = torch.where(u < 5e-4, 10.0 * sigma, torch.where(u > 1.0 - 5e-4, -10.0 * sigma, x))
    return x.clamp_(-2.0, 2.0)


def _scales(tiles, g):
    """Trained scales: 25 +- 20 %, which brings N(0, 0.02) to about half a lattice step."""
    return 25.0 * (0.8 + 0.4 * torch.rand(tiles, device="cuda", generator=g))


def _tiles(case):
    """(number of scales, blocks per scale) of a codec case."""
    tile = case["tile"] if case["tile"] else case["n"]
    return (case["n"] + tile - 1) // tile, tile


def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind in ("encode", "decode", "roundtrip", "host"):
        n = case["n"]
        tiles, tile = _tiles(case)
        x = _values(8 * n, g).view(n, 8).to(DTYPES[case["dtype"]])
        s = {"kind": kind, "scale": _scales(tiles, g), "tile": tile, "dtype": DTYPES[case["dtype"]]}
        if kind == "decode":
            s["codes"] = e8_encode_packed(x, scale=s["scale"], scale_mode=_lib.SCALE_MUL_TILE, blocks_per_tile=tile)
        elif kind == "host":
            s["x"], s["scale"] = x.cpu().pin_memory(), s["scale"].cpu().pin_memory()
            s["codes"] = torch.empty((n, 4), dtype=torch.uint8, pin_memory=True)
            s["out"] = torch.empty((n, 8), dtype=s["dtype"], pin_memory=True)
            # tiles do not straddle the staging chunks; one scale for everything means one chunk
            s["codec"] = HostCodec(chunk_blocks=n) if case["tile"] == 0 else HostCodec()
        else:
            s["x"] = x
        return s
    if kind == "digits":
        config = LatticeConfig(lattice_type="E8", q=case["q"], M=case["M"], beta=case["beta"])
        return {"kind": kind, "x": torch.randn(case["n"], 8, device="cuda", generator=g).clamp_(-2.0, 2.0), "config": config}
    if kind == "exchange":
        n, ranks = case["n"], case["ranks"]
        codec, scale = CudaCodec(), 500.0
        gathered = torch.zeros((ranks, n), dtype=torch.int32, device="cuda")
        for r in range(1, ranks):  # the code streams the other ranks sent
            codec.encode(torch.randn(n, 8, device="cuda", generator=g) * 1e-3, scale, gathered[r])
        grad = torch.randn(n, 8, device="cuda", generator=g) * 1e-3
        return {"kind": kind, "codec": codec, "scale": scale, "grad": grad, "gathered": gathered, "out": torch.empty_like(grad)}
    n_in, n_out, tokens, dtype = case["n_in"], case["n_out"], case["tokens"], DTYPES[case["dtype"]]
    x = torch.randn(tokens, n_in, device="cuda", generator=g).to(dtype)
    bias = torch.randn(n_out, device="cuda", generator=g) * 0.02 if case["bias"] else None
    if kind == "linear":
        bpt = 1 if case["tiling"] == "block" else n_in // 8
        weight = _values(n_out * n_in, g).view(n_out, n_in)
        lin = E8CodeLinear.from_weight(weight, _scales(n_out * (n_in // 8) // bpt, g), bpt, bias, weight_clip_value=case["clip"])
        return {"kind": kind, "x": x, "layer": lin}
    layer = create_e8_hnlq_linear(n_in, n_out, device="cuda", tiling=case["tiling"], bias=case["bias"], init_method="zeros")
    # at the layer's initial scales a weight spread of 20 uses the whole code range (one of 0.02 quantises to zero)
    layer.load_weights(torch.randn(n_out, n_in, device="cuda", generator=g) * 20.0, bias)
    grad = torch.randn(tokens, n_out, device="cuda", generator=g).to(dtype)
    return {"kind": kind, "x": x.requires_grad_(), "grad": grad, "layer": layer}


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "encode":
        return e8_encode_packed(s["x"], scale=s["scale"], scale_mode=_lib.SCALE_MUL_TILE, blocks_per_tile=s["tile"])
    if kind == "decode":
        return e8_decode_packed(s["codes"], scale=s["scale"], scale_mode=_lib.SCALE_MUL_TILE, blocks_per_tile=s["tile"], dtype=s["dtype"])
    if kind == "roundtrip":
        codes = e8_encode_packed(s["x"], scale=s["scale"], scale_mode=_lib.SCALE_MUL_TILE, blocks_per_tile=s["tile"])
        return codes, e8_decode_packed(codes, scale=s["scale"], scale_mode=_lib.SCALE_MUL_TILE, blocks_per_tile=s["tile"], dtype=s["dtype"])
    if kind == "digits":
        digits, _ = e8_encode(s["x"], s["config"])
        return digits, e8_decode(digits, s["config"])
    if kind == "host":
        kw = {"scale": s["scale"], "scale_mode": _lib.SCALE_MUL_TILE, "blocks_per_tile": s["tile"]}
        s["codec"].encode(s["x"], out=s["codes"], **kw)
        s["codec"].decode(s["codes"], dtype=s["dtype"], out=s["out"], **kw)
        return s["codes"], s["out"]
    if kind == "exchange":
        gathered = s["gathered"]
        s["codec"].encode(s["grad"], s["scale"], gathered[0])
        s["codec"].decode_mean(gathered, gathered.shape[0], gathered.shape[1], s["scale"], s["out"])
        return gathered[0], s["out"]
    layer, x = s["layer"], s["x"]
    if kind == "linear":
        with torch.no_grad():
            return layer(x)
    layer.zero_grad(set_to_none=True)
    x.grad = None
    y = layer(x)
    y.backward(s["grad"])
    out = {"y": y.detach(), "dx": x.grad, "dw": layer.weight.grad, "dtheta": layer.theta_beta.grad}
    if layer.bias is not None:
        out["dbias"] = layer.bias.grad
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("encode", "decode", "roundtrip", "host"):
        row = 32 if case["dtype"] == "f32" else 16
        one_way = case["n"] * (row + 4) + 4 * _tiles(case)[0]
        if kind == "roundtrip":  # the codes are written once and need not be read back
            return {"bytes": case["n"] * (2 * row + 4) + 4 * _tiles(case)[0]}
        return {"bytes": 2 * one_way if kind == "host" else one_way}
    if kind == "digits":  # values in, float32 digits out, values out
        return {"bytes": case["n"] * (64 + 32 * case["M"])}
    if kind == "exchange":
        return {"bytes": case["n"] * (64 + 4 * case["ranks"])}
    T, n_in, n_out = case["tokens"], case["n_in"], case["n_out"]
    elem = 4 if case["dtype"] == "f32" else 2
    scales = n_out if case["tiling"] == "row" else n_out * n_in // 8
    bias = 4 * n_out if case["bias"] else 0
    if kind == "linear":
        return {"bytes": n_out * n_in // 2 + 4 * scales + bias + elem * T * (n_in + n_out), "flops": 2 * T * n_in * n_out}
    # weights, scales and activations in, output out; gradient of the output in, four gradients out
    return {"bytes": 8 * n_out * n_in + 8 * scales + 2 * bias + 2 * elem * T * (n_in + n_out), "flops": 6 * T * n_in * n_out}


def tolerance(case):
    if case["kind"] in ("qat", "linear"):
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 1e-5}
    return "exact"  # codes are whole numbers, and every reconstruction is one correctly rounded operation on whole numbers
