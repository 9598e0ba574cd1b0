"""Inference with weights kept as E8 codes: E8CodeLinear.

The weight of a trained HNLQLinearQAT layer is exported as packed q=4, M=2 codes (4 bytes per 8
weights) plus the scales beta, and applied from the codes:

  * few tokens  (T <= small_t_max): by default a decode-ready copy of the codes, one byte per weight in tensor-core order
    (coset_e8_vlut_layout), and coset_e8_vlut_product_checked, which compares the copy with the codes as it reads it, so that
    the result is that of the codes however they were written; `large_t_path="tcgen05"` keeps no copy of any kind and
    reads the code stream (coset_e8_vlut_gemv);
  * many tokens (from 2048 by default): the weight is decoded into a transient bf16 buffer and multiplied by
    this library's tcgen05 GEMM (coset_e8_decode_gemm); nothing dense survives the call;
  * in between, by default, this library's product with a kept dense bf16 copy (coset_e8_dense_linear) up to 2^34 multiply-adds and
    torch's beyond, for very long rows and in graphs of small layers (`large_t_path` chooses).

The math is the reference's one-sided vLUT inner product (coset/legacy/quant/vlut.py:72-117) in
the layer's scale convention W_q = decode(codes) / beta (coset/core/layers.py:453-460).
"""
from typing import Optional

import torch
import torch.nn as nn

from . import _lib
from .core.e8.codecs import _DTYPE_CODES, e8_decode_packed, e8_encode_packed


def e8_vlut_matmul(codes: torch.Tensor, beta: Optional[torch.Tensor], blocks_per_tile: int, x: torch.Tensor,
                   bias: Optional[torch.Tensor] = None, clip: float = 0.0, out_dtype: torch.dtype = torch.float32) -> torch.Tensor:
    """y = x @ Wq.T + bias with Wq = decode(codes) / beta (clamped to +-clip when clip > 0);
    codes int32 [n_out, n_in / 8]; x [T, n_in]; y float32, or bf16 rounded once from the float32 sums."""
    _lib.require_cuda(x, "x")
    if x.dim() != 2:
        raise ValueError(f"x must be [T, n_in], got {tuple(x.shape)}")
    return _lib.native().vlut_linear(x, codes, beta, int(blocks_per_tile), bias, float(clip), _DTYPE_CODES.get(out_dtype, -1))


def e8_dequant_gemm(codes: torch.Tensor, beta: Optional[torch.Tensor], blocks_per_tile: int, x: torch.Tensor,
                    bias: Optional[torch.Tensor] = None, check: bool = False, clip: float = 0.0,
                    status: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Same product as e8_vlut_matmul for many tokens, on the tcgen05 tensor cores: weight tiles are
    decoded to bf16 in shared memory and never written to HBM.  x: bf16 [T, n_in], n_in % 64 == 0.
    check=True synchronises and raises if a bounded barrier wait expired inside the kernel."""
    _lib.require_cuda(codes, "codes")
    _lib.require_cuda(x, "x")
    if x.dtype != torch.bfloat16:
        raise TypeError("e8_dequant_gemm takes bfloat16 activations")
    if codes.dtype != torch.int32 or codes.dim() != 2 or not codes.is_contiguous():
        raise ValueError("codes must be a contiguous int32 tensor [n_out, n_in / 8]")
    n_out, kb = codes.shape
    if x.dim() != 2 or x.shape[1] != kb * 8 or (kb * 8) % 64:
        raise ValueError(f"x must be [T, {kb * 8}] with n_in a multiple of 64, got {tuple(x.shape)}")
    x = x.contiguous()
    T = x.shape[0]
    y = torch.empty((T, n_out), dtype=torch.float32, device=x.device)
    if status is None:
        status = torch.zeros(1, dtype=torch.int32, device=x.device)
    b = beta.to(torch.float32).contiguous().view(-1) if beta is not None else None
    bias32 = bias.to(torch.float32).contiguous() if bias is not None else None
    with torch.cuda.device(x.device):
        rc = _lib.lib().coset_e8_dequant_gemm(_lib.ptr(codes), _lib.ptr(b) if b is not None else None,
                                              int(blocks_per_tile), n_out, kb * 8, _lib.ptr(x), x.stride(0), T,
                                              _lib.ptr(bias32) if bias32 is not None else None, _lib.ptr(y),
                                              y.stride(0), float(clip), _lib.ptr(status), _lib.stream())
    _lib.check(rc, "coset_e8_dequant_gemm")
    if check and int(status.item()) != 0:
        raise RuntimeError("coset_e8_dequant_gemm: a barrier wait expired inside the kernel; the result is invalid")
    return y


def e8_decode_gemm(codes: torch.Tensor, beta: Optional[torch.Tensor], blocks_per_tile: int, x: torch.Tensor,
                   bias: Optional[torch.Tensor] = None, check: bool = False, clip: float = 0.0,
                   scratch: Optional[torch.Tensor] = None, out_dtype=torch.float32,
                   status: Optional[torch.Tensor] = None) -> torch.Tensor:
    """The product of e8_dequant_gemm in two launches: the weight is decoded to bf16 into `scratch` (transient,
    n_out * n_in bf16 values, allocated here when not given) and multiplied by a TMA-fed tcgen05 GEMM on pairs
    of CTAs (cta_group::2).  Same bits as e8_dequant_gemm and, measured, the same speed up to 8192 tokens, a few
    percent more beyond; nothing dense survives the call.  out_dtype: float32 or bfloat16 (rounded once from the
    float32 accumulator)."""
    if out_dtype not in _DTYPE_CODES:
        raise TypeError("out_dtype must be float32 or bfloat16")
    _lib.require_cuda(x, "x")
    if x.dim() != 2:
        raise ValueError(f"x must be [T, n_in] with n_in a multiple of 64, got {tuple(x.shape)}")
    y, status = _lib.native().decode_gemm(x, codes, beta, int(blocks_per_tile), bias, float(clip), scratch, _DTYPE_CODES[out_dtype], status)
    if check and int(status.item()) != 0:
        raise RuntimeError("coset_e8_decode_gemm: a barrier wait expired inside the kernel; the result is invalid")
    return y


class E8CodeLinear(nn.Module):
    """Linear layer that owns E8 codes + scales instead of a dense weight (inference only).

    Its state_dict is self-describing (codes, beta, bias, blocks_per_tile, weight_clip_value), so a
    layer can be rebuilt from a checkpoint alone with `E8CodeLinear.from_state_dict`.
    Up to small_t_max tokens go to the code-domain kernels; more bf16 tokens go to (large_t_path): "tcgen05" --
    this library's tensor-core kernels, which keep no dense weight: decode to a transient bf16 buffer + TMA-fed
    cta_group::2 GEMM from 1024 tokens, the single-launch fused kernel below; "cublas" -- a cached dense bf16 copy
    and the library GEMM; "auto" (default) -- the own kernels from PAIR_GEMM_MIN_T tokens, the kept dense copy for
    the tokens in between, where decoding the whole weight per call costs more than the product itself (multiplied by this library's kernel
    or by torch's, whichever is quicker; see DENSE_OWN_MAX).
    Few tokens use a one-byte-per-weight copy laid out on the first such call ("auto", "cublas"): 9-13 us for 1-16
    tokens and a 4096 x 4096 weight; the kernel checks the copy against the codes in every call.  "tcgen05" keeps nothing and
    stays on the code-domain kernels (9.7-23 us).
    A call under graph capture reads the codes, scales and bias themselves (it decodes the weight where it would use the dense
    copy), so that a replay follows writes to them and reads nothing that a later call gives back.  The dense copy follows
    writes that PyTorch's version counters show; see forget_copies for the others.  The kernels of the two routes add up in
    different orders (and for 3-16 bf16 tokens the one that reads the codes rounds the scaled weights to bf16), so a call and its
    replay agree to the precision of the type, not to the bit.
    small_t_max defaults to 16 ("auto", "cublas") or 48 ("tcgen05"): measured on a 4096 x 4096 layer the
    code-domain kernels take 9.7 / 23 / 44 / 86 us for 1 / 16 / 32 / 64 tokens (they re-read and re-decode the
    codes for every 16 tokens), the library on the cached copy 7-13 us, the fused kernel 64 us.
    weight_clip_value > 0: the weights are clamp(decode(codes) / beta, +-clip), the clamp the training
    layer applies after de-scaling (coset/core/layers.py:463); 0 disables it."""

    # The library's own product with the kept dense copy costs the host one launch where torch's costs a library call and, with a bias, its cast, and that bounds
    # such a call: 4096 x 4096, own / torch with a bias / without, us a call: 17 tokens 8.5 / 19.2 / 14.9, 256 tokens 11.7 / 19.3 / 14.8, 1024 tokens
    # 24.6 / 27.8 / 24.7; 8192 x 8192 and 256 tokens 35 / 37 / 33.5.  Beyond 2^34 multiply-adds torch's is quicker, and so it is where few CTAs sum over
    # a long row ([64, 65536] with 17 tokens 29 / 21 / 17.5; [128, 32768] 16.6 / 21.5 / 17.4).
    DENSE_OWN_MAX, DENSE_OWN_MAX_IN = 1 << 34, 1 << 15
    # In a graph the host costs nothing: the own product pays where its start under the decoding before it counts, in large weights, the sooner with a
    # bias to cast, and where torch's splits long rows (replays with 256 tokens, own / torch, us: 4096 x 4096 with a bias 23.0 / 23.1, without
    # 22.9 / 21.8; 8192 x 8192 76 / 81, 76 / 79; 3072 x 768 without 9.6 / 8.1; 64 x 8192 10.4 / 16.6, 10.3 / 15.4).
    DENSE_CAPTURED_MIN, DENSE_CAPTURED_MIN_NO_BIAS, DENSE_CAPTURED_LONG = 1 << 24, 1 << 25, 1 << 13
    PAIR_GEMM_MIN_T = 2048  # from here on the decode + cta_group::2 GEMM is within 10-25 % of the library on a dense copy

    def __init__(self, codes: torch.Tensor, beta: torch.Tensor, blocks_per_tile: int,
                 bias: Optional[torch.Tensor] = None, small_t_max: Optional[int] = None, large_t_path: str = "auto",
                 weight_clip_value: float = 0.0):
        super().__init__()
        self.out_features, kb = codes.shape
        self.in_features = kb * 8
        if large_t_path not in ("auto", "cublas", "tcgen05"):
            raise ValueError("large_t_path must be 'auto', 'cublas' (dequantise once, keep the dense copy, library GEMM) "
                             "or 'tcgen05' (this library's tensor-core kernels only, no dense copy kept)")
        self.large_t_path = large_t_path
        self.small_t_max = int(small_t_max) if small_t_max is not None else (48 if large_t_path == "tcgen05" else 16)
        self.register_buffer("codes", codes.contiguous())
        self.register_buffer("beta", beta.to(torch.float32).contiguous().view(-1))
        self.register_buffer("bias", bias.detach().clone() if bias is not None else None)
        self.register_buffer("blocks_per_tile_t", torch.tensor(int(blocks_per_tile), dtype=torch.int64))
        self.register_buffer("weight_clip_value_t", torch.tensor(float(weight_clip_value), dtype=torch.float32))
        self.blocks_per_tile = int(blocks_per_tile)
        self.weight_clip_value = float(weight_clip_value)
        self._kept = {}      # copies of the weight in other forms, see _keep
        self._rows = self.out_features  # of the whole weight, where this layer holds a shard of its rows
        self._status = None  # device word the tensor-core kernels set when a bounded wait gave up

    def _load_from_state_dict(self, state_dict, prefix, *args, **kwargs):
        super()._load_from_state_dict(state_dict, prefix, *args, **kwargs)
        self.blocks_per_tile = int(self.blocks_per_tile_t.item())
        self.weight_clip_value = float(self.weight_clip_value_t.item())
        self._kept = {}

    def __getstate__(self):  # a copied or pickled layer makes its own copies of the weight again
        return {**self.__dict__, "_kept": {}}

    def __setstate__(self, state):
        super().__setstate__({k: v for k, v in state.items() if k not in ("_dense", "_dense_key")})
        self.__dict__.setdefault("_kept", {})
        self.__dict__.setdefault("_rows", self.out_features)

    @classmethod
    def from_weight(cls, weight: torch.Tensor, beta: torch.Tensor, blocks_per_tile: int, bias=None, **kw):
        """Quantise a dense float32 weight [n_out, n_in] with scales beta (layer convention)."""
        _lib.require_cuda(weight, "weight")
        n_out, n_in = weight.shape
        if n_in % 8:
            raise ValueError(f"Input dimension {n_in} must be divisible by 8 for E8 lattice")
        packed = e8_encode_packed(weight.contiguous().view(-1, 8), 4, 2, scale=beta.contiguous().view(-1),
                                  scale_mode=_lib.SCALE_MUL_TILE, blocks_per_tile=blocks_per_tile)
        codes = packed.view(torch.int32).view(n_out, n_in // 8)
        return cls(codes, beta, blocks_per_tile, bias, **kw)

    @classmethod
    def from_qat_layer(cls, layer, **kw):
        """Export of a trained HNLQLinearQAT (q must be 4): codes, scales, bias and the layer's
        weight_clip_value, so that this layer computes what the trained one computes."""
        return cls.from_exported(layer.export_quantized(packed=True), **kw)

    @classmethod
    def from_exported(cls, exported: dict, **kw):
        """Rebuild from HNLQLinearQAT.export_quantized(packed=True)."""
        meta = exported["metadata"]
        if meta.get("q") != 4 or meta.get("packed_M", 2) != 2:
            raise ValueError("E8CodeLinear stores q=4, M=2 codes")
        kw.setdefault("weight_clip_value", meta.get("weight_clip_value", 0.0))
        return cls(exported["codes"], exported["beta"], int(exported["blocks_per_tile"]), exported.get("bias"), **kw)

    @classmethod
    def from_state_dict(cls, state_dict: dict, prefix: str = "", **kw):
        """Rebuild from a checkpoint of this class alone (no codes in hand)."""
        g = lambda k: state_dict[prefix + k]
        bias = state_dict.get(prefix + "bias")
        kw.setdefault("weight_clip_value", float(g("weight_clip_value_t")))
        return cls(g("codes"), g("beta"), int(g("blocks_per_tile_t")), bias, **kw)

    def dense_weight(self, dtype=torch.float32) -> torch.Tensor:
        """Wq = clamp(decode(codes) / beta) as a dense [n_out, n_in] tensor."""
        # rounding to bf16 keeps the order, so the clamp of the rounded weights is the rounded clamp
        first = torch.float32 if self.weight_clip_value > 0 and dtype is not torch.bfloat16 else dtype
        w = e8_decode_packed(self.codes.view(-1), 4, 2, scale=self.beta, scale_mode=_lib.SCALE_MUL_TILE,
                             blocks_per_tile=self.blocks_per_tile, dtype=first)
        if self.weight_clip_value > 0:
            w = w.clamp_(-self.weight_clip_value, self.weight_clip_value).to(dtype)
        return w.view(self.out_features, self.in_features)

    def _keep(self, name, sources, settings, make):
        """`make()`, kept until one of the buffers it was made from is seen to be written or replaced (the entry holds the buffers,
        so their identity cannot be taken over by another tensor).  A call on another stream than the one that made it waits there
        for the copy and marks it as used, so that it may be replaced or dropped at any time.  Inside a graph capture it is made
        in the call and not kept: a replay follows its sources, and reads no memory that a later call gives back."""
        if torch._C._cuda_isCurrentStreamCapturing():
            return make()
        device = sources[0].get_device()
        stream = torch._C._cuda_getCurrentRawStream(device)
        entry = self._kept.get(name)
        if entry is not None and entry[1] == settings:
            for t, (kept, version, pointer) in zip(sources, entry[2]):
                if t is not kept or t._version != version or t.data_ptr() != pointer:
                    break
            else:
                if entry[3] != stream:
                    here = torch.cuda.current_stream(device)
                    here.wait_event(entry[4])
                    entry[0].record_stream(here)
                return entry[0]
        if any(t.is_inference() for t in sources):  # no version counter: a write would go unseen
            return make()
        state = [(t, t._version, t.data_ptr()) for t in sources]
        value = make()
        made = torch.cuda.current_stream(device).record_event()
        self._kept[name] = (value, settings, state, stream, made)
        return value

    def forget_copies(self):
        """Drops the copies of the weight in other forms; the next call makes them again.  The dense copy of the library path
        follows writes that the buffers' version counters show; a write to the codes or scales by `.data`, a collective or a
        replayed graph shows in none, and wants this call behind it.  Few tokens do not need it: their kernel checks its copy."""
        self._kept = {}

    def _apply(self, fn, *args, **kwargs):
        self._kept = {}  # neither the copies nor the buffers they were made from outlive a move
        return super()._apply(fn, *args, **kwargs)

    @property
    def _dense(self):
        return self._kept["dense"][0] if "dense" in self._kept else None

    def _product_layout(self):
        """The weight as bytes in tensor-core order (coset_e8_vlut_layout), 1 byte per weight; None where the call has to
        read the codes themselves: under capture, for a graph is replayed on whatever the codes then hold, and for codes
        without a version counter."""
        codes = self._buffers["codes"]
        if torch._C._cuda_isCurrentStreamCapturing() or codes.is_inference():
            return None
        return self._keep("layout", (codes,), None, self._make_layout)

    def _codes_are_faster(self, T, dtype):
        """Whether the kernel that reads the codes beats the one that reads the layout: one or two float32 tokens, where the layout's
        three products per weight cost more than one decoding unless many rows share the chip.  Codes against layout, us: scales
        per block, 1024 x 8192 one token 7.5 / 23.6, two 8.7 / 23.6; 2048 x 4096 8.5 / 13.5, 10.4 / 13.5; 4096 x 4096 14.2 / 15.6,
        15.9 / 15.5; 8192 x 8192 41 / 52, 53 / 52; but 8192 x 512 9.8 / 6.8; per row, 1024 x 8192 10.0 / 15.7, 2048 x 2048
        8.0 / 6.3.  Below 2^22 weights the host takes longer than either.  The rule sees the whole weight, so that the
        shards of a layer return its bits."""
        if T > 2 or dtype is torch.bfloat16 or self._rows * self.in_features < 1 << 22:
            return False
        if self.blocks_per_tile % (self.in_features // 8) == 0:
            return self._rows <= 1024
        return self.in_features >= 1024 and (T == 1 or self._rows <= 2048)

    def _make_layout(self):
        return _lib.native().vlut_layout(self._buffers["codes"])

    def _dense_bf16(self):
        buf = self._buffers
        return self._keep("dense", (buf["codes"], buf["beta"]), (self.weight_clip_value, self.blocks_per_tile), self._make_dense)

    def _make_dense(self):
        return self.dense_weight(torch.bfloat16)

    def check(self):
        """Synchronises and raises if a bounded barrier wait expired inside one of the tensor-core kernels since
        the last check (their results are then invalid).  The kernels never hang: they give up after 0.2 s."""
        if self._status is not None and int(self._status.item()) != 0:
            self._status.zero_()
            raise RuntimeError("E8CodeLinear: a barrier wait expired inside a tensor-core kernel; results since the last check are invalid")

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        # the module's attribute look-up is a Python call per buffer; the dictionaries are read directly
        buf, n_in, dtype = self._buffers, self.in_features, x.dtype
        T = x.numel() // n_in
        if T <= self.small_t_max:
            layout = self._product_layout() if self.large_t_path != "tcgen05" and n_in and not self._codes_are_faster(T, dtype) else None
            if layout is not None:
                return _lib.native().vlut_product_checked(x, buf["codes"], layout, buf["beta"], self.blocks_per_tile, buf["bias"],
                                                          self.weight_clip_value, _lib.DTYPE_BF16 if dtype is torch.bfloat16 else _lib.DTYPE_F32)
            return _lib.native().vlut_linear(x, buf["codes"], buf["beta"], self.blocks_per_tile, buf["bias"], self.weight_clip_value,
                                             _lib.DTYPE_BF16 if dtype is torch.bfloat16 else _lib.DTYPE_F32)
        if dtype is torch.bfloat16:
            if n_in % 64 == 0 and (self.large_t_path == "tcgen05" or (self.large_t_path == "auto" and T >= self.PAIR_GEMM_MIN_T)):
                if self._status is None or self._status.device != x.device:
                    self._status = torch.zeros(1, dtype=torch.int32, device=x.device)
                if T >= 1024:
                    return _lib.native().decode_gemm(x, buf["codes"], buf["beta"], self.blocks_per_tile, buf["bias"], self.weight_clip_value,
                                                     None, _lib.DTYPE_BF16, self._status)[0]
                y = e8_dequant_gemm(buf["codes"], buf["beta"], self.blocks_per_tile, x.reshape(-1, n_in), buf["bias"],
                                    clip=self.weight_clip_value, status=self._status).to(dtype)
                return y.reshape(*x.shape[:-1], self.out_features)
        if x.dim() != 2:  # with other shapes and strides the library may add the bias to the rounded product
            return self.forward(x.reshape(-1, n_in)).reshape(*x.shape[:-1], self.out_features)
        if dtype is torch.float32:
            return torch.nn.functional.linear(x, self.dense_weight(torch.float32), buf["bias"])
        b, w = buf["bias"], self._dense_bf16()
        if dtype is torch.bfloat16 and type(x) is torch.Tensor and torch._C._get_tracing_state() is None and not torch._C._len_torch_function_stack():
            capturing = torch._C._cuda_isCurrentStreamCapturing()
            weights = n_in * self.out_features
            own = (self.large_t_path == "auto" and T < self.PAIR_GEMM_MIN_T and T * weights <= self.DENSE_OWN_MAX and n_in <= self.DENSE_OWN_MAX_IN
                   and not (capturing and n_in < self.DENSE_CAPTURED_LONG and weights < (self.DENSE_CAPTURED_MIN if b is not None else self.DENSE_CAPTURED_MIN_NO_BIAS)))
            status = self._status
            if own and (status is None or status.device != x.device):  # not inside a capture, whose memory is the graph's
                status = self._status = None if capturing else torch.zeros(1, dtype=torch.int32, device=x.device)
            return _lib.native().dense_linear(x, w, b, status, own)
        return torch.nn.functional.linear(x, w.to(dtype), b.to(dtype) if b is not None else None)


def out_feature_shard(n_out: int, world: int, rank: int):
    """[start, stop) of the output features rank `rank` owns: contiguous, equal sizes (n_out must
    divide by world so that the gathered result needs no padding)."""
    if world < 1 or not 0 <= rank < world:
        raise ValueError(f"rank {rank} outside world of {world}")
    if n_out % world:
        raise ValueError(f"out_features {n_out} must be divisible by the world size {world}")
    per = n_out // world
    return rank * per, (rank + 1) * per


def assemble_gathered(gathered: torch.Tensor) -> torch.Tensor:
    """[world, T, n_out / world] (the layout an all-gather of the local products yields) -> [T, n_out]."""
    world, T, per = gathered.shape
    return gathered.permute(1, 0, 2).reshape(T, world * per)


class ColumnParallelE8CodeLinear(nn.Module):
    """E8CodeLinear sharded along the output features over a process group: every rank owns the
    codes and scales of out_features / world rows, multiplies the (replicated) activations with
    them and the slices are exchanged with one all-gather of [T, out_features / world] floats.

    The codes never cross the link; at T = 1 the all-gather is latency-bound.

    transport="peer" (few tokens, T <= local.small_t_max): the product kernel writes every result row
    straight into the result buffer of EVERY rank (symmetric memory, plain stores over NVLink), the
    library's bounded cross-rank arrival follows (coset_b200.peer), and no all-gather is issued."""

    def __init__(self, local: E8CodeLinear, out_features: int, group=None, transport: str = "nccl", timeout_ms: int = 2000):
        super().__init__()
        import torch.distributed as dist
        if transport not in ("nccl", "peer"):
            raise ValueError("transport must be 'nccl' or 'peer'")
        self.transport = transport
        self.timeout_ms = int(timeout_ms)
        self._region, self._cap_tokens, self._parity = None, 0, 0  # symmetric result buffer [2, tokens, out_features]
        self.local = local
        self.group = group
        self.world = dist.get_world_size(group)
        self.rank = dist.get_rank(group)
        self.out_features = out_features
        self.in_features = local.in_features
        lo, hi = out_feature_shard(out_features, self.world, self.rank)
        if local.out_features != hi - lo:
            raise ValueError(f"local shard has {local.out_features} rows, expected {hi - lo}")
        local._rows = out_features

    @classmethod
    def from_weight(cls, weight: torch.Tensor, beta: torch.Tensor, blocks_per_tile: int, bias=None, group=None,
                    transport: str = "nccl", **kw):
        """Quantise this rank's rows of a full [n_out, n_in] weight; beta holds the scales of the
        full weight (one per block for blocks_per_tile = 1, one per row for n_in / 8)."""
        import torch.distributed as dist
        n_out, n_in = weight.shape
        lo, hi = out_feature_shard(n_out, dist.get_world_size(group), dist.get_rank(group))
        tiles_per_row = (n_in // 8) // int(blocks_per_tile)
        if tiles_per_row * int(blocks_per_tile) * 8 != n_in:
            raise ValueError("a scale tile must not straddle two rows")
        b = beta.contiguous().view(-1)[lo * tiles_per_row:hi * tiles_per_row]
        local = E8CodeLinear.from_weight(weight[lo:hi].contiguous(), b, blocks_per_tile,
                                         bias[lo:hi] if bias is not None else None, **kw)
        return cls(local, n_out, group, transport)

    def _forward_peer(self, x2: torch.Tensor) -> torch.Tensor:
        import ctypes
        import torch.distributed as dist
        from .peer import SymmetricRegion
        T = x2.shape[0]
        if T > self._cap_tokens:  # collective: every rank sees the same sequence of token counts
            if self._region is not None:  # peers may still be writing into the old allocation
                torch.cuda.synchronize(x2.device)
                dist.barrier(group=self.group)
            self._cap_tokens = T
            self._region = SymmetricRegion(2 * T * self.out_features * 4, x2.device, self.group, self.timeout_ms)
            self._parity = 0
        region, parity = self._region, self._parity
        self._parity ^= 1
        half_elems = self._cap_tokens * self.out_features
        lo, _ = out_feature_shard(self.out_features, self.world, self.rank)
        offset = (parity * half_elems + lo) * 4  # this rank's columns inside half `parity`
        targets = region.pointers(offset)
        loc = self.local
        x2 = x2.contiguous()
        bias32 = loc.bias.to(torch.float32).contiguous() if loc.bias is not None else None
        with torch.cuda.device(x2.device):
            bias = _lib.ptr(bias32) if bias32 is not None else None
            layout = (loc._product_layout() if loc.large_t_path != "tcgen05" and loc.in_features and not loc._codes_are_faster(T, x2.dtype)
                      else None)
            if layout is not None:  # the kernel of the unsharded layer, so that the results are the same bits
                rc = _lib.lib().coset_e8_vlut_product_checked(
                    _lib.ptr(loc.codes), _lib.ptr(layout), _lib.ptr(loc.beta), loc.blocks_per_tile, loc.out_features, loc.in_features,
                    _lib.ptr(x2), _lib.dtype_code(x2, "x"), x2.stride(0), T, bias, ctypes.cast(targets, ctypes.c_void_p), self.world,
                    _lib.DTYPE_F32, self.out_features, float(loc.weight_clip_value), _lib.stream())
            else:
                rc = _lib.lib().coset_e8_vlut_gemv_scatter(
                    _lib.ptr(loc.codes), _lib.ptr(loc.beta), loc.blocks_per_tile, loc.out_features, loc.in_features,
                    _lib.ptr(x2), _lib.dtype_code(x2, "x"), x2.stride(0), T, bias, ctypes.cast(targets, ctypes.c_void_p), self.world,
                    self.out_features, float(loc.weight_clip_value), _lib.stream())
        _lib.check(rc, "few-token product into every rank's buffer")
        region.arrive()  # bounded: all ranks have written their columns into this rank's buffer
        # the half is written again two calls from now, after the arrival of the call in between
        mine = region.data(torch.float32)[parity * half_elems: parity * half_elems + T * self.out_features]
        return mine.view(T, self.out_features).clone()

    def check(self):
        """Raises if a bounded cross-rank wait of the peer-store path, or a bounded barrier wait inside a
        tensor-core kernel of the local product, gave up (synchronises)."""
        self.local.check()
        if self._region is not None:
            self._region.check()

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        import torch.distributed as dist
        lead = x.shape[:-1]
        x2 = x.reshape(-1, self.in_features)
        if self.transport == "peer" and self.world > 1 and x2.shape[0] <= self.local.small_t_max:
            y = self._forward_peer(x2)
            y = y.to(x.dtype) if x.dtype != torch.float32 else y
            return y.reshape(*lead, self.out_features)
        y_loc = self.local(x2).contiguous()
        gathered = torch.empty(self.world * y_loc.numel(), dtype=y_loc.dtype, device=y_loc.device)
        dist.all_gather_into_tensor(gathered, y_loc.view(-1), group=self.group)
        return assemble_gathered(gathered.view(self.world, *y_loc.shape)).reshape(*lead, self.out_features)
