"""Code-domain matmul (E8CodeLinear) against decode-then-float32-matmul of the CPU restatement
of the reference (BASELINE config: weight stored as E8 codes, activations bf16 / float32)."""
import os

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


def make(n_out, n_in, tiling, beta_value=25.0, seed=0):
    torch.manual_seed(seed)
    W = torch.randn(n_out, n_in) * 0.02
    kb = n_in // 8
    if tiling == "block":
        beta = torch.full((n_out * kb,), beta_value) * (0.75 + 0.5 * torch.rand(n_out * kb))
        bpt = 1
    else:
        beta = torch.full((n_out,), beta_value) * (0.75 + 0.5 * torch.rand(n_out))
        bpt = kb
    digits = O.encode(W.numpy().reshape(-1, 8), beta=beta.numpy(), scale_mode=2, blocks_per_tile=bpt, threads=8)
    w_hat = O.decode(digits, beta=beta.numpy(), scale_mode=2, blocks_per_tile=bpt, threads=8).reshape(n_out, n_in)
    return W, beta, bpt, digits, w_hat


@pytest.mark.parametrize("tiling", ["block", "row"])
@pytest.mark.parametrize("T", [1, 3, 16, 40])
def test_small_t_fp32_activations(tiling, T):
    from coset_b200.vlut import E8CodeLinear
    W, beta, bpt, digits, w_hat = make(256, 512, tiling)
    bias = torch.randn(256)
    lin = E8CodeLinear.from_weight(W.cuda(), beta.cuda(), bpt, bias.cuda(), small_t_max=64)  # every T below: code-domain kernels
    assert np.array_equal(lin.codes.cpu().numpy().view(np.uint32).reshape(-1), O.pack_q4(digits))
    assert np.array_equal(lin.dense_weight().cpu().numpy(), w_hat)  # bit-exact dequantised weight
    x = torch.randn(T, 512)
    want = x.double().numpy() @ w_hat.astype(np.float64).T + bias.double().numpy()
    got = lin(x.cuda()).cpu().numpy()
    assert rel(got, want) < 1e-5


@pytest.mark.parametrize("T", [1, 16, 256])
def test_bf16_activations_config_shape(T):
    """BASELINE vLUT config at reduced width for the CPU oracle: beta = 25 (scaled sigma 0.5)."""
    from coset_b200.vlut import E8CodeLinear
    W, beta, bpt, digits, w_hat = make(512, 1024, "block")
    lin = E8CodeLinear.from_weight(W.cuda(), beta.cuda(), bpt)
    x = torch.randn(T, 1024).to(torch.bfloat16)
    want = x.float().numpy() @ w_hat.T
    got = lin(x.cuda()).float().cpu().numpy()
    assert rel(got, want) < 1e-2


def test_literal_scale_gives_zero_output():
    from coset_b200.vlut import E8CodeLinear
    W = torch.randn(64, 128) * 0.02
    beta = torch.full((64 * 16,), 0.021440971642732620)
    lin = E8CodeLinear.from_weight(W.cuda(), beta.cuda(), 1)
    assert not lin.codes.any()
    assert not lin(torch.randn(4, 128, device="cuda")).any()


def test_export_from_trained_layer():
    """Default weight_clip_value (2.0) with N(0, 20) weights: the clamp is active on most weights and the
    exported layer must still compute what the trained layer computes."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    from coset_b200.vlut import E8CodeLinear
    layer = create_e8_hnlq_linear(128, 64, device="cuda", init_kwargs={"std": 20.0})
    lin = E8CodeLinear.from_qat_layer(layer)
    assert lin.weight_clip_value == 2.0
    x = torch.randn(5, 128, device="cuda")
    with torch.no_grad():
        assert rel(lin(x).cpu().numpy(), layer(x).cpu().numpy()) < 1e-5
    with pytest.raises(ValueError):
        E8CodeLinear.from_weight(torch.zeros(4, 12, device="cuda"), torch.ones(4, device="cuda"), 1)


@pytest.mark.parametrize("tiling", ["block", "row"])
def test_weight_clip_in_every_kernel(tiling):
    """clamp(decode / beta, +-clip) with a clip that cuts about a third of the weights, against the CPU
    restatement: few-token kernel (float32 and bf16 activations), library path and both tcgen05 forms."""
    from coset_b200.vlut import E8CodeLinear, e8_decode_gemm, e8_dequant_gemm
    W, beta, bpt, digits, w_hat = make(256, 512, tiling)
    clip = 0.03
    w_clip = np.clip(w_hat, -clip, clip)
    assert 0.1 < (np.abs(w_hat) > clip).mean() < 0.6
    bias = torch.randn(256)
    lin = E8CodeLinear.from_weight(W.cuda(), beta.cuda(), bpt, bias.cuda(), weight_clip_value=clip, small_t_max=64)
    assert np.array_equal(lin.dense_weight().cpu().numpy(), w_clip)
    for T in (1, 3, 16, 40):
        x = torch.randn(T, 512)
        want = x.double().numpy() @ w_clip.astype(np.float64).T + bias.double().numpy()
        assert rel(lin(x.cuda()).cpu().numpy(), want) < 1e-5, T
    xb = torch.randn(300, 512).to(torch.bfloat16)
    want = xb.float().numpy().astype(np.float64) @ w_clip.astype(np.float64).T + bias.double().numpy()
    assert rel(lin(xb.cuda()).float().cpu().numpy(), want) < 1e-2
    got = e8_dequant_gemm(lin.codes, lin.beta, bpt, xb.cuda(), lin.bias, check=True, clip=clip)
    assert rel(got.cpu().numpy(), want) < 1e-2
    got2 = e8_decode_gemm(lin.codes, lin.beta, bpt, xb.cuda(), lin.bias, check=True, clip=clip)
    assert rel(got2.cpu().numpy(), want) < 1e-2


@pytest.mark.parametrize("form", ["fused", "decode_then_pair_gemm"])
@pytest.mark.parametrize("T,n_out,n_in,tiling", [(128, 128, 64, "block"), (256, 256, 512, "block"), (300, 200, 1024, "row"), (1100, 384, 256, "block"),
                                                  (1, 128, 128, "block"), (513, 640, 512, "row")])
def test_tcgen05_dequant_gemm(T, n_out, n_in, tiling, form):
    """Both tensor-core forms (decode fused into the K loop; decode to a transient bf16 buffer followed by the
    cta_group::2 GEMM) against decode-then-float32-matmul of the CPU restatement.  Shapes: ragged token counts,
    feature counts that are not multiples of a tile (200, 384, 640), one K step and sixteen."""
    from coset_b200.vlut import E8CodeLinear, e8_decode_gemm, e8_dequant_gemm
    gemm = e8_dequant_gemm if form == "fused" else e8_decode_gemm
    W, beta, bpt, digits, w_hat = make(n_out, n_in, tiling, seed=T)
    bias = torch.randn(n_out)
    lin = E8CodeLinear.from_weight(W.cuda(), beta.cuda(), bpt, bias.cuda())
    x = torch.randn(T, n_in).to(torch.bfloat16)
    got = gemm(lin.codes, lin.beta, bpt, x.cuda(), lin.bias, check=True).cpu().numpy()
    want = x.float().numpy().astype(np.float64) @ w_hat.astype(np.float64).T + bias.double().numpy()
    assert rel(got, want) < 1e-2
    # against the same product with bf16-rounded weights the kernel should agree to fp32 accumulation error
    w_bf = torch.from_numpy(w_hat).to(torch.bfloat16).double().numpy()
    want_bf = x.double().numpy() @ w_bf.T + bias.double().numpy()
    assert rel(got, want_bf) < 2e-3  # weights may differ from the exactly divided ones by one bf16 ulp
    if form != "fused":  # bf16 result: the same float32 accumulator plus bias, rounded once by the kernel
        got16 = gemm(lin.codes, lin.beta, bpt, x.cuda(), lin.bias, check=True, out_dtype=torch.bfloat16)
        assert got16.dtype == torch.bfloat16
        assert torch.equal(got16.cpu(), torch.from_numpy(got).to(torch.bfloat16))


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,n_out", [(1, 1), (31, 203), (545, 204), (513, 264), (1030, 520)])
def test_pair_gemm_result_rows(T, n_out, out_dtype):
    """Result rows that are made of 16-byte chunks and rows that are not, tails of every tile, with a bias."""
    from coset_b200.vlut import E8CodeLinear, e8_decode_gemm
    W, beta, bpt, _, w_hat = make(n_out, 192, "row")
    bias = torch.randn(n_out)
    lin = E8CodeLinear.from_weight(W.cuda(), beta.cuda(), bpt, bias.cuda())
    x = torch.randn(T, 192).to(torch.bfloat16)
    wb = torch.from_numpy(w_hat).to(torch.bfloat16).double().numpy()
    want = x.double().numpy() @ wb.T + bias.double().numpy()
    got = e8_decode_gemm(lin.codes, lin.beta, bpt, x.cuda(), lin.bias, check=True, out_dtype=out_dtype).double().cpu().numpy()
    # float32 sums of 192 exact products; the bf16 result (8 significant bits) is rounded once, to 2^-8 of itself at most
    assert got.shape == want.shape and rel(got, want) < (1e-5 if out_dtype == torch.float32 else 2.0 ** -8)


@pytest.mark.parametrize("path", ["auto", "tcgen05", "cublas"])
def test_layer_dispatch_for_many_tokens(path):
    """Every large_t_path of E8CodeLinear at token counts on both sides of its thresholds (64 / 1024 / 2048):
    same product within the bf16 tolerance, result in the activations' type; 'tcgen05' keeps no dense copy."""
    from coset_b200.vlut import E8CodeLinear
    W, beta, bpt, digits, w_hat = make(256, 512, "row", seed=5)
    bias = torch.randn(256)
    lin = E8CodeLinear.from_weight(W.cuda(), beta.cuda(), bpt, bias.cuda(), large_t_path=path)
    assert lin.small_t_max == (48 if path == "tcgen05" else 16)
    for T in (16, 17, 48, 49, 65, 300, 1024, 1100, 2048, 2100):
        x = torch.randn(T, 512).to(torch.bfloat16)
        got = lin(x.cuda())
        assert got.dtype == torch.bfloat16 and tuple(got.shape) == (T, 256)
        want = x.float().numpy().astype(np.float64) @ w_hat.astype(np.float64).T + bias.double().numpy()
        assert rel(got.float().cpu().numpy(), want) < 1e-2, (path, T)
    assert (lin._dense is None) == (path == "tcgen05")
    lin.check()  # no bounded wait gave up in any of the tensor-core kernels above
    if path != "cublas":
        lin._status.fill_(1)  # what a kernel whose wait expired leaves behind
        with pytest.raises(RuntimeError):
            lin.check()
        lin.check()  # reported once, then clear
    with pytest.raises(ValueError):
        E8CodeLinear.from_weight(W.cuda(), beta.cuda(), bpt, large_t_path="fastest")


def test_decode_gemm_through_the_c_abi_with_strides_and_without_scales():
    """coset_e8_decode_gemm called as a foreign runtime would: raw pointers, activation rows and result rows
    with padding between them (ldx > n_in, ldy > n_out), no scales (beta = NULL: weights are the plain
    reconstructions), no bias; and the empty shapes return at once."""
    from coset_b200 import _lib
    L = _lib.lib()
    torch.manual_seed(3)
    n_out, n_in, T = 200, 192, 333
    W = torch.randn(n_out, n_in) * 0.6
    digits = O.encode(W.numpy().reshape(-1, 8), threads=8)
    w_hat = O.decode(digits, threads=8).reshape(n_out, n_in)
    codes = torch.from_numpy(O.pack_q4(digits).view(np.int32).reshape(n_out, n_in // 8)).cuda()
    ldx, ldy = n_in + 16, n_out + 5
    xbuf = torch.zeros(T, ldx, dtype=torch.bfloat16, device="cuda")
    x = torch.randn(T, n_in).to(torch.bfloat16)
    xbuf[:, :n_in] = x.cuda()
    ybuf = torch.full((T, ldy), 7.0, dtype=torch.float32, device="cuda")
    scratch = torch.empty(n_out * n_in, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = L.coset_e8_decode_gemm(_lib.ptr(codes), None, 1, n_out, n_in, _lib.ptr(xbuf), ldx, T, None, _lib.ptr(ybuf), _lib.DTYPE_F32, ldy,
                                0.0, _lib.ptr(scratch), scratch.numel() * 2, _lib.ptr(status), _lib.stream())
    assert rc == 0, L.coset_last_error_string()
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    want = x.float().numpy().astype(np.float64) @ w_hat.astype(np.float64).T
    assert rel(ybuf[:, :n_out].cpu().numpy(), want) < 1e-2
    assert bool((ybuf[:, n_out:] == 7.0).all())  # the padding between result rows is untouched
    assert torch.equal(scratch.view(n_out, n_in).float().cpu(), torch.from_numpy(w_hat).to(torch.bfloat16).float())  # exact: halves of small integers
    for shape in ((0, n_in, T), (n_out, n_in, 0)):
        assert L.coset_e8_decode_gemm(_lib.ptr(codes), None, 1, shape[0], shape[1], _lib.ptr(xbuf), ldx, shape[2], None, _lib.ptr(ybuf),
                                      _lib.DTYPE_F32, ldy, 0.0, _lib.ptr(scratch), scratch.numel() * 2, None, _lib.stream()) == 0
    # refused: scratch too small, n_in not a multiple of 64, unknown result type
    assert L.coset_e8_decode_gemm(_lib.ptr(codes), None, 1, n_out, n_in, _lib.ptr(xbuf), ldx, T, None, _lib.ptr(ybuf), _lib.DTYPE_F32, ldy,
                                  0.0, _lib.ptr(scratch), 16, None, _lib.stream()) < 0
    assert L.coset_e8_decode_gemm(_lib.ptr(codes), None, 1, n_out, 100, _lib.ptr(xbuf), ldx, T, None, _lib.ptr(ybuf), _lib.DTYPE_F32, ldy,
                                  0.0, _lib.ptr(scratch), scratch.numel() * 2, None, _lib.stream()) < 0
    assert L.coset_e8_decode_gemm(_lib.ptr(codes), None, 1, n_out, n_in, _lib.ptr(xbuf), ldx, T, None, _lib.ptr(ybuf), 9, ldy,
                                  0.0, _lib.ptr(scratch), scratch.numel() * 2, None, _lib.stream()) < 0


def test_decode_gemm_scratch_is_checked_and_reusable():
    """The transient weight buffer: refused when too small or of the wrong type; one buffer serves layers of
    different shapes one after the other (nothing in it survives a call)."""
    from coset_b200.vlut import E8CodeLinear, e8_decode_gemm
    scratch = torch.empty(512 * 256, dtype=torch.bfloat16, device="cuda")
    for n_out, n_in in ((512, 256), (128, 192), (256, 512)):
        W, beta, bpt, digits, w_hat = make(n_out, n_in, "block", seed=n_out)
        lin = E8CodeLinear.from_weight(W.cuda(), beta.cuda(), bpt)
        x = torch.randn(70, n_in).to(torch.bfloat16)
        got = e8_decode_gemm(lin.codes, lin.beta, bpt, x.cuda(), None, check=True, scratch=scratch).cpu().numpy()
        assert rel(got, x.float().numpy().astype(np.float64) @ w_hat.astype(np.float64).T) < 1e-2
    with pytest.raises(ValueError):
        e8_decode_gemm(lin.codes, lin.beta, bpt, x.cuda(), None, scratch=scratch[:100])
    with pytest.raises(ValueError):
        e8_decode_gemm(lin.codes, lin.beta, bpt, x.cuda(), None, scratch=scratch.float())
    from coset_b200 import _lib
    assert _lib.lib().coset_e8_decode_gemm_scratch_bytes(256, 512) == 256 * 512 * 2


SHARD_WORKER = r'''
import os, sys
import torch
import torch.distributed as dist
sys.path.insert(0, sys.argv[1])
from coset_b200.vlut import ColumnParallelE8CodeLinear, E8CodeLinear
rank = int(os.environ["RANK"]); local = int(os.environ["LOCAL_RANK"])
torch.cuda.set_device(local)
dist.init_process_group("nccl", device_id=torch.device("cuda", local))
torch.manual_seed(3)
n_out, n_in = 256, 512
W = (torch.randn(n_out, n_in) * 0.02).cuda()
for bpt, nbeta in ((1, n_out * n_in // 8), (n_in // 8, n_out)):
    beta = (20.0 + 10.0 * torch.rand(nbeta)).cuda()
    bias = torch.randn(n_out).cuda()
    full = E8CodeLinear.from_weight(W, beta, bpt, bias)
    shard = ColumnParallelE8CodeLinear.from_weight(W, beta, bpt, bias)
    peer = ColumnParallelE8CodeLinear.from_weight(W, beta, bpt, bias, transport="peer")
    for T in (1, 5, 200):
        x = torch.randn(T, n_in).cuda()
        assert torch.equal(shard(x), full(x)), (bpt, T)
        for _ in range(3):  # several calls: both halves of the result buffer are reused
            assert torch.equal(peer(x), full(x)), ("peer", bpt, T)
torch.cuda.synchronize()
if rank == 0:
    print("SHARD_OK")
dist.destroy_process_group()
'''


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs 2 GPUs")
def test_two_gpu_column_parallel_equals_unsharded(tmp_path):
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    script = tmp_path / "shard_worker.py"
    script.write_text(SHARD_WORKER)
    env = dict(os.environ, NCCL_NVLS_ENABLE="0")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node=2", "--master-addr", "127.0.0.1",
           "--master-port", "29621", str(script), root]
    res = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    assert "SHARD_OK" in res.stdout


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bpt_of", [lambda kb: kb, lambda kb: 1, lambda kb: 3, lambda kb: 2 * kb], ids=["row", "block", "three_blocks", "two_rows"])
@pytest.mark.parametrize("n_out,n_in", [(1, 8), (17, 72), (200, 1032), (16, 4096), (1200, 2048)])
@pytest.mark.parametrize("T,clip", [(1, 0.0), (8, 0.05), (9, 4.0), (17, 0.0)])
def test_few_token_product_edges(n_out, n_in, bpt_of, T, clip, dtype):
    """The layer's few-token product: ragged rows, K that is no multiple of a unit, scale tiles that straddle rows, both
    token tiles and the remainder, a clamp that binds on some weights and one that cannot, any code word and non-zero top
    levels.  The weights are exact in the kernel and the sums are float32, for bf16 activations too, so 1e-5 holds for both."""
    from coset_b200 import _lib
    from coset_b200.core.e8 import e8_decode_packed, e8_encode_packed
    from coset_b200.vlut import E8CodeLinear
    g = torch.Generator(device="cuda").manual_seed(n_out + T)
    kb = n_in // 8
    bpt = bpt_of(kb)
    n = n_out * kb
    beta = 25.0 * (0.75 + 0.5 * torch.rand((n + bpt - 1) // bpt, device="cuda", generator=g))
    codes = e8_encode_packed(torch.randn(n, 8, device="cuda", generator=g) * 0.6).view(torch.int32).view(-1)
    word = torch.randint(0, 1 << 32, (n,), device="cuda", generator=g)
    hit = torch.randint(0, 100, (n,), device="cuda", generator=g)
    word = torch.where(hit == 0, word, word & 0xffff)
    codes = torch.where(hit < 20, (word - ((word >> 31) << 32)).to(torch.int32), codes)
    w = e8_decode_packed(codes, scale=beta, scale_mode=_lib.SCALE_MUL_TILE, blocks_per_tile=bpt).view(n_out, n_in)
    w = w.clamp(-clip, clip) if clip else w
    bias = torch.randn(n_out, device="cuda", generator=g)
    x = torch.randn(T, n_in, device="cuda", generator=g).to(dtype)
    want = (x.double() @ w.double().T + bias.double()).cpu().numpy()
    lin = E8CodeLinear(codes.view(n_out, kb), beta, bpt, bias, small_t_max=64, weight_clip_value=clip)
    product = lambda l, code: _lib.native().vlut_product(x, l._product_layout(), l.out_features, n_in, l.beta, bpt, l.bias, clip, code)
    got = product(lin, _lib.DTYPE_F32)
    assert rel(got.cpu().numpy(), want) < 1e-5
    assert torch.equal(product(lin, _lib.DTYPE_BF16), got.to(torch.bfloat16))
    assert torch.equal(lin(x), got.to(dtype))
    if bpt <= kb and n_out > 1 and bpt != 3:  # a shard of the rows returns the same bits
        half = n_out // 2
        part = E8CodeLinear(lin.codes[:half], beta[:half * (kb // bpt)], bpt, bias[:half], small_t_max=64, weight_clip_value=clip)
        assert torch.equal(product(part, _lib.DTYPE_F32), got[:, :half])


def _kept_copy_layer(n_out=64, n_in=256, seed=5, **kw):
    from coset_b200.vlut import E8CodeLinear
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(n_out, n_in, device="cuda", generator=g) * 0.05
    return E8CodeLinear.from_weight(w, torch.full((n_out,), 25.0, device="cuda"), n_in // 8, **kw), torch.randn(3, n_in, device="cuda", generator=g)


def test_few_tokens_under_capture_read_the_codes_of_the_replay():
    """A graph captured before any eager call keeps nothing that only its replay would compute, and its replay follows
    codes that were written after the capture."""
    lin, x = _kept_copy_layer()
    other, _ = _kept_copy_layer(seed=6)
    want = x.double() @ lin.dense_weight().double().T
    want_other = x.double() @ other.dense_weight().double().T
    other(x)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        y = lin(x)
    torch.cuda.synchronize()
    assert rel(lin(x).cpu().numpy(), want.cpu().numpy()) < 1e-5
    graph.replay()
    assert rel(y.cpu().numpy(), want.cpu().numpy()) < 1e-5
    lin.codes.copy_(other.codes)
    graph.replay()
    assert rel(y.cpu().numpy(), want_other.cpu().numpy()) < 1e-5
    assert rel(lin(x).cpu().numpy(), want_other.cpu().numpy()) < 1e-5


def test_kept_copies_follow_the_buffers():
    """In-place writes, replaced buffers, copies of the layer and buffers without a version counter."""
    import copy
    import pickle
    a, x = _kept_copy_layer()
    b, _ = _kept_copy_layer(seed=6)
    ya, yb = a(x), b(x)
    assert not torch.equal(ya, yb)
    for twin in (copy.deepcopy(a), pickle.loads(pickle.dumps(a))):
        assert torch.equal(twin(x), ya)
        twin.codes.copy_(b.codes)
        assert torch.equal(twin(x), yb)
    old = copy.deepcopy(a)
    del old.__dict__["_kept"]  # a module pickled before it kept copies this way
    assert torch.equal(pickle.loads(pickle.dumps(old))(x), ya)
    a.codes = b.codes.clone()
    assert torch.equal(a(x), yb)
    with torch.inference_mode():
        c, _ = _kept_copy_layer()
        yc = c(x)
        assert rel(yc.cpu().numpy(), ya.cpu().numpy()) < 1e-5
        c.codes.copy_(b.codes)
        assert rel(c(x).cpu().numpy(), yb.cpu().numpy()) < 1e-5


def test_kept_copy_is_complete_for_every_stream():
    """The first call lays the weight out on its own stream; a call on another stream right after reads it complete."""
    streams = [torch.cuda.Stream() for _ in range(2)]
    for seed in range(8):
        lin, x = _kept_copy_layer(2048, 2048, seed)
        torch.cuda.synchronize()
        ys = []
        for s in streams:
            with torch.cuda.stream(s):
                ys.append(lin(x))
        torch.cuda.synchronize()
        assert torch.equal(ys[0], ys[1])


def test_few_tokens_refuse_other_types_at_any_count():
    lin, x = _kept_copy_layer()
    for T in (0, 3):
        with pytest.raises(TypeError):
            lin(x[:T].half())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n_out,n_in", [(1, 8), (17, 72), (200, 1032), (64, 4096)])
@pytest.mark.parametrize("T,clip,row", [(1, 0.0, True), (3, 0.05, False), (16, 0.05, True)])
def test_few_tokens_follow_writes_that_no_version_shows(n_out, n_in, T, clip, row, dtype):
    """All codes, one code and the last code written through `.data`, the codes written by a replayed graph and by the encoder's
    `out`: the product is that of the codes, to the bit that a fresh layer returns, and of the old codes once they are back."""
    from coset_b200 import _lib
    from coset_b200.core.e8 import e8_encode_packed
    from coset_b200.vlut import E8CodeLinear
    g = torch.Generator(device="cuda").manual_seed(n_out + T)
    kb = n_in // 8
    bpt = kb if row else 1
    beta = 25.0 * (0.75 + 0.5 * torch.rand(n_out * kb // bpt, device="cuda", generator=g))
    weights = [torch.randn(n_out * kb, 8, device="cuda", generator=g) * s for s in (0.02, 0.03)]
    encode = lambda w, **kw: e8_encode_packed(w, scale=beta, scale_mode=_lib.SCALE_MUL_TILE, blocks_per_tile=bpt, **kw)
    old, new = (encode(w).view(torch.int32).view(n_out, kb) for w in weights)
    x = torch.randn(T, n_in, device="cuda", generator=g).to(dtype)
    fresh = lambda codes: E8CodeLinear(codes.clone(), beta, bpt, None, weight_clip_value=clip)(x)
    layer = E8CodeLinear(old.clone(), beta, bpt, None, weight_clip_value=clip)
    assert torch.equal(layer(x), fresh(old))
    version = layer.codes._version
    for what in ("all", "one", "last"):
        codes = old.clone()
        if what == "all":
            codes.copy_(new)
        else:
            at = (n_out // 2, kb // 2) if what == "one" else (n_out - 1, kb - 1)
            codes[at] = codes[at] ^ 0x1234
        layer.codes.data.copy_(codes)
        assert layer.codes._version == version
        assert torch.equal(layer(x), fresh(codes)), what
    layer.codes.data.copy_(old)
    assert torch.equal(layer(x), fresh(old))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer.codes.copy_(new)
    assert torch.equal(layer(x), fresh(old))
    graph.replay()
    assert torch.equal(layer(x), fresh(new))
    encode(weights[0], out=layer.codes)
    assert torch.equal(layer(x), fresh(old))


@pytest.mark.parametrize("n_out,n_in,T", [(17, 72, 1), (64, 4096, 3), (16, 8192, 16)])
def test_few_tokens_read_the_layout_while_the_codes_are_those_it_was_made_from(n_out, n_in, T):
    """A layout whose bytes are zeroed behind the layer's back (its hash is not) gives a product of zeros: the units are taken from
    the layout and not made anew."""
    layer, _ = _kept_copy_layer(n_out, n_in)
    x = torch.randn(T, n_in, device="cuda").to(torch.bfloat16)
    assert bool((layer(x) != 0).any())
    layer._product_layout()[:((n_out + 15) // 16) * ((n_in + 63) // 64) * 1024] = 64
    assert not bool((layer(x) != 0).any())


@pytest.mark.parametrize("row,clip", [(True, 0.0), (True, 0.05), (False, 0.0), (False, 0.05)])
@pytest.mark.parametrize("T,n_out,n_in", [(1, 320, 64), (8, 384, 256), (16, 320, 7424)])
def test_few_float32_tokens_keep_float32_precision(T, n_out, n_in, row, clip):
    """The root mean square of the error against 64 bits stays below 2^-23 of the results' at any K: two roundings of the scales
    (reciprocal, product) and one of the result at 2^-24 at most each, and sums whose own error does not grow with K."""
    from coset_b200.core.e8 import e8_decode_packed
    layer, _ = _kept_copy_layer(n_out, n_in, seed=n_in)
    if not row:
        from coset_b200.vlut import E8CodeLinear
        g = torch.Generator(device="cuda").manual_seed(T)
        beta = 25.0 * (0.8 + 0.4 * torch.rand(n_out * n_in // 8, device="cuda", generator=g))
        layer = E8CodeLinear(layer.codes, beta, 1, None)
    layer.weight_clip_value = clip
    x = torch.randn(T, n_in, device="cuda", generator=torch.Generator(device="cuda").manual_seed(T))
    w = e8_decode_packed(layer.codes.view(-1)).double().view(layer.beta.numel(), -1) / layer.beta.double().view(-1, 1)
    w = w.view(n_out, n_in).clamp(-clip, clip) if clip else w.view(n_out, n_in)
    want = x.double() @ w.T
    assert float((layer(x).double() - want).norm() / want.norm()) < 2.0 ** -23


def _awkward(kind, T, n_in):
    x = torch.randn(T, n_in, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7))
    if kind == "infinity":
        x[0, 3], x[T - 1, n_in - 1] = float("inf"), float("-inf")
    elif kind == "nan":
        x[T // 2, 5] = float("nan")
    elif kind == "large":
        x = x.clamp(-3, 3) * 3e36
    return x


@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 1e-2), (torch.float32, 1e-5)])
@pytest.mark.parametrize("row", [True, False])
@pytest.mark.parametrize("clip", [0.0, 0.05, 2.0, float("inf")])
@pytest.mark.parametrize("kind", ["plain", "infinity", "nan", "large"])
@pytest.mark.parametrize("T,n_in", [(1, 256), (3, 1032), (16, 4096)])
def test_few_tokens_with_awkward_values(T, n_in, kind, clip, row, dtype, tol):
    """Infinities, NaN, activations whose unscaled sums overflow and an infinite clamp, against the sum in 64 bits: the same
    results are finite, infinite and NaN, from the layout and from the codes."""
    from coset_b200 import _lib
    from coset_b200.vlut import E8CodeLinear
    layer, _ = _kept_copy_layer(40, n_in)
    bpt = n_in // 8 if row else 1
    layer = E8CodeLinear(layer.codes, torch.full((40 * n_in // 8 // bpt,), 25.0, device="cuda"), bpt, torch.randn(40, device="cuda"), weight_clip_value=clip)
    x = _awkward(kind, T, n_in).to(dtype)
    w = layer.dense_weight().double()
    want = (x.double().unsqueeze(1) * w).sum(2) + layer.bias.double()  # not matmul: 0 * inf must count
    trusted = _lib.native().vlut_product(x, layer._product_layout(), 40, n_in, layer.beta, bpt, layer.bias, clip, _lib.DTYPE_F32)
    for got in (layer(x).double(), trusted.double()):
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
        assert torch.equal(got[got.isinf()], want[want.isinf()])
        assert rel(got[got.isfinite()].cpu().numpy(), want[want.isfinite()].cpu().numpy()) < tol


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("row", [True, False])
@pytest.mark.parametrize("scale", [0.0, 1e-39, float("inf"), float("nan")])
def test_few_tokens_with_awkward_scales_and_a_clamp(scale, row, dtype):
    """A scale of zero or NaN: the weights are the clamped values that a minimum and a maximum make of them, as in the kernels
    that read the codes."""
    from coset_b200.vlut import E8CodeLinear, e8_vlut_matmul
    layer, _ = _kept_copy_layer(40, 256)
    bpt = 32 if row else 1
    beta = torch.full((40 * 32 // bpt,), 25.0, device="cuda")
    beta[::3] = scale
    layer = E8CodeLinear(layer.codes, beta, bpt, None, weight_clip_value=0.5)
    x = torch.randn(2, 256, device="cuda").to(dtype)
    want = e8_vlut_matmul(layer.codes, beta, bpt, x, None, 0.5, dtype)
    assert bool(want.isfinite().all())
    torch.testing.assert_close(layer(x), want, rtol=1e-2 if dtype == torch.bfloat16 else 1e-5, atol=1e-4)


@pytest.mark.parametrize("rows", [64, 1 << 20, 1 << 31, 1 << 32, (1 << 32) + 1])
def test_one_scale_for_more_rows_than_there_are(rows):
    """A scale tile may be larger than the weight, by any factor: the kernel's row count per scale is no wider than an int."""
    from coset_b200.vlut import E8CodeLinear
    layer, x = _kept_copy_layer(64, 256)
    want = x.double() @ layer.dense_weight().double().T
    got = E8CodeLinear(layer.codes, torch.full((1,), 25.0, device="cuda"), rows * 32, None)(x)
    assert rel(got.cpu().numpy(), want.cpu().numpy()) < 1e-5


@pytest.mark.parametrize("clip", [0.0, 0.05])
@pytest.mark.parametrize("T", [3, 64])
def test_capture_after_an_eager_call_follows_every_buffer(T, clip):
    """An eager call first, as a warm-up does, then a capture: its replay follows in-place writes to codes, scales and bias, before
    and after an eager call has replaced the copies that the layer keeps."""
    import gc
    layer, _ = _kept_copy_layer(64, 256, weight_clip_value=clip)
    layer.bias = torch.randn(64, device="cuda")
    other, _ = _kept_copy_layer(64, 256, seed=6)
    x = torch.randn(T, 256, device="cuda").to(torch.bfloat16)
    want = lambda: x.double() @ layer.dense_weight().double().T + layer.bias.double()
    layer(x)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        y = layer(x)
    same = lambda got: rel(got.float().cpu().numpy(), want().cpu().numpy()) < 1e-2
    for write in (lambda: None, lambda: layer.bias.add_(3.0), lambda: layer.bias.data.mul_(-2.0), lambda: layer.codes.copy_(other.codes), lambda: layer.beta.mul_(0.5)):
        write()
        graph.replay()
        assert same(y)
        assert same(layer(x))
        gc.collect()
        filler = [torch.full((1 << 16,), 3e38, device="cuda") for _ in range(64)]  # into whatever the eager call gave back
        graph.replay()
        assert same(y)
        del filler


@pytest.mark.parametrize("T", [3, 64])
def test_kept_copies_do_not_outlive_a_move_and_can_be_dropped(T):
    layer, _ = _kept_copy_layer(64, 256)
    x = torch.randn(T, 256, device="cuda").to(torch.bfloat16)
    y = layer(x)
    assert layer._kept
    layer.cpu()
    assert not layer._kept
    layer.cuda()
    assert torch.equal(layer(x), y)
    other, _ = _kept_copy_layer(64, 256, seed=6)
    layer.codes.data.copy_(other.codes)
    layer.forget_copies()
    assert torch.equal(layer(x), other(x))


def test_kept_copy_replaced_while_another_stream_reads_it():
    """A copy that another stream still reads is not given back to the allocator when a write replaces it."""
    side = torch.cuda.Stream()
    layer, _ = _kept_copy_layer(2048, 2048)
    x = torch.randn(64, 2048, device="cuda").to(torch.bfloat16)
    other, _ = _kept_copy_layer(2048, 2048, seed=6)
    want = layer(x)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        y = layer(x)
    layer.codes = other.codes
    layer(x)
    filler = [torch.full((2048, 2048), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    del filler


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", ["rows", "three", "four", "transposed", "strided", "expanded"])
def test_library_path_rounds_once_for_every_shape(shape, dtype):
    """The tokens of the library path, given in any number of dimensions and any strides, are those of the plain rows, to the bit."""
    layer, _ = _kept_copy_layer(64, 256)
    layer.bias = torch.randn(64, device="cuda") * 10
    x = torch.randn(12, 16, 256, device="cuda").to(dtype)
    want = layer(x.view(192, 256)).view(12, 16, 64)
    if shape == "rows":
        got = layer(torch.cat([x, x], 2).view(192, 512)[:, :256]).view(12, 16, 64)
    elif shape == "three":
        got = layer(x)
    elif shape == "four":
        got = layer(x.view(4, 3, 16, 256)).view(12, 16, 64)
    elif shape == "transposed":
        got = layer(x.transpose(0, 1).contiguous().transpose(0, 1))
    elif shape == "strided":
        got = layer(torch.cat([x, x], 2)[..., :256])
    else:
        got, want = layer(x[:1].expand(12, 16, 256)), want[:1].expand(12, 16, 64)
    assert got.shape == want.shape and torch.equal(got, want)


@pytest.mark.parametrize("n_out,n_in,row,T,dtype,codes", [
    (512, 8192, False, 1, torch.float32, True), (512, 8192, False, 2, torch.float32, True), (512, 8192, False, 3, torch.float32, False),
    (512, 8184, False, 1, torch.float32, False), (1024, 4096, True, 1, torch.float32, True), (1032, 4096, True, 1, torch.float32, False),
    (4104, 1024, False, 1, torch.float32, True), (4104, 1024, False, 2, torch.float32, False), (4608, 1016, False, 1, torch.float32, False),
    (1024, 4096, False, 1, torch.bfloat16, False)])
def test_one_or_two_float32_tokens_read_the_codes(n_out, n_in, row, T, dtype, codes):
    """The line between the two kernels, a shard that keeps to the rule of the whole weight, and the same result from both."""
    from coset_b200 import _lib
    from coset_b200.vlut import E8CodeLinear, e8_vlut_matmul
    layer, _ = _kept_copy_layer(n_out, n_in)
    bpt = n_in // 8 if row else 1
    beta = torch.full((n_out * n_in // 8 // bpt,), 25.0, device="cuda")
    layer = E8CodeLinear(layer.codes, beta, bpt, None)
    x = torch.randn(T, n_in, device="cuda").to(dtype)
    from_codes = e8_vlut_matmul(layer.codes, beta, bpt, x, None, 0.0, dtype)
    from_layout = _lib.native().vlut_product(x, layer._product_layout(), n_out, n_in, beta, bpt, None, 0.0, _lib.DTYPE_BF16 if dtype == torch.bfloat16 else _lib.DTYPE_F32)
    assert torch.equal(layer(x), from_codes if codes else from_layout)
    assert rel(from_layout.float().cpu().numpy(), from_codes.float().cpu().numpy()) < (1e-2 if dtype == torch.bfloat16 else 1e-6)
    shard = E8CodeLinear(layer.codes[:n_out // 2], beta[:beta.numel() // 2], bpt, None)
    shard._rows = n_out
    assert torch.equal(shard(x), layer(x)[:, :n_out // 2])


@pytest.mark.parametrize("bias_dtype", [torch.float32, torch.bfloat16, torch.float64])
def test_library_path_with_biases_of_other_types_and_gradients(bias_dtype):
    """The bias is rounded to bf16 in the call, whatever it is; the product stays differentiable in the activations, under vmap too."""
    layer, _ = _kept_copy_layer(64, 256)
    x = torch.randn(32, 256, device="cuda").to(torch.bfloat16).requires_grad_()
    layer.bias = torch.randn(128, device="cuda").to(bias_dtype)[::2]
    dense, doubled = layer.dense_weight(torch.bfloat16), x.detach().view(2, 32, 128).repeat(1, 1, 2)
    for bias in (layer.bias, layer.bias.contiguous()):
        layer.bias = bias
        plain = lambda v: torch.nn.functional.linear(v, dense, bias.to(torch.bfloat16))
        y, want = layer(x), plain(x)
        assert torch.equal(y, want)
        assert torch.equal(torch.autograd.grad(y.float().sum(), x)[0], torch.autograd.grad(want.float().sum(), x)[0])
        assert torch.equal(torch.vmap(layer)(doubled), torch.vmap(plain)(doubled))


@pytest.mark.parametrize("clip", [0.05, 0.02, 0.0625, 1e-3, 2.0, float("inf")])
def test_dense_bf16_weight_is_the_rounded_clamp(clip):
    layer, _ = _kept_copy_layer(64, 4096, weight_clip_value=clip)
    beta = layer.beta.clone()
    layer.beta.copy_(beta * (0.5 + torch.rand_like(beta)))
    assert torch.equal(layer.dense_weight(torch.bfloat16), layer.dense_weight(torch.float32).to(torch.bfloat16))


@pytest.mark.parametrize("T,n_out,n_in", [(1, 1, 8), (17, 64, 8), (32, 256, 64), (33, 257, 72), (64, 4096, 128), (65, 264, 4104), (130, 136, 8192),
                                          (257, 1000, 520), (300, 768, 3072), (600, 99, 192), (1030, 3080, 136)])
@pytest.mark.parametrize("form", ["rows", "padded", "offset"])
def test_product_with_the_kept_dense_weight(T, n_out, n_in, form):
    """Every tile's edges, one to four pairs over K, ragged K, result rows with and without 16-byte chunks; tokens in rows, in padded
    rows and at an address that is no multiple of 16."""
    from coset_b200 import _lib
    x = torch.randn(T, n_in, device="cuda").bfloat16()
    w = (torch.randn(n_out, n_in, device="cuda") * 0.02).bfloat16()
    bias = torch.randn(n_out, device="cuda")
    if form == "padded":
        x = torch.cat([x, torch.full((T, 16), float("nan"), device="cuda", dtype=torch.bfloat16)], 1)[:, :n_in]
    elif form == "offset":
        x = torch.cat([torch.zeros(1, device="cuda", dtype=torch.bfloat16), x.reshape(-1)])[1:].view(T, n_in)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for b in (bias, None):
        got = _lib.native().dense_linear(x, w, b, status, True)
        want = x.double() @ w.double().T + (b.double() if b is not None else 0.0)
        # one rounding to 8 significant bits, and float32 sums of K exact products and the bias, each of which may round or truncate
        # its part of a sum that is no larger than the sum of the magnitudes
        bound = 2.0 ** -8 * want.abs() + 2.0 ** -22 * (x.double().abs() @ w.double().abs().T + (b.abs().double() if b is not None else 0.0))
        assert got.dtype == torch.bfloat16 and bool(((got.double() - want).abs() <= bound).all())
    assert int(status.item()) == 0


def test_product_with_the_kept_dense_weight_refuses():
    from coset_b200 import _lib
    L = _lib.lib()
    w, x, y = (torch.zeros(64, 64, dtype=torch.bfloat16, device="cuda") for _ in range(3))
    call = lambda n_out=64, n_in=64, ldx=64, T=64, ldy=64, wp=w.data_ptr(), xp=x.data_ptr(): L.coset_e8_dense_linear(
        wp, n_out, n_in, xp, ldx, T, None, 0, y.data_ptr(), ldy, None, _lib.stream())
    assert call() == 0 and call(T=0) == 0 and call(n_out=0) == 0
    for bad in (dict(n_in=60), dict(n_in=0), dict(ldx=56), dict(ldx=68), dict(ldy=63), dict(wp=None), dict(xp=None), dict(wp=w.data_ptr() + 2), dict(xp=x.data_ptr() + 8), dict(T=-1)):
        assert call(**bad) < 0, bad


@pytest.mark.parametrize("how", ["autograd", "tangent", "autocast", "vmap", "mode"])
def test_product_with_the_kept_dense_weight_is_torchs_for_who_looks_at_it(how):
    from torch.utils._python_dispatch import TorchDispatchMode
    layer, _ = _kept_copy_layer(64, 256)
    layer.bias = torch.randn(64, device="cuda")
    x = torch.randn(32, 256, device="cuda").bfloat16()
    w = layer.dense_weight(torch.bfloat16)
    if how == "autograd":
        x.requires_grad_()
        layer(x).sum().backward()
        assert torch.allclose(x.grad.float(), w.float().sum(0).expand(32, 256), rtol=2.0 ** -6, atol=1e-3)
    elif how == "tangent":
        with torch.autograd.forward_ad.dual_level():
            t = torch.autograd.forward_ad.unpack_dual(layer(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)))).tangent
            assert t is not None and torch.allclose(t.float(), w.float().sum(1).expand(32, 64), rtol=2.0 ** -6, atol=1e-3)
    elif how == "autocast":
        with torch.autocast("cuda", dtype=torch.float16):
            assert layer(x).dtype == torch.float16
    elif how == "vmap":
        batch = torch.randn(3, 32, 256, device="cuda").bfloat16()
        got = torch.func.vmap(layer)(batch)
        assert torch.allclose(got.float(), torch.stack([layer(b) for b in batch]).float(), rtol=2.0 ** -6, atol=2.0 ** -6)
    else:
        class Seen(TorchDispatchMode):
            calls = []

            def __torch_dispatch__(self, func, types, args=(), kwargs=None):
                self.calls.append(str(func))
                return func(*args, **(kwargs or {}))
        layer(x)
        with Seen() as seen:
            layer(x)
        assert any("mm" in c or "linear" in c for c in seen.calls)


def test_products_of_different_plans_from_several_threads():
    """The plans of these calls ask for different amounts of shared memory of the same kernels: no thread's call is refused for another's, and each has
    the bits it has alone."""
    import threading
    from coset_b200 import _lib
    calls = []
    for T, n_out, n_in in ((32, 64, 64), (64, 4096, 4096), (256, 512, 256), (512, 1024, 1024)):
        x, w = torch.randn(T, n_in, device="cuda").bfloat16(), torch.randn(n_out, n_in, device="cuda").bfloat16()
        calls.append((x, w, _lib.native().dense_linear(x, w, None, None, True)))
    torch.cuda.synchronize()
    start, failures = threading.Barrier(len(calls)), []

    def work(x, w, want):
        try:
            start.wait()
            for _ in range(1500):
                got = _lib.native().dense_linear(x, w, None, None, True)
            assert torch.equal(got, want)
        except Exception as e:  # noqa: BLE001 - reported by the test's own thread
            failures.append(repr(e))
    threads = [threading.Thread(target=work, args=c) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


@pytest.mark.parametrize("tokens,split", [(32, 4), (64, 2), (128, 1), (256, 4), (224, 2)])
def test_a_wait_that_gave_up_leaves_no_number(tokens, split):
    """Each pair in turn takes its wait for run out: the results of every tile it has a part in are not a number, the status says so, and the
    next call is as good as any."""
    from coset_b200 import _lib
    T, n_out, n_in = tokens + 5, 264, 520
    x, w = torch.randn(T, n_in, device="cuda").bfloat16(), torch.randn(n_out, n_in, device="cuda").bfloat16()
    want = x.double() @ w.double().T
    bound = 2.0 ** -8 * want.abs() + 2.0 ** -22 * (x.double().abs() @ w.double().abs().T)
    for late in (-1, *range(split), -1):
        y, status = torch.zeros(T, n_out, device="cuda", dtype=torch.bfloat16), torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.check(_lib.lib().coset_e8_dense_linear_late(_lib.ptr(w), n_out, n_in, _lib.ptr(x), T, _lib.ptr(y), tokens, split, late, _lib.ptr(status), _lib.stream()), "late")
        if late < 0:
            assert bool(((y.double() - want).abs() <= bound).all()) and int(status.item()) == 0
        else:
            assert bool(y.isnan().all()) and int(status.item()) == 1


@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("how", ["captured", "long"])
def test_kept_dense_weight_is_torchs_where_that_is_quicker(how, bias):
    """In a graph, for a weight whose own product is the slower one, and for rows so long that few CTAs would sum over each: torch's bits."""
    n_out, n_in = (256, 4096) if how == "captured" else (64, (1 << 15) + 8)
    layer, _ = _kept_copy_layer(n_out, n_in)
    layer.bias = torch.randn(n_out, device="cuda") if bias else None
    x = torch.randn(64, n_in, device="cuda").bfloat16()
    want = torch.nn.functional.linear(x, layer.dense_weight(torch.bfloat16), layer.bias.bfloat16() if bias else None)
    if how == "long":
        assert torch.equal(layer(x), want)
        return
    layer(x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = layer(x)
    graph.replay()
    assert torch.equal(y, want)
