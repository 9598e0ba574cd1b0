"""HNLQLinearQAT on the GPU against golden outputs of the reference layer (row tiling) and of
the function-assembled expectation for block tiling (the reference layer raises there)."""
import numpy as np
import pytest
import torch

from conftest import bits

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


def make_layer(g, tag, tiling="row"):
    from coset_b200.core.e8 import create_e8_hnlq_linear
    W = g[f"{tag}_W"]
    o, i = W.shape
    layer = create_e8_hnlq_linear(i, o, q=4, M=2, tiling=tiling, device="cuda")
    with torch.no_grad():
        layer.weight.copy_(dev(W))
        layer.bias.copy_(dev(g[f"{tag}_bias"]))
        if tiling == "row":
            layer.theta_beta.copy_(dev(g[f"{tag}_theta"]))
            layer.sigma_ema.copy_(dev(g[f"{tag}_sigma"]))
            layer.xmax_ema.copy_(dev(g[f"{tag}_xmax"]))
    return layer


@pytest.mark.parametrize("tag", ["small", "big", "mid"])
def test_fake_quant_kernel_bit_exact(golden_layer, tag):
    from coset_b200.core.layers import e8_fake_quantize
    g = golden_layer
    W = dev(g[f"{tag}_W"])
    o, i = W.shape
    wq = e8_fake_quantize(W, dev(g[f"{tag}_beta"]), i // 8, 4, 2.0)
    assert np.array_equal(bits(wq.cpu().numpy()), bits(g[f"{tag}_Wq"]))
    wqb = e8_fake_quantize(W, dev(g[f"{tag}_blk_beta"]).reshape(-1), 1, 4, 2.0)
    assert np.array_equal(bits(wqb.cpu().numpy()), bits(g[f"{tag}_blk_Wq"]))


@pytest.mark.parametrize("tag", ["small", "big", "mid"])
def test_block_tiling_gradients(golden_layer, tag):
    from coset_b200.core.layers import e8_fake_quantize
    g = golden_layer
    W = dev(g[f"{tag}_W"]).requires_grad_(True)
    o, i = W.shape
    beta = dev(g[f"{tag}_blk_beta"]).reshape(-1).requires_grad_(True)
    wq = e8_fake_quantize(W, beta, 1, 4, 2.0)
    y = torch.nn.functional.linear(dev(g[f"{tag}_x"]), wq, dev(g[f"{tag}_bias"]))
    ((y - dev(g[f"{tag}_t"])) ** 2).mean().backward()
    assert rel(W.grad.cpu().numpy(), g[f"{tag}_blk_dW"]) < 1e-5
    want = g[f"{tag}_blk_dbeta"].reshape(-1)
    assert np.abs(beta.grad.cpu().numpy() - want).max() <= 1e-5 * max(np.abs(want).max(), 1e-12) + 1e-12


def expected_from_oracle(W, beta, theta, bmin, bmax, bias, x, t, blocks_per_tile, clip=2.0):
    """Forward and backward of the reference graph clamp(ste(e8_quantize(W beta)) / beta) evaluated on
    the CPU in float64 around the oracle's quantised weights (coset/core/layers.py:415-470, 472-484):
    the straight-through estimator passes dWq where the clamp is inactive, dbeta collects
    dWq * (W - Wq_unclipped) / beta per tile and dtheta = dbeta * sigmoid'(theta) * (bmax - bmin)."""
    from oracle import oracle as O
    o, i = W.shape
    wq, un = O.fake_quant(W.reshape(-1, 8), beta.reshape(-1), blocks_per_tile, 4, clip)
    wq64 = torch.from_numpy(wq.reshape(o, i).astype(np.float64)).requires_grad_(True)
    x64 = torch.from_numpy(x.astype(np.float64)).requires_grad_(True)
    b64 = torch.from_numpy(bias.astype(np.float64)).requires_grad_(True)
    y = torch.nn.functional.linear(x64, wq64, b64)
    ((y - torch.from_numpy(t.astype(np.float64))) ** 2).mean().backward()
    g = wq64.grad.numpy().reshape(-1, 8)
    inside = (np.abs(un.astype(np.float64)) <= clip)  # clamp passes the gradient on the closed interval
    dW = (g * inside).reshape(o, i)
    beta_blocks = np.repeat(beta.reshape(-1).astype(np.float64), blocks_per_tile)[:, None]
    per_block = (g * inside * (W.reshape(-1, 8).astype(np.float64) - un.astype(np.float64)) / beta_blocks).sum(axis=1)
    dbeta = per_block.reshape(-1, blocks_per_tile).sum(axis=1)
    sg = 1.0 / (1.0 + np.exp(-theta.astype(np.float64)))
    dtheta = dbeta * sg * (1.0 - sg) * (bmax.astype(np.float64) - bmin.astype(np.float64))
    return {"Wq": wq.reshape(o, i), "y": y.detach().numpy(), "dW": dW, "dx": x64.grad.numpy(), "dbias": b64.grad.numpy(),
            "dtheta": dtheta}


@pytest.mark.parametrize("tag", ["small", "big", "mid"])
def test_layer_forward_backward_row_tiling(golden_layer, tag):
    """Every assertion always runs.  The layer's scale comes from the device sigmoid and may differ
    from the fixture's CPU value in the last bit, so the expectation is (1) the oracle evaluated with
    the layer's own scales, bit for bit for the weights and to 1e-5 for outputs and gradients, and
    (2) the reference layer's fixture on every row whose codes are the fixture's (a last-bit change of
    the scale rescales a row by that bit; a changed code is an O(1) jump), which must be nearly all rows."""
    g = golden_layer
    layer = make_layer(g, tag)
    beta = layer._beta().detach().cpu().numpy()
    assert rel(beta, g[f"{tag}_beta"]) < 1e-6
    x = dev(g[f"{tag}_x"]).requires_grad_(True)
    y = layer(x)
    ((y - dev(g[f"{tag}_t"])) ** 2).mean().backward()
    wq = layer._quantize_weights().detach().cpu().numpy()
    o, i = wq.shape
    want = expected_from_oracle(g[f"{tag}_W"], beta, g[f"{tag}_theta"], g[f"{tag}_bmin"], g[f"{tag}_bmax"],
                                g[f"{tag}_bias"], g[f"{tag}_x"], g[f"{tag}_t"], i // 8)
    got = {"y": y.detach().cpu().numpy(), "dW": layer.weight.grad.cpu().numpy(), "dx": x.grad.cpu().numpy(),
           "dbias": layer.bias.grad.cpu().numpy(), "dtheta": layer.theta_beta.grad.cpu().numpy()}
    # (1) against the oracle with the layer's own scales
    assert np.array_equal(bits(wq), bits(want["Wq"]))
    for k in ("y", "dW", "dx", "dbias"):
        assert rel(got[k], want[k]) < 1e-5, k
    assert np.abs(got["dtheta"] - want["dtheta"]).max() <= 2e-4 * np.abs(want["dtheta"]).max() + 1e-9
    # (2) against the reference layer's own outputs, row by row
    want_wq = g[f"{tag}_Wq"]
    same = (np.abs(wq - want_wq) <= 1e-6 * np.abs(want_wq)).all(axis=1)
    assert same.mean() >= 0.95, same.mean()
    assert (beta == g[f"{tag}_beta"]).mean() >= 0.5  # most scales are bit-identical to the CPU value
    assert rel(got["y"][:, same], g[f"{tag}_y"][:, same]) < 1e-5
    assert rel(got["dW"][same], g[f"{tag}_dW"][same]) < 1e-5
    assert rel(got["dbias"][same], g[f"{tag}_dbias"][same]) < 1e-5
    wt = g[f"{tag}_dtheta"]
    assert np.abs(got["dtheta"][same] - wt[same]).max() <= 2e-4 * np.abs(wt).max() + 1e-9
    if same.all():
        assert rel(got["dx"], g[f"{tag}_dx"]) < 1e-5


def test_state_dict_keys_and_warmup(golden_layer):
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(64, 48, warmup_epochs=2, device="cuda")
    assert set(layer.state_dict().keys()) == {"weight", "bias", "theta_beta", "G", "Ginv", "sigma_ema", "xmax_ema",
                                              "step_count", "gamma_inv"}
    assert not layer.is_quantization_enabled()
    x = torch.randn(4, 64, device="cuda")
    y0 = layer(x)
    assert torch.allclose(y0, torch.nn.functional.linear(x, layer.weight, layer.bias))
    layer.update_epoch(1)
    assert not layer.is_quantization_enabled()
    layer.update_epoch(2)
    assert layer.is_quantization_enabled()
    layer(x)
    assert int(layer.step_count) == 1
    other = create_e8_hnlq_linear(64, 48, device="cuda")
    other.load_state_dict(layer.state_dict())
    assert other._step_host == 1
    with pytest.raises(ValueError):
        create_e8_hnlq_linear(60, 48)
    with pytest.raises(ValueError):
        layer.load_weights(torch.zeros(3, 3))


def test_bf16_activations(golden_layer):
    g = golden_layer
    layer = make_layer(g, "mid")
    x = dev(g["mid_x"])
    y32 = layer(x)
    y16 = layer(x.to(torch.bfloat16))
    assert y16.dtype == torch.bfloat16
    assert rel(y16.detach().float().cpu().numpy(), y32.detach().cpu().numpy()) < 1e-2
    y16.float().sum().backward()
    assert layer.weight.grad is not None and layer.theta_beta.grad is not None


def test_training_step_is_graph_capturable():
    """Forward + backward of the layer enqueue work only on the current stream: one CUDA graph replays
    the step and yields the gradients of the eager step."""
    import warnings
    from coset_b200.core.e8 import create_e8_hnlq_linear
    torch.manual_seed(0)
    layer = create_e8_hnlq_linear(64, 48, q=4, M=2, init_kwargs={"std": 20.0}, device="cuda")
    x = torch.randn(32, 64, device="cuda")
    t = torch.randn(32, 48, device="cuda")

    def step():
        ((layer(x) - t) ** 2).mean().backward()

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            layer.zero_grad(set_to_none=True)
            step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    layer.zero_grad(set_to_none=True)
    g = torch.cuda.CUDAGraph()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        with torch.cuda.graph(g):
            step()
    g.replay()
    torch.cuda.synchronize()
    gw, gt = layer.weight.grad.clone(), layer.theta_beta.grad.clone()
    layer.zero_grad(set_to_none=True)
    step()
    torch.cuda.synchronize()
    assert torch.equal(gw, layer.weight.grad)
    assert torch.allclose(gt, layer.theta_beta.grad, rtol=1e-6, atol=0)


def test_graphed_train_step_keeps_the_statistics_schedule():
    """GraphedTrainStep replays forward + loss + backward as one CUDA graph and does the layer's host-side
    bookkeeping itself: after 520 steps (two statistics updates, weights changed in between) the EMA
    buffers, the step counter, the loss and the gradients are those of 520 eager steps."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    from coset_b200.core.layers import GraphedTrainStep
    torch.manual_seed(0)
    a = create_e8_hnlq_linear(64, 48, q=4, M=2, init_kwargs={"std": 20.0}, device="cuda")
    b = create_e8_hnlq_linear(64, 48, q=4, M=2, device="cuda")
    b.load_state_dict(a.state_dict())
    x = torch.randn(32, 64, device="cuda")
    t = torch.randn(32, 48, device="cuda")
    loss_fn = lambda y, tt: ((y - tt) ** 2).mean()
    step = GraphedTrainStep(b, loss_fn, (x, t))
    assert int(b.step_count) == int(a.step_count) == 0
    delta = torch.randn_like(a.weight) * 3.0
    for i in range(1, 521):
        a.zero_grad(set_to_none=True)
        la = loss_fn(a(x), t)
        la.backward()
        lb = step(x, t)
        if i == 300:
            with torch.no_grad():
                a.weight.add_(delta)
                b.weight.add_(delta)
    torch.cuda.synchronize()
    assert int(a.step_count) == int(b.step_count) == 520
    assert torch.equal(a.sigma_ema, b.sigma_ema) and torch.equal(a.xmax_ema, b.xmax_ema)
    assert not torch.equal(a.sigma_ema, torch.ones_like(a.sigma_ema))
    assert torch.equal(la, lb)
    assert torch.equal(a.weight.grad, b.weight.grad)
    assert torch.allclose(a.theta_beta.grad, b.theta_beta.grad, rtol=1e-6, atol=0)


@pytest.mark.parametrize("tiling", ["row", "block"])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 1e-2)])
def test_one_node_equals_the_composed_path(tiling, dtype, tol):
    """The layer's single autograd node against the composed path (which diagnostics force: quantised weights as one
    node, then F.linear), forward, backward and the gradient of a gradient (create_graph)."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    torch.manual_seed(3)
    grads = []
    for diagnostics in (False, True):
        layer = create_e8_hnlq_linear(72, 40, device="cuda", tiling=tiling, init_method="zeros", enable_diagnostics=diagnostics)
        torch.manual_seed(4)
        layer.load_weights(torch.randn(40, 72) * 20.0, torch.randn(40))
        x = torch.randn(3, 11, 72, device="cuda").to(dtype).requires_grad_()
        y = layer(x)
        gx, = torch.autograd.grad((y.float() ** 2).sum(), x, create_graph=True)
        (y.float().sum() + (gx.float() ** 2).sum()).backward()
        grads.append((y.detach(), gx.detach(), x.grad, layer.weight.grad, layer.theta_beta.grad, layer.bias.grad))
    for one, composed in zip(*grads):
        assert one.shape == composed.shape and one.dtype == composed.dtype
        assert rel(one.float().cpu().numpy(), composed.float().cpu().numpy()) < tol


def test_forward_mode_derivative_in_the_input():
    """The product is linear in x: the tangent is t W_q^T."""
    import torch.autograd.forward_ad as fa
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(64, 32, device="cuda")
    layer.load_weights(torch.randn(32, 64, device="cuda") * 20.0, torch.randn(32, device="cuda"))
    x, t = torch.randn(8, 64, device="cuda"), torch.randn(8, 64, device="cuda")
    with fa.dual_level():
        y, tangent = fa.unpack_dual(layer(fa.make_dual(x, t)))
    torch.testing.assert_close(y.detach(), layer(x).detach(), rtol=1e-5, atol=1e-4)
    torch.testing.assert_close(tangent.detach(), (layer(t) - layer.bias).detach(), rtol=1e-5, atol=1e-3)


def test_bias_of_another_type_is_refused_for_float32():
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(64, 32, device="cuda")
    layer.bias.data = layer.bias.data.to(torch.bfloat16)
    with pytest.raises(RuntimeError):
        layer(torch.randn(8, 64, device="cuda"))
    assert layer(torch.randn(8, 64, device="cuda").to(torch.bfloat16)).dtype == torch.bfloat16


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(0, 8), (1, 1), (255, 31), (256, 32), (257, 33), (4096, 776), (3, 4100), (5000, 64)])
def test_column_sum(rows, cols, dtype):
    """Ragged row groups and column strips, rows that are and are not a multiple of 16 bytes, an unaligned matrix.  The sums
    are float32 with at most rows / 256 + 40 additions in a chain."""
    from coset_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    for offset in (0, 1):
        x = torch.randn(rows * cols + offset, device="cuda", generator=g).to(dtype)[offset:].view(rows, cols)
        want, size = x.double().sum(0), x.double().abs().sum(0)
        for out_dtype, code in ((torch.float32, _lib.DTYPE_F32), (torch.bfloat16, _lib.DTYPE_BF16)):
            y = torch.full((cols,), float("nan"), device="cuda", dtype=out_dtype)
            rc = _lib.lib().coset_column_sum(x.data_ptr(), _lib.dtype_code(x, "x"), rows, cols, _lib.ptr(y), code, _lib.stream())
            _lib.check(rc, "coset_column_sum")
            bound = size * (rows / 256 + 40) * 2.0 ** -24 + (want.abs() * 2.0 ** -8 if out_dtype is torch.bfloat16 else 0)
            assert bool(((y.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("grad", ["dense", "expanded"])
def test_bias_gradient_of_any_layout(grad):
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(64, 40, device="cuda")
    x = torch.randn(3, 50, 64, device="cuda")
    y = layer(x)
    if grad == "dense":
        gy = torch.randn_like(y)
        y.backward(gy)
    else:
        gy = torch.ones_like(y)
        y.sum().backward()
    torch.testing.assert_close(layer.bias.grad, gy.sum((0, 1)), rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("tiling", ["row", "block"])
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 1e-2)])
@pytest.mark.parametrize("made", ["without", "removed"])
def test_layer_without_a_bias(made, tiling, dtype, tol):
    """bias=False, and a bias taken away later, against the composed path: no_grad, backward and the gradient of a gradient."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    results = []
    for diagnostics in (False, True):
        layer = create_e8_hnlq_linear(72, 40, device="cuda", tiling=tiling, init_method="zeros", bias=made == "removed", enable_diagnostics=diagnostics)
        layer.bias = None
        g = torch.Generator(device="cuda").manual_seed(4)
        with torch.no_grad():
            layer.weight.copy_(torch.randn(40, 72, device="cuda", generator=g) * 20.0)
        x = torch.randn(3, 11, 72, device="cuda", generator=g).to(dtype).requires_grad_()
        with torch.no_grad():
            still = layer(x)
        y = layer(x)
        gx, = torch.autograd.grad((y.float() ** 2).sum(), x, create_graph=True)
        (y.float().sum() + (gx.float() ** 2).sum()).backward()
        assert torch.equal(still, y)
        results.append((y.detach(), gx.detach(), x.grad, layer.weight.grad, layer.theta_beta.grad))
    for one, composed in zip(*results):
        assert one.shape == composed.shape and one.dtype == composed.dtype
        assert rel(one.float().cpu().numpy(), composed.float().cpu().numpy()) < tol


@pytest.mark.parametrize("how", ["parametrised", "pruned", "plain attribute"])
def test_bias_that_is_no_plain_parameter(how):
    """The layer reads its bias as an attribute: one that a parametrisation computes, a pruned one, a plain tensor."""
    from torch.nn.utils import parametrize, prune
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(64, 32, device="cuda")
    with torch.no_grad():
        layer.bias.copy_(torch.randn(32))
    x = torch.randn(8, 64, device="cuda")
    y, bias = layer(x).detach(), layer.bias.detach().clone()
    if how == "parametrised":
        class Double(torch.nn.Module):
            def forward(self, b):
                return 2 * b
        parametrize.register_parametrization(layer, "bias", Double())
    elif how == "pruned":
        prune.l1_unstructured(layer, "bias", 0.5)
    else:
        del layer._parameters["bias"]
        layer.bias = torch.ones(32, device="cuda")
    steps = layer._step_host
    got = layer(x)
    torch.testing.assert_close(got.detach(), y - bias + layer.bias.detach(), rtol=1e-5, atol=1e-4)
    assert layer._step_host == steps + 1
    if how == "parametrised":
        got.sum().backward()
        torch.testing.assert_close(layer.parametrizations.bias.original.grad, torch.full((32,), 16.0, device="cuda"))


@pytest.mark.parametrize("tiling", ["row", "block"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_traced_layer_follows_its_weights(tiling, dtype):
    """A trace quantises the weights it finds when it runs, and its gradients reach weight, scale and bias."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(64, 32, device="cuda", tiling=tiling)
    with torch.no_grad():
        layer.weight.copy_(torch.randn(32, 64) * 20.0)
        layer.bias.copy_(torch.randn(32))
    x = torch.randn(8, 64, device="cuda").to(dtype)
    traced = torch.jit.trace(layer, x, check_trace=False)
    with torch.no_grad():
        layer.weight.mul_(1.5)
        layer.bias.add_(1.0)
    y = traced(x)
    assert torch.equal(y, layer(x))
    y.float().sum().backward()
    got = [p.grad.clone() for p in (layer.weight, layer.theta_beta, layer.bias)]
    layer.zero_grad()
    layer(x).float().sum().backward()
    for a, b in zip(got, (layer.weight.grad, layer.theta_beta.grad, layer.bias.grad)):
        torch.testing.assert_close(a, b, rtol=1e-2 if dtype == torch.bfloat16 else 1e-5, atol=1e-3)


def test_subclasses_and_function_modes_see_the_product():
    from torch.overrides import TorchFunctionMode
    from coset_b200.core.e8 import create_e8_hnlq_linear

    class Marked(torch.Tensor):
        pass

    class Names(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(getattr(func, "__name__", ""))
            return func(*args, **(kwargs or {}))

    seen = []
    layer = create_e8_hnlq_linear(64, 32, device="cuda")
    x = torch.randn(8, 64, device="cuda")
    want = layer(x)
    assert type(layer(x.as_subclass(Marked))) is Marked
    with Names():
        y = layer(x)
    assert "linear" in seen and torch.equal(y, want)


@pytest.mark.parametrize("rows,cols", [(1, 8), (32, 128), (128, 768), (333, 1001), (8192, 256)])
def test_column_sum_of_float32_is_rounded_once(rows, cols):
    """The sum keeps what rounding takes from it: what is left is the rounding of the result and, at 2^-48 a term, that of the
    corrections.  An infinite sum stays infinite."""
    from coset_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows, cols, device="cuda", generator=g) * 10.0 ** torch.randint(-3, 4, (rows, cols), device="cuda", generator=g)
    x[rows // 2, 3] = float("inf")
    x[rows - 1, 5] = float("nan")
    y = torch.empty(cols, device="cuda")
    rc = _lib.lib().coset_column_sum(x.data_ptr(), _lib.DTYPE_F32, rows, cols, _lib.ptr(y), _lib.DTYPE_F32, _lib.stream())
    _lib.check(rc, "coset_column_sum")
    want, size = x.double().sum(0), x.double().abs().sum(0)
    assert y[3] == float("inf") and y[5].isnan()
    fine = want.isfinite()
    bound = want.abs() * 2.0 ** -24 + size * rows * 2.0 ** -47
    assert bool(((y.double() - want).abs() <= bound)[fine].all())


@pytest.mark.parametrize("frozen,kept", [(True, False), (False, True)])
def test_frozen_layer_does_not_hold_on_to_its_input(frozen, kept):
    """The input serves the gradients of the weight and its scale alone: with both frozen it is free after the forward pass, and
    the gradients of the bias and of what came before are what they are with a trained weight."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(256, 64, device="cuda")
    with torch.no_grad():
        layer.weight.copy_(torch.randn(64, 256) * 20.0)
    layer.weight.requires_grad_(not frozen)
    layer.theta_beta.requires_grad_(not frozen)
    x = torch.randn(4096, 256, device="cuda").requires_grad_()
    layer(x * 2).sum().backward()
    want, bias = x.grad.clone(), layer.bias.grad.clone()
    x.grad = layer.bias.grad = None
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    y = layer(x * 2)
    held = torch.cuda.memory_allocated() - before - y.numel() * 4
    assert (held >= x.numel() * 4) == kept, held
    y.sum().backward()
    assert torch.equal(x.grad, want) and torch.equal(layer.bias.grad, bias)
    assert (layer.weight.grad is None) == frozen


@pytest.mark.parametrize("tokens,n_out,n_in", [(1, 8, 8), (63, 72, 136), (128, 768, 768), (257, 264, 520), (1000, 1024, 64), (4096, 200, 328)])
@pytest.mark.parametrize("bias", [True, False])
def test_bf16_products_of_a_training_step(tokens, n_out, n_in, bias):
    """The layer's own products, forward and backward: edges of the tiles, K in one part and in several, against 64 bits."""
    from coset_b200 import _lib
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(n_in, n_out, device="cuda", tiling="row", bias=bias, init_method="zeros")
    layer.load_weights(torch.randn(n_out, n_in, device="cuda") * 20.0, torch.randn(n_out, device="cuda") if bias else None)
    x = torch.randn(tokens, n_in, device="cuda").bfloat16().requires_grad_()
    g = torch.randn(tokens, n_out, device="cuda").bfloat16()
    y = layer(x)
    y.backward(g)
    wq = layer._quantize_weights(torch.bfloat16).detach().double()
    b = layer.bias.detach().bfloat16().double() if bias else torch.zeros(n_out, device="cuda", dtype=torch.float64)
    xd, gd = x.detach().double(), g.double()
    # one rounding to 8 significant bits, and float32 sums whose parts round or truncate relative to the sum of the magnitudes
    for got, want, size in ((y.detach(), xd @ wq.T + b, xd.abs() @ wq.abs().T + b.abs()), (x.grad, gd @ wq, gd.abs() @ wq.abs())):
        assert got.dtype == torch.bfloat16 and bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -22 * size).all())
    dw = torch.empty(n_out, n_in, dtype=torch.bfloat16, device="cuda")
    assert _lib.lib().coset_dense_weight_grad(_lib.ptr(g), _lib.ptr(x), tokens, n_out, n_in, _lib.ptr(dw), None, _lib.stream()) == 0
    want, size = gd.T @ xd, gd.abs().T @ xd.abs()
    assert bool(((dw.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -22 * size).all())


@pytest.mark.parametrize("T,n_out,n_in", [(1, 1, 1), (3, 5, 7), (33, 65, 31), (32, 64, 128), (128, 96, 129), (70, 130, 1000), (257, 200, 64), (64, 1024, 2048)])
def test_float32_products_of_a_training_step(T, n_out, n_in):
    """Odd lengths and whole tiles, one to eight parts of K, against 64 bits and the library's error."""
    from coset_b200 import _lib
    L, st = _lib.lib(), _lib.stream()
    x, w, b, g = (torch.randn(*s, device="cuda") for s in ((T, n_in), (n_out, n_in), (n_out,), (T, n_out)))
    y, dx, dw = torch.empty(T, n_out, device="cuda"), torch.empty_like(x), torch.empty_like(w)
    assert L.coset_f32_linear(_lib.ptr(x), _lib.ptr(w), _lib.ptr(b), T, n_out, n_in, _lib.ptr(y), st) == 0
    assert L.coset_f32_input_grad(_lib.ptr(g), _lib.ptr(w), T, n_out, n_in, _lib.ptr(dx), st) == 0
    assert L.coset_f32_weight_grad(_lib.ptr(g), _lib.ptr(x), T, n_out, n_in, _lib.ptr(dw), st) == 0
    xd, wd, bd, gd = x.double(), w.double(), b.double(), g.double()
    for got, want, size in ((y, xd @ wd.T + bd, xd.abs() @ wd.abs().T + bd.abs()), (dx, gd @ wd, gd.abs() @ wd.abs()), (dw, gd.T @ xd, gd.abs().T @ xd.abs())):
        # chains of 128 roundings and at most 24 more additions, each within 2^-24 of the sum of the magnitudes
        assert bool(((got.double() - want).abs() <= 152 * 2.0 ** -24 * size).all())
    assert L.coset_f32_linear(_lib.ptr(x), _lib.ptr(w), None, T, n_out, n_in, _lib.ptr(dx) if T * n_in >= T * n_out else _lib.ptr(y), st) == 0
    assert L.coset_f32_linear(_lib.ptr(x), None, None, T, n_out, n_in, _lib.ptr(y), st) < 0 and L.coset_f32_linear(_lib.ptr(x), _lib.ptr(w), None, T, n_out, 0, _lib.ptr(y), st) < 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("form", ["expanded", "strided", "offset", "three"])
def test_own_products_with_awkward_tensors(form, dtype):
    """Gradients and inputs that the own products cannot read, or read only as rows, give what plain ones give."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(64, 48, device="cuda", tiling="row", init_method="zeros")
    layer.load_weights(torch.randn(48, 64, device="cuda") * 20.0, torch.randn(48, device="cuda"))
    x, g = torch.randn(24, 64, device="cuda").to(dtype), torch.randn(24, 48, device="cuda").to(dtype)
    if form == "expanded":
        g = g[:1].expand(24, 48)

    def step(x, g):
        layer.zero_grad()
        x = x.detach().requires_grad_()
        y = layer(x)
        y.backward(g)
        return [t.reshape(-1).float() for t in (y.detach(), x.grad, layer.weight.grad, layer.theta_beta.grad, layer.bias.grad)]
    want = step(x, g.contiguous())
    if form == "strided":
        x, g = torch.cat([x, x], 1)[:, :64], torch.cat([g, g], 1)[:, :48]
    elif form == "offset":
        x = torch.cat([x.new_zeros(1), x.reshape(-1)])[1:].view(24, 64)
        g = torch.cat([g.new_zeros(1), g.reshape(-1)])[1:].view(24, 48)
    elif form == "three":
        x, g = x.view(4, 6, 64), g.view(4, 6, 48)
    unit = 2.0 ** -7 if dtype == torch.bfloat16 else 64 * 2.0 ** -23  # sums of at most 64 products in another order, then the type's rounding
    for a, b in zip(step(x, g), want):
        assert torch.allclose(a, b, rtol=unit, atol=unit * float(b.abs().max()))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_own_products_are_for_tensors_of_one_device(dtype):
    """A tensor elsewhere is torch's to refuse; the own kernels would read another device's memory."""
    from coset_b200 import _lib
    from coset_b200.core.e8 import create_e8_hnlq_linear
    own = _lib.native().own_product
    x, w, b = torch.randn(64, 128, device="cuda").to(dtype), torch.randn(96, 128, device="cuda"), torch.randn(96, device="cuda")
    assert own(x, w, b) and own(x, w, None) and own(x.view(8, 8, 128), w, b)
    assert not own(x, w.cpu(), None) and not own(x.cpu(), w, None) and not own(x, w, b.cpu())
    if torch.cuda.device_count() > 1:
        with pytest.raises(RuntimeError, match="device"):
            create_e8_hnlq_linear(128, 96, device="cuda:0")(x.to("cuda:1"))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_bias_that_is_no_row_is_torchs(dtype):
    """A bias of another shape is broadcast, or refused, by torch's product; the own one would add it per feature."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(128, 96, device="cuda")
    b = torch.randn(96, device="cuda")
    x = torch.randn(96, 128, device="cuda").to(dtype)
    without = create_e8_hnlq_linear(128, 96, device="cuda", bias=False)
    without.load_state_dict({k: v for k, v in layer.state_dict().items() if k != "bias"})
    unit = 2.0 ** -7 if dtype == torch.bfloat16 else 128 * 2.0 ** -23  # one more rounding of the result; sums of 128 products in another order
    for shape in ((1, 96), (96, 1)):
        layer.bias = torch.nn.Parameter(b.view(shape))
        with torch.no_grad():
            want = without(x).float() + b.to(dtype).float().view(shape)  # 96 tokens: a column is a value per token
            assert torch.allclose(layer(x).float(), want, rtol=unit, atol=unit * float(want.abs().max()))
    with pytest.raises(RuntimeError), torch.no_grad():
        layer(x[:64])


@pytest.mark.parametrize("dtype,tokens", [(torch.float32, 65535 * 32 + 1), (torch.bfloat16, 65535 * 256 + 1)])
def test_training_step_of_more_tokens_than_the_own_products_take(dtype, tokens):
    """One tile of tokens more than a grid of the own kernels holds: torch's products, as for any long and narrow step."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(8, 8, device="cuda", tiling="row", init_method="zeros", bias=False)
    layer.load_weights(torch.randn(8, 8, device="cuda") * 20.0)
    x = torch.randn(tokens, 8, device="cuda").to(dtype).requires_grad_()
    y = layer(x)
    y.backward(x.detach())
    wq = layer._quantize_weights(dtype).detach()
    assert torch.equal(y, torch.nn.functional.linear(x, wq)) and torch.equal(x.grad, torch.mm(x.detach(), wq)) and layer.weight.grad is not None


@pytest.mark.parametrize("dtype,tokens,own", [(torch.bfloat16, 257, False), (torch.float32, 257, True), (torch.float32, 1601, False)])
def test_captured_step_records_the_quicker_products(dtype, tokens, own):
    """A captured step records torch's products where they are quicker on the device, bit for bit, and agrees with the eager step either way."""
    from coset_b200 import _lib
    from coset_b200.core.e8 import create_e8_hnlq_linear
    from coset_b200.core.layers import GraphedTrainStep
    layer = create_e8_hnlq_linear(520, 264, device="cuda", tiling="row", init_method="zeros")
    layer.load_weights(torch.randn(264, 520, device="cuda") * 20.0, torch.randn(264, device="cuda"))
    x, g = torch.randn(tokens, 520, device="cuda").to(dtype), torch.randn(tokens, 264, device="cuda").to(dtype)
    seen = {}

    def loss(y, g):
        seen["y"] = y
        if torch.cuda.is_current_stream_capturing():
            seen["own"] = _lib.native().own_product(x, layer.weight, layer.bias)
        return (y * g).sum()
    step = GraphedTrainStep(layer, loss, (x, g))
    step(x, g)
    assert seen["own"] == own and _lib.native().own_product(x, layer.weight, layer.bias)
    replayed = [seen["y"].detach().clone(), layer.weight.grad.clone(), layer.bias.grad.clone()]
    wq, b = layer._quantize_weights(dtype).detach(), layer.bias.detach().to(dtype)
    if not own:
        assert torch.equal(replayed[0], torch.nn.functional.linear(x, wq, b))
    layer.zero_grad()
    y = layer(x)
    (y * g).sum().backward()
    unit = 2.0 ** -7 if dtype == torch.bfloat16 else 1601 * 2.0 ** -23  # the type's rounding; sums of at most 1601 products in another order
    for a, b in zip(replayed, (y.detach(), layer.weight.grad, layer.bias.grad)):
        assert torch.allclose(a.float(), b.float(), rtol=unit, atol=unit * float(b.abs().max()))


@pytest.mark.parametrize("how", ["allow_tf32", "high"])
def test_float32_step_follows_the_callers_choice_of_tf32(how):
    """Where torch may multiply in TF32 the layer's products are torch's, forward and backward; elsewhere the own ones, in float32."""
    from coset_b200 import _lib
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(256, 192, device="cuda", tiling="row", init_method="zeros", bias=False)
    layer.load_weights(torch.randn(192, 256, device="cuda") * 20.0)
    x, g = torch.randn(128, 256, device="cuda").requires_grad_(), torch.randn(128, 192, device="cuda")
    wq = layer._quantize_weights().detach()
    assert _lib.native().own_product(x, layer.weight, None)
    precision = torch.get_float32_matmul_precision()
    try:
        if how == "high":
            torch.set_float32_matmul_precision("high")
        else:
            torch.backends.cuda.matmul.allow_tf32 = True
        assert not _lib.native().own_product(x, layer.weight, None)
        y = layer(x)
        y.backward(g)
        assert torch.equal(y, torch.nn.functional.linear(x, wq)) and torch.equal(x.grad, torch.mm(g, wq))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = False
        torch.set_float32_matmul_precision(precision)
    assert _lib.native().own_product(x, layer.weight, None)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gradients_of_a_batch_of_output_gradients(dtype):
    """is_grads_batched: the backward pass gets a batch of a transform, which has no memory of its own to look at."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(256, 192, device="cuda", tiling="row", init_method="zeros")
    layer.load_weights(torch.randn(192, 256, device="cuda") * 20.0)
    x, g = torch.randn(64, 256, device="cuda").to(dtype).requires_grad_(), torch.randn(3, 64, 192, device="cuda").to(dtype)
    got, = torch.autograd.grad(layer(x), x, g, is_grads_batched=True)
    unit = 2.0 ** -7 if dtype == torch.bfloat16 else 192 * 2.0 ** -23  # the type's rounding; sums of 192 products in another order
    for one, batch in zip(g, got):
        want, = torch.autograd.grad(layer(x), x, one)
        assert torch.allclose(batch.float(), want.float(), rtol=unit, atol=unit * float(want.abs().max()))


@pytest.mark.parametrize("dtype,cast", [(torch.float32, torch.bfloat16), (torch.float32, torch.float16), (torch.bfloat16, torch.float16)])
def test_backward_under_autocast_multiplies_in_its_type(dtype, cast):
    """A backward pass inside an autocast region: its products are torch's, in the region's type, as in a composed layer."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(256, 192, device="cuda", tiling="row", init_method="zeros", bias=False)
    layer.load_weights(torch.randn(192, 256, device="cuda") * 20.0)
    x, g = torch.randn(64, 256, device="cuda").to(dtype).requires_grad_(), torch.randn(64, 192, device="cuda").to(dtype)
    wq = layer._quantize_weights(dtype).detach()
    y = layer(x)
    with torch.autocast("cuda", dtype=cast):
        y.backward(g)
    assert torch.equal(x.grad, torch.mm(g.to(cast), wq.to(cast)).to(dtype))


@pytest.mark.parametrize("dtype,tokens,n_out,n_in", [(torch.float32, 32, 32, 64), (torch.float32, 128, 768, 768), (torch.bfloat16, 8, 32, 64), (torch.bfloat16, 300, 264, 1032)])
def test_traced_layer_agrees_to_the_rounding_of_the_type(dtype, tokens, n_out, n_in):
    """A trace records torch's product; the eager layer's own one adds up in another order: the smallest own step in float32 and larger ones."""
    from coset_b200 import _lib
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(n_in, n_out, device="cuda", tiling="row", init_method="zeros")
    layer.load_weights(torch.randn(n_out, n_in, device="cuda") * 20.0, torch.randn(n_out, device="cuda"))
    x = torch.randn(tokens, n_in, device="cuda").to(dtype)
    assert _lib.native().own_product(x, layer.weight, layer.bias)
    traced = torch.jit.trace(layer, x, check_trace=False)
    with torch.no_grad():
        y, t = layer(x).float(), traced(x).float()
    wq, b = layer._quantize_weights(dtype).detach().float(), layer.bias.detach().to(dtype).float()
    size = x.float().abs() @ wq.abs().T + b.abs()
    # each side rounds to the type once (to half a unit); their float32 sums of n_in products differ by at most that many roundings each way
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    assert bool(((y - t).abs() <= unit * torch.maximum(y.abs(), t.abs()) + 2 * (n_in + 1) * 2.0 ** -24 * size).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,n_out,n_in", [(64, 128, 256), (200, 328, 520), (1000, 512, 264)])
def test_chained_products_read_what_the_call_before_wrote(dtype, T, n_out, n_in):
    """The products start while the one before them drains: a chain in which each overwrites what the one before has read leaves what the calls
    leave one by one."""
    from coset_b200 import _lib
    L, P, f32 = _lib.lib(), _lib.ptr, dtype == torch.float32
    g = torch.Generator(device="cuda").manual_seed(T)
    first = [torch.randn(s, device="cuda", generator=g).to(dtype) for s in ((T, n_in), (n_out, n_in))]

    def chain(wait):
        x, w = (t.clone() for t in first)
        y, left = torch.empty(T, n_out, device="cuda", dtype=dtype), []
        for _ in range(12):
            st = _lib.stream()
            for call in ((lambda: L.coset_f32_linear(P(x), P(w), None, T, n_out, n_in, P(y), st)) if f32 else
                         (lambda: L.coset_e8_dense_linear(P(w), n_out, n_in, P(x), n_in, T, None, 0, P(y), n_out, None, st)),
                         (lambda: L.coset_f32_input_grad(P(y), P(w), T, n_out, n_in, P(x), st)) if f32 else
                         (lambda: L.coset_dense_input_grad(P(y), P(w), T, n_out, n_in, P(x), None, st)),
                         (lambda: L.coset_f32_weight_grad(P(y), P(x), T, n_out, n_in, P(w), st)) if f32 else
                         (lambda: L.coset_dense_weight_grad(P(y), P(x), T, n_out, n_in, P(w), None, st))):
                assert call() == 0
                wait()
            left.append([t.clone() for t in (x, w, y)])
            for t in (x, w):  # back to the size of the start
                t.div_(t.float().abs().amax().to(dtype) + 1e-6)
        return left
    for a, b in zip(chain(torch.cuda.synchronize), chain(lambda: None)):
        assert all(torch.equal(s, t) and bool(s.isfinite().all()) for s, t in zip(a, b))


def test_steps_and_products_from_two_threads():
    """A training layer and a code layer each, on a stream of their own, in two threads: the results are those of one thread."""
    import threading
    from coset_b200.core.e8 import create_e8_hnlq_linear
    from coset_b200.vlut import E8CodeLinear

    def work(seed, results):
        g = torch.Generator(device="cuda").manual_seed(seed)
        with torch.cuda.stream(torch.cuda.Stream()):
            for dtype, tokens, n_out, n_in in ((torch.bfloat16, 300 + 256 * seed, 256, 512), (torch.float32, 64 + 64 * seed, 192, 256)):
                layer = create_e8_hnlq_linear(n_in, n_out, device="cuda", tiling="row", init_method="zeros")
                layer.load_weights(torch.randn(n_out, n_in, device="cuda", generator=g) * 20.0, torch.randn(n_out, device="cuda", generator=g))
                code = E8CodeLinear.from_qat_layer(layer)
                x = torch.randn(tokens, n_in, device="cuda", generator=g).to(dtype).requires_grad_()
                up = torch.randn(tokens, n_out, device="cuda", generator=g).to(dtype)
                for _ in range(200):
                    layer.zero_grad(set_to_none=True)
                    x.grad = None
                    y = layer(x)
                    y.backward(up)
                    with torch.no_grad():
                        z = code(x.detach())
                results += [t.detach().clone() for t in (y, z, x.grad, layer.weight.grad, layer.theta_beta.grad, layer.bias.grad)]
            torch.cuda.current_stream().synchronize()
    alone, together, failures = ([], []), ([], []), []
    for seed in (0, 1):
        work(seed, alone[seed])

    def guarded(seed):
        try:
            work(seed, together[seed])
        except Exception as e:  # noqa: BLE001 - reported by the test's own thread
            failures.append(repr(e))
    threads = [threading.Thread(target=guarded, args=(seed,)) for seed in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
    for a, b in zip(alone, together):
        assert len(a) == len(b) == 12
        for s, t in zip(a, b):
            assert torch.allclose(s.float(), t.float(), rtol=1e-6, atol=0) if s.dim() == 1 else torch.equal(s, t)


@pytest.mark.parametrize("tokens,n_out,n_in", [(1, 768, 768), (2, 512, 1024), (8, 256, 256), (16, 64, 64), (31, 128, 4096), (32, 256, 256), (48, 64, 2048), (128, 768, 768), (2048, 16, 768)])
def test_float32_step_is_as_precise_as_torchs(tokens, n_out, n_in):
    """Against 64 bits, forward and backward: no further off than torch's products of the same values (two such errors differ by a few percent of themselves)."""
    from coset_b200.core.e8 import create_e8_hnlq_linear
    g = torch.Generator(device="cuda").manual_seed(tokens + n_in)
    layer = create_e8_hnlq_linear(n_in, n_out, device="cuda", tiling="row", init_method="zeros", bias=False)
    layer.load_weights(torch.randn(n_out, n_in, device="cuda", generator=g) * 20.0)
    x, up = torch.randn(tokens, n_in, device="cuda", generator=g).requires_grad_(), torch.randn(tokens, n_out, device="cuda", generator=g)
    y = layer(x)
    y.backward(up)
    wq, xs = layer._quantize_weights().detach(), x.detach()
    for got, torchs, exact in ((y.detach(), torch.nn.functional.linear(xs, wq), xs.double() @ wq.double().T), (x.grad, torch.mm(up, wq), up.double() @ wq.double())):
        assert float((got.double() - exact).norm()) <= 1.1 * float((torchs.double() - exact).norm())


@pytest.mark.parametrize("form", ["expanded", "strided", "offset", "three"])
def test_own_float32_products_with_awkward_tensors(form):
    """From 32 tokens on, where float32 steps take the own products: gradients and inputs that they cannot read, or read only as rows."""
    from coset_b200 import _lib
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(64, 48, device="cuda", tiling="row", init_method="zeros")
    layer.load_weights(torch.randn(48, 64, device="cuda") * 20.0, torch.randn(48, device="cuda"))
    x, g = torch.randn(40, 64, device="cuda"), torch.randn(40, 48, device="cuda")
    assert _lib.native().own_product(x, layer.weight, layer.bias)
    if form == "expanded":
        g = g[:1].expand(40, 48)

    def step(x, g):
        layer.zero_grad()
        x = x.detach().requires_grad_()
        y = layer(x)
        y.backward(g)
        return [t.reshape(-1) for t in (y.detach(), x.grad, layer.weight.grad, layer.theta_beta.grad, layer.bias.grad)]
    want = step(x, g.contiguous())
    if form == "strided":
        x, g = torch.cat([x, x], 1)[:, :64], torch.cat([g, g], 1)[:, :48]
    elif form == "offset":
        x, g = torch.cat([x.new_zeros(1), x.reshape(-1)])[1:].view(40, 64), torch.cat([g.new_zeros(1), g.reshape(-1)])[1:].view(40, 48)
    elif form == "three":
        x, g = x.view(4, 10, 64), g.view(4, 10, 48)
    unit = 64 * 2.0 ** -23  # sums of at most 64 products in another order
    for a, b in zip(step(x, g), want):
        assert torch.allclose(a, b, rtol=unit, atol=unit * float(b.abs().max()))


@pytest.mark.parametrize("what", ["bf16", "f32", "code"])
def test_capture_behind_eager_steps_of_the_own_products(what):
    """A graph may record torch's products where the eager steps before were the own kernels': in a process that has made no cuBLAS handle, the capture does."""
    import os
    import subprocess
    import sys
    child = os.path.join(os.path.dirname(os.path.abspath(__file__)), "capture_child.py")
    done = subprocess.run([sys.executable, child, what], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and "ok" in done.stdout, done.stderr[-2000:]
