"""CPU-only checks: host-side mirrors, and that the C-ABI library loads and exports every
symbol the public header declares (no compute calls: there is no GPU here)."""
import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol():
    from coset_b200 import _lib, build
    build.build()
    header = open(os.path.join(ROOT, "include", "coset_b200.h")).read()
    declared = set(re.findall(r"\b(coset_[a-z0-9_]+)\s*\(", header))
    assert declared, "no declarations found"
    L = ctypes.CDLL(_lib.LIB_PATH)
    for name in declared:
        assert hasattr(L, name), f"{name} declared in include/coset_b200.h but not exported"
    assert declared == set(_lib.SIGNATURES), declared ^ set(_lib.SIGNATURES)
    assert _lib.lib().coset_version() >= 100
    assert _lib.lib().coset_e8_code_bytes(4, 2) == 4
    assert _lib.lib().coset_e8_code_bytes(16, 3) == 12
    assert _lib.lib().coset_e8_code_bytes(64, 2) == 0


def test_bad_arguments_are_rejected_without_a_gpu():
    from coset_b200 import _lib
    L = _lib.lib()
    assert L.coset_e8_encode(None, 0, None, 0, -1, 1, 4, 2, 0, None, None) < 0
    assert L.coset_e8_encode(None, 0, None, 0, 8, 1, 4, 2, 0, None, None) < 0
    assert b"null" in L.coset_last_error_string()
    assert L.coset_e8_encode(None, 0, None, 0, 0, 1, 99, 2, 0, None, None) < 0
    assert L.coset_e8_decode(None, None, 7, 0, 1, 4, 2, 0, None, 0, None) < 0
    assert L.coset_e8_encode(None, 0, None, 0, 0, 1, 4, 2, 0, None, None) == 0  # empty input is fine


def test_lattice_config_mirror():
    from coset_b200.core.base import LatticeConfig
    c = LatticeConfig(lattice_type="E8", q=4, M=2)
    assert (c.beta, c.alpha, c.decoding, c.with_dither, c.max_scaling_iterations) == (1.0, 1.0, "full", False, 10)
    assert LatticeConfig.from_dict(c.to_dict()) == c
    with pytest.raises(TypeError):
        LatticeConfig(q=4, M=2)
    with pytest.raises(TypeError):
        LatticeConfig(lattice_type="E8", q=4, M=2, bogus=1)


def test_cpu_tensors_are_refused():
    from coset_b200.core.e8 import e8_encode, e8_quantize, E8Lattice
    from coset_b200.core.base import LatticeConfig
    c = LatticeConfig(lattice_type="E8", q=4, M=2)
    with pytest.raises(ValueError, match="CUDA"):
        e8_encode(torch.zeros(4, 8), c)
    with pytest.raises(ValueError, match="CUDA"):
        e8_quantize(torch.zeros(4, 8), 4)
    with pytest.raises(ValueError, match="CUDA"):
        E8Lattice(device="cpu").projection(torch.zeros(4, 8))


def test_lattice_constants_and_helpers_on_cpu():
    from coset_b200.core.e8 import E8Lattice
    L = E8Lattice(device="cpu")
    assert L.name == "E8" and L.d == 8 and L.r_pack == 0.5 and abs(L.r_cov - 2 ** 0.5 / 2) < 1e-12
    assert abs(L.compute_delta0(4, 2, 0.95) - 2 * 0.95 * 0.5 / 15) < 1e-15
    assert torch.equal(L.G @ L.G_inv, torch.eye(8))
    assert L.custom_round(torch.tensor([0.5, -0.5, 1.5, 2.5, -2.5])).tolist() == [0.0, 0.0, 1.0, 3.0, -2.0]
    z = torch.randint(0, 4, (100, 8)).float()
    assert torch.equal(L.encode_coords(L.decode_coords(z, 4), 4), z)


def test_layer_bounds_and_state_on_cpu(golden_layer):
    """_bounds / beta reproduce the reference's numbers; construction works without a GPU."""
    import numpy as np
    from coset_b200.core.e8 import create_e8_hnlq_linear
    g = golden_layer
    layer = create_e8_hnlq_linear(64, 48, device="cpu")
    with torch.no_grad():
        layer.theta_beta.copy_(torch.from_numpy(g["small_theta"]))
        layer.sigma_ema.copy_(torch.from_numpy(g["small_sigma"]))
        layer.xmax_ema.copy_(torch.from_numpy(g["small_xmax"]))
    bmin, bmax = layer._bounds()
    assert np.array_equal(bmin.numpy(), g["small_bmin"]) and np.array_equal(bmax.numpy(), g["small_bmax"])
    assert np.allclose(layer._beta().detach().numpy(), g["small_beta"], rtol=1e-6)
    assert abs(layer.Delta0 - float(g["small_Delta0"])) < 1e-15
    assert float(layer.gamma_inv) == float(g["small_gamma_inv"]) == 12.0
    fresh = create_e8_hnlq_linear(768, 3072, device="cpu")
    assert abs(float(fresh._beta()[0]) - 0.021440971642732620) < 1e-9
    with pytest.raises(ValueError, match="CUDA"):
        layer(torch.zeros(2, 64))
    layer.disable_quantization()
    assert layer(torch.zeros(2, 64)).shape == (2, 48)


def test_scale_bounds_cache_follows_the_statistics():
    """The cached (beta_min, beta_max) are recomputed after any write to the statistics buffers and
    after a hyper-parameter change, and equal the reference formula (coset/core/layers.py:381-396)."""
    import torch
    from coset_b200.core.e8 import create_e8_hnlq_linear
    layer = create_e8_hnlq_linear(64, 8, device="cpu")

    def formula():
        qM = float(layer.q ** layer.M)
        g = float(layer.gamma_inv)
        bmin = (layer.Delta0 / qM) / (layer.eta * g * layer.sigma_ema)
        bmax = torch.minimum((layer.Delta0 * (qM - 1)) / (2 * g * layer.xmax_ema),
                             (layer.Delta0 * (qM - 1)) / (2 * layer.eta * g * layer.sigma_ema))
        return torch.minimum(bmin, bmax * 0.9), bmax

    for mutate in (lambda: None, lambda: layer.sigma_ema.mul_(3.0), lambda: layer.xmax_ema.add_(0.5),
                   lambda: layer.sigma_ema.copy_(torch.rand(8) + 0.1), lambda: setattr(layer, "eta", 0.2)):
        mutate()
        got = layer._bounds()
        again = layer._bounds()
        assert got[0] is again[0]  # served from the cache while nothing changes
        want = formula()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    beta = layer._beta()
    assert torch.equal(beta, want[0] + torch.sigmoid(layer.theta_beta) * (want[1] - want[0]))
    layer.load_state_dict({k: (v * 2 if k == "xmax_ema" else v) for k, v in layer.state_dict().items()})
    assert torch.equal(layer._bounds()[1], formula()[1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float64])
def test_low_precision_parameters_are_refused_before_any_launch(dtype):
    """The fused weight kernels read float32 rows; a layer converted with .bfloat16() / .half() /
    .double() must be refused on the host, not misread on the device."""
    from coset_b200.core.layers import e8_fake_quantize
    from coset_b200.core.d4.layers import d4_fake_quantize, d4_quantize
    w8 = torch.zeros(4, 16, dtype=dtype)
    beta = torch.ones(4)
    with pytest.raises(TypeError, match="float32"):
        e8_fake_quantize(w8, beta, 2)
    with pytest.raises(TypeError, match="float32"):
        d4_fake_quantize(w8, beta, 4)
    with pytest.raises(TypeError, match="float32"):
        d4_quantize(torch.zeros(4, 4, dtype=dtype))


def test_torch_module_is_built_again_for_another_torch(monkeypatch, tmp_path):
    """The module's ABI follows the installed torch and Python: a module of another version counts as out of date, one of this not."""
    from coset_b200 import build
    build.build()
    built = []
    monkeypatch.setattr(build, "TORCH_STAMP", str(tmp_path / "version"))
    monkeypatch.setattr(build, "_build_torch_module", built.append)
    (tmp_path / "version").write_text("torch 1.0\n")
    build.build()
    assert built == [False]
    build.build()
    assert built == [False]


def test_sizes_of_the_training_layers_own_products():
    """What the rule takes fits the kernels' grids, which refuse more than 65535 tiles of tokens; long and narrow steps, whose weight gradient
    would run on a few CTAs, and wide ones, which the device bounds, stay with torch."""
    from coset_b200 import _lib
    own = lambda *sizes, capturing=False: _lib.native().own_product_sizes(*sizes, capturing)
    f32, bf16 = _lib.DTYPE_F32, _lib.DTYPE_BF16
    assert own(f32, 128, 768, 768) and own(f32, 16384, 16, 64) and own(f32, 1024, 512, 512) and own(f32, 8192, 10, 768)
    assert own(bf16, 4096, 3072, 768) and own(bf16, 8192, 4096, 64) and own(bf16, 32768, 64, 64) and own(bf16, 1, 8, 8)
    for tokens in (2097121, 1 << 22):  # 65536 tiles of 32 tokens and more, within 2^28 multiply-adds
        assert not own(f32, tokens, 8, 8)
    for tokens in (65535 * 256 + 1, 1 << 28):
        assert not own(bf16, tokens, 8, 8)
    for tokens, n_out, n_in in ((262144, 16, 64), (65536, 64, 64), (8192, 10, 3200), (0, 64, 64), (2048, 512, 512), (32, 24, 64), (31, 768, 768), (64, 1 << 11, (1 << 11) + 8)):
        assert not own(f32, tokens, n_out, n_in)
    for tokens, n_out, n_in in ((262144, 64, 64), (8192, 64, 6144), (4096, 256, 8192), (64, 1 << 11, (1 << 11) + 8), (64, 60, 64), (64, 64, 60), (8192, 2048, 2048)):
        assert not own(bf16, tokens, n_out, n_in)
    assert not own(f32, 1 << 40, 8, 8) and not own(bf16, 64, 1 << 40, 1 << 40)  # no overflow on the way
    for tokens in range(1, 1 << 25, 99991):
        assert not own(f32, tokens, 8, 8) or tokens <= 65535 * 32
        assert not own(bf16, tokens, 8, 8) or tokens <= 65535 * 32
    # a graph keeps what is quicker on the device
    assert own(f32, 128, 768, 768, capturing=True) and own(f32, 32, 48, 64, capturing=True) and own(f32, 4096, 64, 64, capturing=True)
    for tokens, n_out, n_in in ((1024, 512, 512), (16384, 16, 64)):
        assert own(f32, tokens, n_out, n_in) and not own(f32, tokens, n_out, n_in, capturing=True)
    for tokens, n_out, n_in in ((4096, 3072, 768), (128, 768, 768), (8, 64, 64)):
        assert own(bf16, tokens, n_out, n_in) and not own(bf16, tokens, n_out, n_in, capturing=True)


@pytest.mark.parametrize("size", [2 ** 31 - 1, 2 ** 31 - 8, 2 ** 31 - 512])
def test_dense_products_refuse_sizes_that_their_counts_cannot_hold(size):
    """Before anything is launched: with a tile added such a size wraps around (a count of -1 tiles is not more than the grid takes)."""
    from coset_b200 import _lib
    L = _lib.lib()
    memory = torch.zeros(64, dtype=torch.float32)
    p = (memory.data_ptr() + 127) // 128 * 128
    wide = size // 8 * 8
    if wide > 2 ** 31 - 513:
        assert L.coset_e8_dense_linear(p, 64, wide, p, wide, 64, None, 0, p, 64, None, None) == -2
        assert L.coset_dense_input_grad(p, p, 64, wide, 64, p, None, None) == -2 and L.coset_dense_weight_grad(p, p, 64, 64, wide, p, None, None) == -2
    assert L.coset_e8_dense_linear(p, 64, 64, p, 64, size, None, 0, p, 64, None, None) == -2
    assert L.coset_dense_weight_grad(p, p, size, 64, 64, p, None, None) == -2
    for sizes in ((size, 64, 64), (64, size, 64), (64, 64, size)):
        assert L.coset_f32_linear(p, p, None, *sizes, p, None) == -2
        assert L.coset_f32_input_grad(p, p, *sizes, p, None) == -2 and L.coset_f32_weight_grad(p, p, *sizes, p, None) == -2
