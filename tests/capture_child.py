"""Run by test_gpu_layer.py in a process of its own, in which no torch product has run: captures after eager steps that the own kernels multiplied."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import torch

from coset_b200.core.e8 import create_e8_hnlq_linear
from coset_b200.core.layers import GraphedTrainStep
from coset_b200.vlut import E8CodeLinear


def layer(dtype, tokens, n_out, n_in):
    made = create_e8_hnlq_linear(n_in, n_out, device="cuda", tiling="row", init_method="zeros")
    made.load_weights(torch.randn(n_out, n_in, device="cuda") * 20.0, torch.randn(n_out, device="cuda"))
    return made, torch.randn(tokens, n_in, device="cuda").to(dtype), torch.randn(tokens, n_out, device="cuda").to(dtype)


def step(dtype, tokens, n_out, n_in):
    made, x, g = layer(dtype, tokens, n_out, n_in)
    graphed = GraphedTrainStep(made, lambda y, g: (y.float() * g.float()).sum(), (x, g))
    loss = graphed(x, g).clone()
    got = made.weight.grad.clone()
    made.zero_grad()
    want = (made(x).float() * g.float()).sum()
    want.backward()
    unit = 2.0 ** -6 if dtype == torch.bfloat16 else 1e-4
    assert torch.allclose(got, made.weight.grad, rtol=unit, atol=unit * float(got.abs().max())), "gradients"
    assert bool(loss.isfinite())


def code(tokens, n_out, n_in):
    made, x, _ = layer(torch.bfloat16, tokens, n_out, n_in)
    made = E8CodeLinear.from_qat_layer(made)
    with torch.no_grad():
        want = made(x)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = made(x)
        graph.replay()
    assert torch.allclose(y.float(), want.float(), rtol=2.0 ** -6, atol=2.0 ** -6 * float(want.float().abs().max())), "result"


if __name__ == "__main__":
    what = sys.argv[1]
    if what == "code":
        code(64, 256, 512)
    else:
        step(torch.bfloat16 if what == "bf16" else torch.float32, *((300, 264, 520) if what == "bf16" else (1601, 264, 520)))
    torch.cuda.synchronize()
    print("ok")
