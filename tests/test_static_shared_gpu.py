"""Kernels whose dynamic shared memory is just what a launch may have without asking for more, with mods that read captured tensors, whose
table of addresses is static shared memory on top: the general backward takes 48 KB where head dim and value dim add up to 112."""
import pytest
import torch

from _util import DTYPES, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,Dv", [(80, 32), (96, 16), (64, 48), (80, 16)])  # (the last: below)
def test_general_backward(D, Dv):
    import flaxattention_b200 as fa

    H, S = 2, 255
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k = (torch.randn(1, H, S, D, generator=g, device="cuda").to(DTYPES["f16"]).requires_grad_() for _ in range(2))
    v, dout = (torch.randn(1, H, S, Dv, generator=g, device="cuda").to(DTYPES["f16"]) for _ in range(2))
    v.requires_grad_()
    table = torch.randn(S, generator=g, device="cuda")
    out = fa.flax_attention_pallas(q, k, v, score_mod=lambda s, b, h, i, j: s + table[j])
    got = torch.autograd.grad(out, (q, k, v), dout)
    x = [t.detach().double().requires_grad_() for t in (q, k, v)]
    p = torch.softmax(x[0] @ x[1].transpose(-1, -2) * D ** -0.5 + table.double(), -1)
    for a, r in zip(got, torch.autograd.grad(p @ x[2], x, dout.double())):
        assert rel_err(a, r) <= 5e-2  # the bar of the other backward tests
