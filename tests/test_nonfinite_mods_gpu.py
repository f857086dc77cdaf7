"""score_mods that are not finite, or whose derivative is not, at positions that do not count: masked ones, and the query
rows beyond the last that fill up a tile.  Nothing of them may reach the gradients: 0 times infinity in a probability's product would be NaN for a whole row of dQ and dK.

Tolerance: gradients <= 5e-2 relative to a reference in 64 bits of the same inputs for 16-bit types, the bar of the other
backward tests, and 1e-4 for fp32."""
import pytest
import torch

from _util import DTYPES, rel_err
from flaxattention_b200 import fnp
from flaxattention_b200.masks import causal_mask

pytestmark = pytest.mark.gpu


def _grads(score, mask, Sq, Skv, D, dt, H=2):
    import flaxattention_b200 as fa

    g = torch.Generator(device="cuda").manual_seed(7)
    x = [torch.randn(1, H, s, D, generator=g, device="cuda").to(DTYPES[dt]) for s in (Sq, Skv, Skv, Sq)]
    q, k, v = (t.requires_grad_(True) for t in x[:3])
    bm = None if mask is None else fa.create_block_mask(mask, None, None, Sq, Skv)
    out = fa.flax_attention_pallas(q, k, v, score_mod=score, block_mask=bm)
    return x, torch.autograd.grad(out, (q, k, v), x[3])


def _check(x, got, values, keep, dt):
    """Against softmax(values(score, q, kv)) over the positions `keep` allows, where values is finite."""
    q, k, v = (t.detach().double().requires_grad_(True) for t in x[:3])
    i, j = torch.arange(q.shape[2], device="cuda")[:, None], torch.arange(k.shape[2], device="cuda")[None]
    s = values(q @ k.transpose(-1, -2) * q.shape[-1] ** -0.5, i, j)
    if keep is not None:
        s = s.masked_fill(~keep(i, j), -1e30)
    p = torch.softmax(s, -1)
    if keep is not None:
        p = p * keep(i, j).any(-1, keepdim=True)  # (rows without a visible key)
    ref = torch.autograd.grad(p @ v, (q, k, v), x[3].double())
    for name, a, r in zip(("dq", "dk", "dv"), got, ref):
        assert torch.isfinite(a.float()).all(), name
        assert rel_err(a, r) <= (1e-4 if dt == "f32" else 5e-2), (name, rel_err(a, r))


def _below(b, h, q, kv):
    return q > kv


MASKED = {  # infinite, or with an infinite derivative, on the diagonal: affine in the score, and not
    "affine": (lambda s, b, h, q, kv: s / (q - kv), lambda s, i, j: s / (i - j).clamp(min=1)),
    "square": (lambda s, b, h, q, kv: s * s / (q - kv), lambda s, i, j: s * s / (i - j).clamp(min=1)),
}


@pytest.mark.parametrize("D,dt", [(64, "bf16"), (64, "f32"), (128, "bf16"), (128, "f16"), (32, "f16")])
@pytest.mark.parametrize("Sq,Skv", [(128, 128), (300, 257)])
@pytest.mark.parametrize("name", list(MASKED))
def test_masked_positions(name, Sq, Skv, D, dt):
    score, values = MASKED[name]
    x, got = _grads(score, _below, Sq, Skv, D, dt)
    _check(x, got, values, lambda i, j: i > j, dt)


BEYOND = {  # not finite from q = Sq on
    "inverse": lambda Sq: (lambda s, b, h, q, kv: s / (Sq - q), lambda s, i, j: s / (Sq - i)),
    "root": lambda Sq: (lambda s, b, h, q, kv: s * fnp.sqrt((Sq - 1 - q) * 1.0), lambda s, i, j: s * (Sq - 1.0 - i).sqrt()),
    "log": lambda Sq: (lambda s, b, h, q, kv: s + fnp.log((Sq - q) * 1.0), lambda s, i, j: s + (Sq - i).double().log()),
    "square": lambda Sq: (lambda s, b, h, q, kv: s * s / (Sq - q), lambda s, i, j: s * s / (Sq - i)),
}


@pytest.mark.parametrize("D,dt", [(64, "bf16"), (64, "f32"), (128, "bf16"), (32, "f16")])
@pytest.mark.parametrize("Sq", [129, 192, 255, 1000])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("name", list(BEYOND))
def test_rows_beyond_the_last(name, masked, Sq, D, dt):
    score, values = BEYOND[name](Sq)
    x, got = _grads(score, causal_mask if masked else None, Sq, 200, D, dt)
    _check(x, got, values, (lambda i, j: i >= j) if masked else None, dt)
