"""GPU parity of the tcgen05 backward at the edges of its tiles and items: one pair and one item, ragged last tiles, kv tiles that no
query sees (one, and several in a row), items of a single pair, grouped heads; and masks taken from the bit matrix against masks
evaluated in the kernel, which have to agree bit by bit in dK and dV (accumulated in a fixed order).

Tolerance: gradients <= 5e-2 relative to an fp32 reference of the same inputs, the bar of the other backward tests."""
import pytest
import torch

from _util import DTYPES, rel_err

pytestmark = pytest.mark.gpu


def _inputs(B, Hq, Hkv, Sq, Skv, D, dt):
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v, do = (torch.randn(B, h, s, D, generator=g, device="cuda").to(DTYPES[dt]) for h, s in
                   ((Hq, Sq), (Hkv, Skv), (Hkv, Skv), (Hq, Sq)))
    return [t.requires_grad_(True) for t in (q, k, v)], do


def _masks():
    from flaxattention_b200.masks import causal_mask, generate_sliding_window

    def far(b, h, q, kv):      # the keys 128 .. 639 are seen by nobody
        return (kv < 128) | (kv >= 640)

    def one_tile(b, h, q, kv):  # every kv tile pairs with one q tile
        return q // 128 == kv // 128

    def by_head(b, h, q, kv):
        return q >= kv - 64 * h

    return {None: None, "causal": causal_mask, "window": generate_sliding_window(40), "far": far, "one_tile": one_tile, "by_head": by_head}


def _grads(x, do, mask, bits=None):
    import flaxattention_b200 as fa

    q, k, v = x
    bm = None
    if mask is not None:
        by_head = mask.__name__ == "by_head"
        bm = fa.create_block_mask(mask, q.shape[0] if by_head else None, q.shape[1] if by_head else None, q.shape[2], k.shape[2], _mask_bits=bits)
    out, lse = fa.flax_attention_pallas(q, k, v, block_mask=bm, enable_gqa=q.shape[1] != k.shape[1], return_lse=True)
    return torch.autograd.grad(out, x, do)


def _reference(x, do, mask):
    q, k, v = (t.detach().float().requires_grad_(True) for t in x)
    G = q.shape[1] // k.shape[1]
    s = q @ k.repeat_interleave(G, 1).transpose(-1, -2) * q.shape[-1] ** -0.5
    if mask is not None:
        i, j = torch.arange(q.shape[2], device="cuda")[:, None], torch.arange(k.shape[2], device="cuda")[None]
        keep = torch.stack([torch.as_tensor(mask(0, h, i, j)).expand(q.shape[2], k.shape[2]) for h in range(q.shape[1])])[None]
        s = s.masked_fill(~keep, -1e30)
    p = torch.softmax(s, -1)
    if mask is not None:
        p = p * keep.any(-1, keepdim=True)  # (rows without a visible key)
    return torch.autograd.grad(p @ v.repeat_interleave(G, 1), (q, k, v), do.float())


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,dt,mask", [
    (1, 1, 1, 128, 128, "bf16", None),
    (1, 3, 3, 129, 257, "f16", None),
    (2, 2, 2, 1000, 383, "bf16", "causal"),
    (1, 4, 2, 640, 640, "f16", "window"),
    (2, 4, 4, 300, 1153, "bf16", "far"),
    (1, 2, 1, 2048, 2048, "f16", "one_tile"),
    (2, 4, 2, 511, 513, "bf16", "by_head"),
])
def test_gradients_at_the_edges(D, B, Hq, Hkv, Sq, Skv, dt, mask):
    m = _masks()[mask]
    x, do = _inputs(B, Hq, Hkv, Sq, Skv, D, dt)
    got, ref = _grads(x, do, m), _reference(x, do, m)
    for name, a, r in zip(("dq", "dk", "dv"), got, ref):
        assert not torch.isnan(a.float()).any(), name
        assert rel_err(a, r) <= 5e-2, (name, rel_err(a, r))
    if m is not None:
        plain = _grads(x, do, m, bits=False)
        assert torch.equal(got[1], plain[1]) and torch.equal(got[2], plain[2])
        assert rel_err(got[0], plain[0]) <= 1e-2  # (dQ: fp32 sums in another order, rounded to 16 bits)


@pytest.mark.parametrize("D", [64, 128])
def test_a_masked_score_that_overflows_leaves_no_trace(D):
    """The exponential of a masked position is taken and dropped: far above the row's maximum it is infinite."""
    (q, k, v), do = _inputs(1, 2, 2, 256, 256, D, "bf16")
    with torch.no_grad():
        k[:, :, 200:, 0] = 60.0
        q[:, :, :200, 0] = 600.0
    m = _masks()["causal"]
    got, ref = _grads((q, k, v), do, m), _reference((q, k, v), do, m)
    for name, a, r in zip(("dq", "dk", "dv"), got, ref):
        assert not torch.isnan(a.float()).any(), name
        assert rel_err(a, r) <= 5e-2, (name, rel_err(a, r))
