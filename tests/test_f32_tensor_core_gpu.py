"""fp32 inputs of head dim 64 on the tensor cores (operands as three bf16 parts): forward and gradients
against an fp64 evaluation, at lengths around the 128-row tiles, the 64-row query tiles of the backward and
the ends of their ranges.  Bounds: 2e-5 of the largest value, the rounding of a few dozen fp32
operations in a row; with an ALiBi bias of up to |bias| the exponents are rounded at |bias| * 2^-23."""
import pytest
import torch

from _util import qkv

pytestmark = pytest.mark.gpu


def _reference(q, k, v, dout, alibi, mask):
    q, k, v = (t.double().requires_grad_(True) for t in (q, k, v))
    G = q.shape[1] // k.shape[1]
    kk, vv = k.repeat_interleave(G, 1), v.repeat_interleave(G, 1)
    s = q @ kk.transpose(-1, -2) * q.shape[-1] ** -0.5
    qi, ki = torch.arange(q.shape[2], device="cuda")[:, None], torch.arange(k.shape[2], device="cuda")[None, :]
    if alibi:
        h = torch.arange(q.shape[1], device="cuda")[:, None, None]
        s = s + (qi - ki) * torch.exp2(-((h + 1) * 8.0 / q.shape[1])).double()
    if mask is not None:
        s = s.masked_fill(~mask(0, 0, qi, ki), float("-inf"))
    out = torch.softmax(s, -1) @ vv
    return (out.detach(), torch.logsumexp(s, -1).detach()) + torch.autograd.grad(out, (q, k, v), dout.double())


@pytest.mark.parametrize("Hq,Hkv,Sq,Skv,score,mask", [
    (2, 2, 1, 1, None, None), (2, 2, 63, 65, None, None), (2, 1, 64, 128, None, None), (2, 2, 129, 127, "alibi", None),
    (2, 2, 257, 257, "alibi", "causal"), (4, 1, 321, 511, "doubled", "window"), (1, 1, 2048, 2048, None, "causal"),
    (1, 1, 190, 4099, None, None),
])
def test_against_fp64(Hq, Hkv, Sq, Skv, score, mask):
    import flaxattention_b200 as fa
    from flaxattention_b200.masks import causal_mask, generate_sliding_window
    from flaxattention_b200.mods import generate_alibi_bias

    B, D = 2, 64
    q, k, v = (t.cuda() for t in qkv(B, Hq, Hkv, Sq, Skv, D))
    dout = torch.randn(B, Hq, Sq, D, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    m = {None: None, "causal": causal_mask, "window": generate_sliding_window(100)}[mask]
    bm = None if m is None else fa.create_block_mask(m, None, None, Sq, Skv)

    def doubled(score, b, h, q_idx, kv_idx):
        return score * 2.0

    s = {None: None, "alibi": generate_alibi_bias(Hq), "doubled": doubled}[score]
    tq, tk, tv = (t.clone().requires_grad_(True) for t in (q, k, v))
    out, lse = fa.flax_attention(tq, tk, tv, score_mod=s, block_mask=bm, enable_gqa=Hq != Hkv, return_lse=True)
    got = (out.detach(), lse.detach()) + torch.autograd.grad(out, (tq, tk, tv), dout)
    torch.cuda.synchronize()
    fa.check_status()
    want = _reference(q * (2.0 if score == "doubled" else 1.0), k, v, dout, score == "alibi", m)
    bound = 2e-5 + (4 * max(Sq, Skv) * 0.25 * 2.0 ** -23 if score == "alibi" else 0.0)
    for name, a, b in zip(("out", "lse", "dq", "dk", "dv"), got, want):
        if name == "dq" and score == "doubled":
            b = b * 2.0
        fin = torch.isfinite(b)
        assert torch.equal(torch.isfinite(a), fin), name
        assert (a.double() - b)[fin].abs().max().item() <= bound * max(1.0, b[fin].abs().max().item()), name


def test_scores_that_grow_along_the_row():
    """A bias that grows by hundreds from one key tile to the next: the running maximum moves every step."""
    import flaxattention_b200 as fa

    def growing(score, b, h, q_idx, kv_idx):
        return score + kv_idx * 2.0

    q, k, v = (t.cuda() for t in qkv(1, 2, 2, 130, 700, 64))
    out, lse = fa.flax_attention(q, k, v, score_mod=growing, return_lse=True)
    torch.cuda.synchronize()
    s = q.double() @ k.double().transpose(-1, -2) * 0.125 + torch.arange(700, device="cuda") * 2.0
    assert (lse.double() - torch.logsumexp(s, -1)).abs().max().item() <= 1500 * 2.0 ** -22
    # exponents are rounded at 1400 * log2(e) * 2^-24, twice
    assert (out.double() - torch.softmax(s, -1) @ v.double()).abs().max().item() <= 2e-3
