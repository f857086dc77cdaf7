"""GPU parity of the two forms of the 16-bit forward (one or two query tiles per CTA) on both sides of the line
between them: D = 64 up to 2048 keys, or no more query tiles than SMs (148), take one.

Tolerance: O and LSE max-abs <= 2e-2 against fp32, the bar of the other forward tests."""
import pytest
import torch

from _util import DTYPES, max_abs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Sq,Skv,D,dt,mask", [
    (1, 2, 128, 2048, 64, "f16", None),      # one: a single tile, the last length of D = 64
    (1, 2, 257, 2049, 64, "bf16", "causal"),  # one: few tiles, ragged on both sides
    (2, 9, 1100, 2049, 64, "bf16", None),    # two: 162 tiles of 2049 keys, the last pair half empty
    (2, 9, 1100, 2300, 64, "f16", "causal"),
    (2, 40, 300, 130, 64, "f16", "window"),  # one: more CTAs than fit, rows without a visible tile
    (2, 74, 128, 200, 128, "bf16", None),    # one: 148 tiles
    (1, 149, 128, 200, 128, "bf16", None),   # two: 149 tiles, every second tile of a pair beyond the end
    (4, 20, 200, 700, 128, "f16", "causal"),  # two
    (1, 4, 1025, 1025, 128, "bf16", "window"),  # one
])
def test_forward_on_both_sides_of_the_line(B, H, Sq, Skv, D, dt, mask):
    import flaxattention_b200 as fa
    from flaxattention_b200.masks import causal_mask, generate_sliding_window

    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(B, H, s, D, generator=g, device="cuda").to(DTYPES[dt]) for s in (Sq, Skv, Skv))
    mod = {None: None, "causal": causal_mask, "window": generate_sliding_window(100)}[mask]
    bm = None if mod is None else fa.create_block_mask(mod, None, None, Sq, Skv)
    out, lse = fa.flax_attention_pallas(q, k, v, block_mask=bm, return_lse=True)
    s = q.float() @ k.float().transpose(-1, -2) * D ** -0.5
    if mod is not None:
        s.masked_fill_(~mod(0, 0, torch.arange(Sq, device="cuda")[:, None], torch.arange(Skv, device="cuda")[None]), float("-inf"))
    ref_lse = torch.logsumexp(s, -1)
    seen = torch.isfinite(ref_lse)
    ref = torch.where(seen[..., None], torch.exp(s - ref_lse.masked_fill(~seen, 0.0)[..., None]) @ v.float(), 0.0)
    assert max_abs(out, ref) <= 2e-2
    assert torch.equal(seen, torch.isfinite(lse)) and max_abs(lse[seen], ref_lse[seen]) <= 2e-2


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mask", ["causal", "window"])
@pytest.mark.parametrize("mod", [None, "alibi"])
def test_results_do_not_depend_on_the_form(D, mask, mod):
    """256 tiles take two per CTA where no hint says otherwise, the 128 of one batch entry take one, and the hint decides for
    either: the same bits every time."""
    import flaxattention_b200 as fa
    from flaxattention_b200.masks import causal_mask, generate_sliding_window
    from flaxattention_b200.mods import generate_alibi_bias

    B, H, S = 2, 4, 4096
    g = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = (torch.randn(B, H, S, D, generator=g, device="cuda").bfloat16() for _ in range(3))
    bm = fa.create_block_mask(causal_mask if mask == "causal" else generate_sliding_window(300), None, None, S, S)
    score = None if mod is None else generate_alibi_bias(H)
    results = []
    for hint, n in ((0, B), (0, 1), (1, B), (65535, B)):
        bm._kv_tiles = hint
        results.append(fa.flax_attention_pallas(q[:n], k[:n], v[:n], score_mod=score, block_mask=bm, return_lse=True))
    for out, lse in results[1:]:
        assert torch.equal(out, results[0][0][:len(out)]) and torch.equal(lse, results[0][1][:len(lse)])
