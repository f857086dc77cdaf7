"""GPU parity of the two forms of the 16-bit forward (one or two query tiles per CTA) on both sides of the line
between them: D = 64 up to 2048 keys, no more query tiles than SMs (148), or a BlockMask whose hint says that few tiles are listed, take one.

Tolerance: O and LSE max-abs <= 2e-2 against fp32, the bar of the other forward tests."""
import pytest
import torch

from _util import DTYPES, max_abs

pytestmark = pytest.mark.gpu


def _compare(B, H, Sq, Skv, D, dt, mask, hint):
    import flaxattention_b200 as fa
    from flaxattention_b200.masks import causal_mask, generate_sliding_window

    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(B, H, s, D, generator=g, device="cuda").to(DTYPES[dt]) for s in (Sq, Skv, Skv))
    mod = {None: None, "causal": causal_mask, "window": generate_sliding_window(100),
           "first": lambda b, h, q, kv: ((q // 128) % 2 == 0) & (kv >= q // 2),
           "second": lambda b, h, q, kv: ((q // 128) % 2 == 1) & ((kv < 200) | (kv % 3 == 0)),
           "in turn": lambda b, h, q, kv: (q // 128 + kv // 128) % 2 == 0}[mask]
    bm = None if mod is None else fa.create_block_mask(mod, None, None, Sq, Skv)
    if hint is not None:
        bm._kv_tiles = hint
    out, lse = fa.flax_attention_pallas(q, k, v, block_mask=bm, return_lse=True)
    s = q.float() @ k.float().transpose(-1, -2) * D ** -0.5
    if mod is not None:
        s.masked_fill_(~mod(0, 0, torch.arange(Sq, device="cuda")[:, None], torch.arange(Skv, device="cuda")[None]), float("-inf"))
    ref_lse = torch.logsumexp(s, -1)
    seen = torch.isfinite(ref_lse)
    ref = torch.where(seen[..., None], torch.exp(s - ref_lse.masked_fill(~seen, 0.0)[..., None]) @ v.float(), 0.0)
    assert max_abs(out, ref) <= 2e-2
    assert torch.equal(seen, torch.isfinite(lse)) and max_abs(lse[seen], ref_lse[seen]) <= 2e-2


@pytest.mark.parametrize("B,H,Sq,Skv,D,dt,mask", [
    (1, 2, 128, 2048, 64, "f16", None),      # one: a single tile, the last length of D = 64
    (1, 2, 257, 2049, 64, "bf16", "causal"),  # one: few tiles, ragged on both sides
    (2, 9, 1100, 2049, 64, "bf16", None),    # two: 162 tiles of 2049 keys, the last pair half empty
    (2, 9, 1100, 2300, 64, "f16", "causal"),  # one, by the hint
    (2, 40, 300, 130, 64, "f16", "window"),  # one: more CTAs than fit, rows without a visible tile
    (2, 74, 128, 200, 128, "bf16", None),    # one: 148 tiles
    (1, 149, 128, 200, 128, "bf16", None),   # two: 149 tiles, every second tile of a pair beyond the end
    (4, 20, 200, 700, 128, "f16", "causal"),  # one, by the hint
    (1, 4, 1025, 1025, 128, "bf16", "window"),  # one
])
def test_forward_on_both_sides_of_the_line(B, H, Sq, Skv, D, dt, mask):
    _compare(B, H, Sq, Skv, D, dt, mask, None)


@pytest.mark.parametrize("hint", [1, 65535])
@pytest.mark.parametrize("mask", ["causal", "window", "first", "second", "in turn"])
@pytest.mark.parametrize("B,H,Sq,Skv,D,dt", [
    (2, 9, 1100, 2300, 64, "f16"),   # 162 tiles, the last pair of a head half empty
    (1, 31, 513, 2177, 64, "bf16"),  # 155 tiles, one row in the last
    (2, 26, 300, 700, 128, "f16"),   # 156 tiles, three per head
    (1, 38, 512, 900, 128, "bf16"),  # 152 tiles
])
def test_both_forms_under_tables(B, H, Sq, Skv, D, dt, mask, hint):
    """Steps of the two-tile form in which only one tile of the CTA has a key tile, at the start, at the end or all along, tiles and rows
    without any."""
    _compare(B, H, Sq, Skv, D, dt, mask, hint)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mask", [None, "causal", "window"])
@pytest.mark.parametrize("mod", [None, "alibi"])
@pytest.mark.parametrize("entry", ["flax_attention", "flax_attention_pallas"])  # (scores rounded to the input type, and not)
def test_results_do_not_depend_on_the_form(D, mask, mod, entry):
    """256 tiles take two per CTA where no hint says otherwise, the 128 of one batch entry take one, and the hint decides for
    either (at head dim 64 not with a score_mod under tables, unless scores are rounded): the same bits every time."""
    import flaxattention_b200 as fa
    from flaxattention_b200.masks import causal_mask, generate_sliding_window
    from flaxattention_b200.mods import generate_alibi_bias

    B, H, S = 2, 4, 4096
    g = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = (torch.randn(B, H, S, D, generator=g, device="cuda").bfloat16() for _ in range(3))
    m = {None: None, "causal": causal_mask, "window": generate_sliding_window(300)}[mask]
    bm = None if m is None else fa.create_block_mask(m, None, None, S, S)
    score = None if mod is None else generate_alibi_bias(H)
    results = []
    for hint, n in ((0, B), (0, 1), (1, B), (65535, B)):
        if bm is not None:
            bm._kv_tiles = hint
        results.append(getattr(fa, entry)(q[:n], k[:n], v[:n], score_mod=score, block_mask=bm, return_lse=True))
    for out, lse in results[1:]:
        assert torch.equal(out, results[0][0][:len(out)]) and torch.equal(lse, results[0][1][:len(lse)])
