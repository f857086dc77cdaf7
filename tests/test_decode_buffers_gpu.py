"""The general decode kernel with two and with three buffers of K and of V (three where the grid puts at most two CTAs on an SM),
at tile counts around the number of buffers, over table walks of one and of several tiles per block."""
import pytest
import torch

from _util import DTYPES, lse_err, max_abs, qkv
from oracle.attention_oracle import flax_attention_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Skv,block,mask", [(100, 128, None), (129, 128, "offset"), (384, 128, "offset"), (500, 256, "window"),
                                            (640, 256, "offset"), (897, 512, "window")])
@pytest.mark.parametrize("B,Hq,Hkv", [(2, 8, 8), (20, 16, 16), (3, 16, 4)])  # 320 CTAs: two buffers; the others: three
@pytest.mark.parametrize("D,dt,Sq", [(64, "f16", 1), (64, "bf16", 13), (128, "bf16", 2), (128, "f16", 16), (80, "f16", 3)])
def test_two_and_three_buffers(B, Hq, Hkv, D, dt, Sq, Skv, block, mask):
    import flaxattention_b200 as fa
    from flaxattention_b200.masks import generate_causal_offset, generate_sliding_window
    from flaxattention_b200.mods import generate_alibi_bias

    alibi = generate_alibi_bias(Hq)
    m = {None: None, "offset": generate_causal_offset(Skv - Sq), "window": generate_sliding_window(Skv)}[mask]
    q, k, v = qkv(B, Hq, Hkv, Sq, Skv, D, dtype=DTYPES[dt])
    ref, ref_lse = flax_attention_oracle(q, k, v, alibi, m)
    bm = None if m is None else fa.create_block_mask(m, B, 1, Sq, Skv, BLOCK_SIZE=(128, block))
    for splits in (1, 2):
        out, lse = fa.flax_attention(q.cuda(), k.cuda(), v.cuda(), score_mod=alibi, block_mask=bm, enable_gqa=Hq != Hkv, return_lse=True,
                                     kernel_options={"path": "decode", "num_splits": splits, "kernels": "general"})
        assert max_abs(out.cpu(), ref) <= 2e-2
        err, same = lse_err(lse.cpu(), ref_lse)
        assert same and err <= 2e-2 * max(1.0, ref_lse[torch.isfinite(ref_lse)].abs().max().item())
