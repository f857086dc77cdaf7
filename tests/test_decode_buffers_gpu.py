"""The general decode kernel with two and with three buffers of K and of V, by TMA (up to 16 rows, head dim 64 and 128) and by
cp.async, at tile counts around the number of buffers, over table walks of one and of several tiles per block and of half a tile, and
over the strides that the entry points take."""
import pytest
import torch

from _util import DTYPES, lse_err, max_abs, qkv
from oracle.attention_oracle import flax_attention_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Skv,block,mask", [(100, 128, None), (129, 128, "offset"), (384, 128, "offset"), (500, 256, "window"),
                                            (640, 256, "offset"), (897, 512, "window"), (700, 64, "window")])
@pytest.mark.parametrize("B,Hq,Hkv", [(2, 8, 8), (20, 16, 16), (3, 16, 4)])  # (320 CTAs: two buffers; few: three)
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


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["heads inside", "one batch entry for all", "one head for all", "part of a longer row"])
def test_strides(D, kind):
    import flaxattention_b200 as fa

    B, H, Sq, Skv = 3, 4, 5, 777
    q, k, v = (t.cuda() for t in qkv(B, H, H, Sq, Skv, D, dtype=torch.float16))
    if kind == "heads inside":
        k, v = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (k, v))
    elif kind == "one batch entry for all":
        k, v = (t[:1].expand(B, -1, -1, -1) for t in (k, v))
    elif kind == "one head for all":
        k, v = (t[:, :1].expand(-1, H, -1, -1) for t in (k, v))
    else:
        both = torch.cat([k, v], -1)
        k, v = both[..., :D], both[..., D:]
    out, lse = fa.flax_attention(q, k, v, return_lse=True, kernel_options={"path": "decode", "kernels": "general"})
    ref, ref_lse = flax_attention_oracle(q.cpu(), k.cpu().contiguous(), v.cpu().contiguous())
    assert max_abs(out.cpu(), ref) <= 2e-2
    err, same = lse_err(lse.cpu(), ref_lse)
    assert same and err <= 2e-2 * max(1.0, ref_lse.abs().max().item())
    fa.check_status()
