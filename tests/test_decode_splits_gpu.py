"""The merge of decode splits: inside a thread-block cluster (up to 8 splits that are resident together) and through
memory with the combine kernel (more), over head dims where a row's columns fill part of a warp, a warp, or
more, with packed heads, and with splits that hold no visible key.

Bound: the merge is fp32 (relative error a few 2^-24 per split), but each split rounds its probabilities to fp16 under its own
running maximum: 2^-11 relative on either side, so the results differ from those of one split by at most 2^-10 max|v| and half
a unit in the last place of each (2^-10 relative); lse, whose sums are not rounded, by 1e-5."""
import pytest
import torch

from _util import lse_err, qkv
from oracle.attention_oracle import flax_attention_oracle

pytestmark = pytest.mark.gpu


def _run(q, k, v, mask, splits):
    import flaxattention_b200 as fa

    bm = fa.create_block_mask(mask, None, None, q.shape[2], k.shape[2]) if mask is not None else None
    out, lse = fa.flax_attention(q.cuda(), k.cuda(), v.cuda(), block_mask=bm, enable_gqa=q.shape[1] != k.shape[1], return_lse=True,
                                 kernel_options={"path": "decode", "kernels": "general", "num_splits": splits, "round_scores": False})
    torch.cuda.synchronize()
    return out.cpu(), lse.cpu()


@pytest.mark.parametrize("Hq,Hkv,Sq,Skv,D,Dv,mask", [
    (3, 3, 1, 2048, 64, 64, None),
    (8, 2, 2, 1111, 128, 128, None),        # packed heads, ragged
    (2, 2, 16, 1024, 128, 48, "literal"),   # twelve groups of four columns; only the first split sees keys
    (2, 2, 33, 900, 64, 16, None),          # three row groups
    (1, 1, 5, 2000, 256, 144, "window"),    # columns beyond 128, splits without visible keys
    (1, 1, 64, 1500, 256, 256, None),
])
@pytest.mark.parametrize("splits", [2, 3, 8, 9, 33, 70])
def test_splits_give_the_result_of_one(Hq, Hkv, Sq, Skv, D, Dv, mask, splits):
    from flaxattention_b200.masks import causal_mask, generate_sliding_window

    q, k, v = qkv(2, Hq, Hkv, Sq, Skv, D, Dv, dtype=torch.float16)
    m = {None: None, "literal": causal_mask, "window": generate_sliding_window(700)}[mask]
    one, lse1 = _run(q, k, v, m, 1)
    out, lse = _run(q, k, v, m, splits)
    assert not torch.isnan(out.float()).any()
    err = (out.double() - one.double()).abs()
    assert (err <= 2.0 ** -10 * (v.abs().max().item() + one.double().abs())).all(), err.max()
    e, same = lse_err(lse, lse1)
    assert same and e <= 1e-5 * max(1.0, lse1[torch.isfinite(lse1)].abs().max().item())


def test_many_splits_match_the_oracle():
    q, k, v = qkv(1, 2, 2, 3, 4096, 64, dtype=torch.bfloat16)
    out, lse = _run(q, k, v, None, 32)
    ref, ref_lse = flax_attention_oracle(q.float(), k.float(), v.float())
    assert (out.double() - ref.double()).abs().max().item() <= 2e-2
    assert lse_err(lse, ref_lse)[0] <= 1e-4


@pytest.mark.parametrize("Hq,Hkv,Sq,Skv,D,Dv", [
    (3, 3, 1, 2000, 64, 64),
    (8, 2, 2, 1111, 128, 128),   # eight rows of a packed tile: the second part lies over all eight spare rows
    (2, 2, 9, 1024, 128, 48),    # the first that takes a second instruction
    (4, 1, 4, 900, 64, 16),      # the last, four heads to a tile
    (2, 2, 16, 1100, 64, 64),
    (1, 1, 5, 1500, 256, 256),
])
@pytest.mark.parametrize("splits", [1, 2, 9])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_up_to_16_rows_lose_no_more_than_the_output_rounds(Hq, Hkv, Sq, Skv, D, Dv, splits, dt):
    """Against 64 bits of the same inputs.  Bound: half a unit in the last place of the result, and of the sum a part of
    max|v|: what two parts leave of a probability (2^-17 bf16, 2^-23 fp16, relative), and exponential and fp32 sums (2^-22 and
    at most 2^-19 over up to 30 steps of 16 keys in a warp and 16 merges).  Probabilities of one part miss it."""
    q, k, v = qkv(2, Hq, Hkv, Sq, Skv, D, Dv, dtype=dt)
    out, _ = _run(q, k, v, None, splits)
    G = Hq // Hkv
    kd, vd = (t.double().repeat_interleave(G, 1) for t in (k, v))
    ref = torch.softmax(q.double() @ kd.transpose(-1, -2) * D ** -0.5, -1) @ vd
    bf16 = dt == torch.bfloat16
    half = torch.ldexp(torch.ones_like(ref), torch.frexp(ref).exponent - (9 if bf16 else 12)).clamp(min=0.0 if bf16 else 2.0 ** -25)
    over = ((out.double() - ref).abs() - half).max().item()
    assert over <= (2.0 ** -17 + 2.0 ** -18 if bf16 else 2.0 ** -18) * v.double().abs().max().item()
