"""The bit matrices of a mask that reads the batch or head index belong to the entries they were made for: a call over others
(a broadcast mask over several heads, another offset) evaluates mask_mod, as it does without matrices."""
import pytest
import torch


def by_head(b, h, q, kv):
    return kv <= q + 40 * h


def _mask(B, H, at):
    from flaxattention_b200.blockmask import BlockMask

    z = torch.zeros(B, H, 4, 4, dtype=torch.int32)
    n = torch.zeros(B, H, 4, dtype=torch.int32)
    bits = torch.arange(B * H, dtype=torch.int32).view(B, H, 1, 1).expand(B, H, 512, 16).contiguous()
    return BlockMask(n, z, n, z, n, z, n, z, (128, 128), by_head, bits, bits, _bits_at=at)


def test_entries_of_other_indices_are_not_covered():
    free = _mask(1, 1, (None, None))
    assert free.bits_cover(3, 4, 0, 0) and free.bits_cover(3, 4, 5, 6)
    one = _mask(1, 1, (None, 0))  # made for head 0
    assert one.bits_cover(3, 1, 7, 0) and not one.bits_cover(3, 4, 0, 0) and not one.bits_cover(3, 1, 0, 2)
    four = _mask(1, 4, (None, 8))
    assert four.bits_cover(2, 4, 0, 8) and not four.bits_cover(2, 4, 0, 0) and not four.bits_cover(2, 2, 0, 8)


def test_a_shard_has_the_entries_of_its_heads():
    m = _mask(1, 4, (None, 8)).shard(slice(0, 2), slice(2, 4))
    assert m.bits_cover(2, 2, 0, 10) and not m.bits_cover(2, 2, 0, 8)
    assert m.mask_bits[0, :, 0, 0].tolist() == [2, 3]
    whole = _mask(1, 1, (None, 0)).shard(slice(0, 2), slice(2, 4))  # (a broadcast axis is kept whole)
    assert not whole.bits_cover(2, 2, 0, 2)
    both = _mask(2, 4, (3, 0)).shard(slice(1, 2), slice(None))
    assert both.bits_cover(1, 4, 4, 0) and both.to("cpu").bits_cover(1, 4, 4, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("H,h_offset", [(None, 0), (4, 0), (4, 3), (None, 2)])
@pytest.mark.parametrize("options", [None, {"path": "fwd"}])  # (options: through the Python layer)
@pytest.mark.parametrize("D,dt", [(64, torch.bfloat16), (128, torch.bfloat16), (64, torch.float32)])
def test_results_are_those_without_matrices(D, dt, options, H, h_offset):
    import flaxattention_b200 as fa

    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = (torch.randn(1, 4, 384, D, generator=g, device="cuda").to(dt) for _ in range(4))
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    got = []
    for bits in (None, False):
        bm = fa.create_block_mask(by_head, None, H, 384, 384, _mask_bits=bits)
        assert (bm.mask_bits is not None) == (bits is None)
        out, lse = fa.flax_attention(q, k, v, block_mask=bm, return_lse=True, kernel_options=options, h_offset=h_offset)
        got.append((out, lse, *torch.autograd.grad(out, (k, v), do)))
    for a, b in zip(*got):
        assert torch.equal(a, b)
