"""The one-evaluation mask construction (fa_mask_scan_kernel) at the edges of its 128 x 128 sub-tiles and
32-bit words: tables and both bit matrices against the CPU oracle, and bit matrices over captured
tensors that change after they were built."""
import numpy as np
import pytest
import torch

from cases import TABLE_KEYS, head_dependent
from oracle.blockmask_oracle import create_block_mask_oracle

pytestmark = pytest.mark.gpu


def _unpack(bits, n):
    a = bits.cpu().numpy().view(np.uint32)
    return ((a[..., None] >> np.arange(32, dtype=np.uint32)) & 1).astype(bool).reshape(*a.shape[:-1], -1)[..., :n]


@pytest.mark.parametrize("Q,KV,block", [
    (1, 32, (128, 32)), (50, 192, (64, 64)), (127, 512, (128, 128)), (128, 128, (128, 128)), (192, 320, (96, 160)),
    (256, 384, (32, 384)), (512, 640, (256, 64)), (384, 288, (128, 288)), (130, 200, (130, 100)),
])
def test_tables_and_bits_at_word_and_tile_edges(Q, KV, block):
    import flaxattention_b200 as fa

    B, H = 2, 3
    whole_words = block[1] % 32 == 0 or KV <= block[1]
    bm = fa.create_block_mask(head_dependent, B, H, Q, KV, BLOCK_SIZE=block)
    torch.cuda.synchronize()
    want = create_block_mask_oracle(head_dependent, B, H, Q, KV, BLOCK_SIZE=block)
    for k in TABLE_KEYS:
        assert np.array_equal(getattr(bm, k).cpu().numpy(), want[k]), k
    assert (bm.mask_bits is not None) == whole_words
    if whole_words:
        q, kv = np.arange(Q)[:, None], np.arange(KV)[None, :]
        for b in range(B):
            for h in range(H):
                dense = head_dependent(b, h, q, kv)
                assert np.array_equal(_unpack(bm.mask_bits, KV)[b, h][:Q], dense)
                assert np.array_equal(_unpack(bm.mask_bits_t, Q)[b, h][:KV], dense.T)


def test_bits_over_a_captured_tensor_are_dropped_when_it_changes():
    """The tables keep what they were built from; on the partial tiles the mask is evaluated again."""
    import flaxattention_b200 as fa

    S = 256
    limit = torch.full((S,), 200, dtype=torch.int32, device="cuda")

    def up_to_limit(b, h, q_idx, kv_idx):
        return kv_idx < limit[q_idx]

    q, k, v = (torch.randn(1, 2, S, 64, device="cuda", dtype=torch.float16) for _ in range(3))
    bm = fa.create_block_mask(up_to_limit, None, None, S, S)
    assert bm.bits_hold() and bm.mask_bits_t is not None
    fa.flax_attention(q, k, v, block_mask=bm)
    limit.fill_(150)  # the second key block is still partial
    assert not bm.bits_hold()
    got = fa.flax_attention(q, k, v, block_mask=bm)
    fresh = fa.flax_attention(q, k, v, block_mask=fa.create_block_mask(up_to_limit, None, None, S, S))
    assert torch.equal(got, fresh)


def test_the_size_limit_counts_both_matrices(monkeypatch):
    """256 x 256: 8 KiB row-major and as much transposed."""
    import flaxattention_b200 as fa
    from flaxattention_b200 import blockmask
    from flaxattention_b200.masks import causal_mask

    for limit, row_major, transposed in ((8191, False, False), (8192, True, False), (16383, True, False), (16384, True, True)):
        monkeypatch.setattr(blockmask, "_MASK_BITS_MAX_BYTES", limit)
        bm = fa.create_block_mask(causal_mask, None, None, 256, 256)
        assert (bm.mask_bits is not None, bm.mask_bits_t is not None) == (row_major, transposed)
        q, k, v = (torch.randn(1, 2, 256, 64, device="cuda").requires_grad_(True) for _ in range(3))
        plain = fa.create_block_mask(causal_mask, None, None, 256, 256, _mask_bits=False)
        grads = [torch.autograd.grad(fa.flax_attention(q, k, v, block_mask=m).sum(), (k, v)) for m in (bm, plain)]
        assert all(torch.equal(a, b) for a, b in zip(*grads))


@pytest.mark.parametrize("Q,KV,block", [(96, 96, (48, 48)), (192, 200, (64, 50)), (130, 300, (26, 100))])
def test_bits_asked_for_beside_blocks_of_part_words(Q, KV, block):
    import flaxattention_b200 as fa

    bm = fa.create_block_mask(head_dependent, 1, 3, Q, KV, BLOCK_SIZE=block, _mask_bits=True)
    want = create_block_mask_oracle(head_dependent, 1, 3, Q, KV, BLOCK_SIZE=block)
    for k in TABLE_KEYS:
        assert np.array_equal(getattr(bm, k).cpu().numpy(), want[k]), k
    q, kv = np.arange(Q)[:, None], np.arange(KV)[None, :]
    for h in range(3):
        dense = head_dependent(0, h, q, kv)
        assert np.array_equal(_unpack(bm.mask_bits, KV)[0, h][:Q], dense)
        assert np.array_equal(_unpack(bm.mask_bits_t, Q)[0, h][:KV], dense.T)


@pytest.mark.parametrize("Q,KV,block", [(1, 300, 128), (31, 256, 128), (64, 160, (64, 32)), (128, 384, 128), (300, 500, 128), (256, 256, 256)])
@pytest.mark.parametrize("name", ["key", "query", "in_part", "all_but_one"])
def test_positions_decided_by_range_and_by_evaluation(name, Q, KV, block):
    """Masks over captured ids: per key, per query, with groups of 32 keys that interval arithmetic decides between others that it
    does not, and with one position that differs from all others."""
    import flaxattention_b200 as fa

    ids = torch.arange(1024, device="cuda", dtype=torch.int32) // 37
    host = ids.cpu().numpy()
    mod = {
        "key": lambda b, h, q, kv: kv < ids[kv] * 40 + 5,
        "query": lambda b, h, q, kv: kv < ids[q] * 40 + 5,
        "in_part": lambda b, h, q, kv: (kv < 70) | ((ids[q] == ids[kv]) & (kv < 190)),
        "all_but_one": lambda b, h, q, kv: (q != 30) | (kv != 100),
    }[name]
    q, kv = np.arange(Q)[:, None], np.arange(KV)[None, :]
    dense = {"key": kv < host[kv] * 40 + 5, "query": kv < host[q] * 40 + 5,
             "in_part": (kv < 70) | ((host[q] == host[kv]) & (kv < 190)), "all_but_one": (q != 30) | (kv != 100)}[name]
    dense = np.broadcast_to(dense, (Q, KV))
    bm = fa.create_block_mask(mod, None, None, Q, KV, BLOCK_SIZE=block)
    torch.cuda.synchronize()
    assert np.array_equal(_unpack(bm.mask_bits, KV)[0, 0][:Q], dense)
    assert np.array_equal(_unpack(bm.mask_bits_t, Q)[0, 0][:KV], dense.T)


@pytest.mark.parametrize("reads", ["nothing", "batch", "head", "both"])
def test_entries_that_share_their_rows(reads):
    """A warp of the table kernel writes one distinct row to several entries, and what is left of them at the end: 13 x 61 entries of
    5 x 7 blocks, four to a warp (793, 61 and 13 are one more than a multiple).  The mask keeps and drops whole 128 x 128 blocks,
    with ragged ones at both ends."""
    import flaxattention_b200 as fa

    B, H, Q, KV = 13, 61, 600, 860
    n = {"nothing": lambda b, h: 0, "batch": lambda b, h: b, "head": lambda b, h: h, "both": lambda b, h: b + h}[reads]
    mod = lambda b, h, q, kv: (kv < 128) | ((q + 40 >= kv) & (q < kv + 300 + 7 * n(b, h)))  # noqa: E731
    bm = fa.create_block_mask(mod, B, H, Q, KV)
    torch.cuda.synchronize()
    nQ, nKV = 5, 7
    q, kv = np.arange(Q)[:, None], np.arange(KV)[None, :]
    kinds = {}
    tables = {k: getattr(bm, k).cpu().numpy() for k in TABLE_KEYS}
    # (the bits of 793 distinct masks are beyond the size that is kept without being asked for)
    bits = None if reads == "both" else (_unpack(bm.mask_bits, KV), _unpack(bm.mask_bits_t, Q))
    for b in range(B):
        for h in range(H):
            i = int(n(b, h))
            if i not in kinds:
                dense = np.broadcast_to(mod(b, h, q, kv), (Q, KV))
                want = create_block_mask_oracle(lambda _b, _h, q, kv, b=b, h=h: mod(b, h, q, kv), 1, 1, Q, KV)
                kinds[i] = dense, want
                if bits is not None:
                    at = min(b, bits[0].shape[0] - 1), min(h, bits[0].shape[1] - 1)
                    assert np.array_equal(bits[0][at][:Q], dense) and np.array_equal(bits[1][at][:KV], dense.T)
            for k in TABLE_KEYS:
                assert np.array_equal(tables[k][b, h], kinds[i][1][k][0, 0]), (k, b, h)
    assert tables["kv_indices"].shape[-2:] == (nQ, nKV)
