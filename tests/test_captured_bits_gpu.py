"""Bit matrices over captured tensors (BlockMask.mask_bits) against the mask evaluated in place, after writes
that a tensor's version counter does not show.  The matrix and the evaluation select the same scores, so
the results are compared bit for bit (dQ, whose sums have no fixed order, by its norm)."""
import pytest
import torch

from _util import rel_err

pytestmark = pytest.mark.gpu
S = 256


def _problem(dtype):
    limit = torch.full((S,), 200, dtype=torch.int32, device="cuda")

    def up_to_limit(b, h, q_idx, kv_idx):
        return kv_idx < limit[q_idx]

    g = torch.Generator("cuda").manual_seed(1)
    q, k, v, do = (torch.randn(1, 2, S, 64, device="cuda", generator=g).to(dtype) for _ in range(4))
    return limit, up_to_limit, q, k, v, do


def _by_data(limit):
    limit.data.fill_(150)


def _by_alias(limit):
    torch.from_dlpack(torch.utils.dlpack.to_dlpack(limit)).fill_(150)


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("options", [None, {}])  # the native call and the Python one
@pytest.mark.parametrize("write", [_by_data, _by_alias])
def test_a_write_behind_the_version_counter_is_seen(dtype, options, write):
    import flaxattention_b200 as fa

    limit, mask, q, k, v, do = _problem(dtype)
    bm = fa.create_block_mask(mask, None, None, S, S)
    plain = fa.create_block_mask(mask, None, None, S, S, _mask_bits=False)
    assert bm.mask_bits is not None and plain.mask_bits is None
    for change in (False, True):
        if change:
            write(limit)
            assert bm.bits_hold()  # what the host can see
        res = []
        for m in (bm, plain, bm):
            ts = [t.clone().requires_grad_(True) for t in (q, k, v)]
            out = fa.flax_attention(*ts, block_mask=m, kernel_options=options)
            res.append((out.detach(), *torch.autograd.grad(out, ts, do)))
        for got in (res[0], res[2]):
            assert torch.equal(got[0], res[1][0]) and torch.equal(got[2], res[1][2]) and torch.equal(got[3], res[1][3])
            assert rel_err(got[1], res[1][1]) <= (1e-6 if dtype == torch.float32 else 1e-3)


def test_a_change_between_forward_and_backward_is_seen():
    import flaxattention_b200 as fa

    limit, mask, q, k, v, do = _problem(torch.float32)
    res = []
    for bits in (None, False):
        limit.fill_(200)
        bm = fa.create_block_mask(mask, None, None, S, S, _mask_bits=bits)
        for _ in range(2):  # the second call is taken natively
            limit.data.fill_(200)
            ts = [t.clone().requires_grad_(True) for t in (q, k, v)]
            out = fa.flax_attention(*ts, block_mask=bm)
            limit.data.fill_(150)
            res.append(torch.autograd.grad(out, ts, do)[1:])
    assert all(torch.equal(a, b) for r in res[1:] for a, b in zip(r, res[0]))


def test_a_replayed_graph_sees_the_contents_of_its_time():
    import flaxattention_b200 as fa

    limit, mask, q, k, v, _ = _problem(torch.bfloat16)
    bm = fa.create_block_mask(mask, None, None, S, S)
    for _ in range(2):
        fa.flax_attention(q, k, v, block_mask=bm)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fa.flax_attention(q, k, v, block_mask=bm)
    for n in (200, 150, 200):
        limit.fill_(n)
        graph.replay()
        want = fa.flax_attention(q, k, v, block_mask=fa.create_block_mask(mask, None, None, S, S, _mask_bits=False))
        assert torch.equal(out, want)


def test_the_host_pipeline_sees_a_change():
    import flaxattention_b200 as fa

    limit, mask, q, k, v, _ = _problem(torch.float16)
    bm = fa.create_block_mask(mask, None, None, S, S)
    pipe = fa.HostPipeline(1, 2, 2, S, S, 64, block_mask=bm, backward=False)
    hq, hk, hv = (t.cpu().pin_memory() for t in (q, k, v))
    ho = torch.empty_like(hq).pin_memory()
    for n in (200, 150):
        limit.fill_(n)
        pipe.step(hq, hk, hv, ho)
        torch.cuda.synchronize()
        assert torch.equal(ho.cuda(), fa.flax_attention_pallas(q, k, v, block_mask=bm))


@pytest.mark.parametrize("n,dtype", [(1, torch.uint8), (15, torch.uint8), (17, torch.uint8), (1, torch.int64), (4100, torch.int32),
                                     (9000, torch.float32)])
@pytest.mark.parametrize("offset", [0, 1, 4])
def test_snapshot_of_any_length_and_alignment(n, dtype, offset):
    """One changed byte, at either end or in the middle, is found; nothing outside the ranges is looked at."""
    from flaxattention_b200 import _cabi

    L = _cabi.lib()
    base = torch.randint(0, 100, (n + offset + 1,), device="cuda").to(dtype)
    other = torch.randint(0, 100, (33,), device="cuda").to(torch.int32)
    t = base[offset:offset + n]
    addr, size, count = _cabi.ranges([t, other])
    snap = torch.empty(L.fa_snapshot_bytes(size, count), dtype=torch.uint8, device="cuda")
    holds = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def check():
        _cabi.check(L.fa_snapshot_holds(addr, size, count, snap.data_ptr(), holds.data_ptr(), stream))
        return holds.item()

    _cabi.check(L.fa_snapshot(addr, size, count, snap.data_ptr(), stream))
    assert check() == 1
    base[offset + n] += 1
    if offset:
        base[offset - 1] += 1
    assert check() == 1
    for where in {0, n // 2, n - 1}:
        t[where] += 1
        assert check() == 0
        t[where] -= 1
        assert check() == 1
    other[32] += 1
    assert check() == 0
