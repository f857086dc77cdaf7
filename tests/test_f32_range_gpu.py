"""fp32 inputs of head dim 64 with values that have no bf16 parts (infinities, NaN) or whose products leave the range
of the partial products: the heads with such a value take the fp32 kernels, behind the tensor-core ones, and
give what these give; the other heads are not touched, unless they share a group of 32 rows with one (short
sequences).  2^30 is the bound: one below it keeps the parts."""
import pytest
import torch

from _util import qkv

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def _run(q, k, v, do, options, **kw):
    import flaxattention_b200 as fa

    ts = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out, lse = fa.flax_attention(*ts, return_lse=True, enable_gqa=q.shape[1] != k.shape[1], kernel_options=options, **kw)
    return [out.detach(), lse.detach(), *torch.autograd.grad(out, ts, do)]


@pytest.mark.parametrize("where,value", [
    ("v", INF), ("v", 3.395e38), ("v", NAN), ("q", INF), ("q", -1e30), ("q", NAN), ("k", -INF), ("k", 3.4e38), ("do", INF),
    ("do", -2.0 ** 30),
])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,mask", [(2, 2, 2, 300, 300, None), (1, 4, 2, 129, 77, None), (2, 2, 1, 257, 257, "causal"),
                                                  (1, 2, 2, 1, 33, None)])
def test_values_beyond_the_parts(where, value, B, Hq, Hkv, Sq, Skv, mask):
    import flaxattention_b200 as fa
    from flaxattention_b200.masks import causal_mask

    bm = fa.create_block_mask(causal_mask, None, None, Sq, Skv) if mask else None
    q, k, v = (t.cuda() for t in qkv(B, Hq, Hkv, Sq, Skv, 64))
    do = torch.randn(B, Hq, Sq, 64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    clean = _run(q, k, v, do, None, block_mask=bm)
    t = {"q": q, "k": k, "v": v, "do": do}[where]
    head = t.shape[1] - 1
    t[B - 1, head, t.shape[2] // 2, 63] = value
    want = _run(q, k, v, do, {"kernels": "general"}, block_mask=bm)
    G = Hq // Hkv
    kv = head // G if where in ("q", "do") else head  # the kv head the value belongs to
    for options in (None, {}):  # the native call and the Python one
        got = _run(q, k, v, do, options, block_mask=bm)
        for name, a, b, c in zip(("out", "lse", "dq", "dk", "dv"), got, want, clean):
            hit = slice(kv, kv + 1) if name in ("dk", "dv") else slice(kv * G, kv * G + G)
            x, y = a[B - 1, hit], b[B - 1, hit]
            if name in ("out", "lse"):  # every head decides for itself, and dO has no say
                hit = slice(head, head + 1) if where == "q" else slice(0, 0) if where == "do" else hit
                x, y = a[B - 1, hit], b[B - 1, hit]
                assert torch.equal(torch.nan_to_num(x, 7.0), torch.nan_to_num(y, 7.0)), name
            if name == "dq" and value == 3.4e38:
                continue  # (dP - delta) * k: what is left of dP - delta after rounding, times 3.4e38
            fin = torch.isfinite(y)
            assert torch.equal(torch.isnan(x), torch.isnan(y)) and torch.equal(torch.isfinite(x), fin), name
            assert torch.equal(x[~fin & ~torch.isnan(y)], y[~fin & ~torch.isnan(y)]), name
            # the same kernels; delta is summed in another order (64 products)
            assert (x - y)[fin].abs().max().item() <= 1e-5 * max(1.0, y[fin].abs().max().item()) if fin.any() else True, name
            others = torch.ones_like(a, dtype=torch.bool)
            others[B - 1, hit] = False
            # (dq: no fixed order over the kv tiles; short sequences: see above)
            tol = 1e-5 * max(1.0, c.abs()[torch.isfinite(c)].max().item()) if name == "dq" or Sq < 32 else 0.0
            assert (a - c)[others].abs().max().item() <= tol if others.any() else True, name


def test_the_largest_values_that_keep_the_parts():
    """Just below 2^30: no fp32 kernel runs, and the result is that of the parts, against fp64."""
    q, k, v = (t.cuda() for t in qkv(1, 2, 2, 130, 130, 64))
    do = torch.randn(1, 2, 130, 64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    v[0, 0, 5, :] = 2.0 ** 30 * (1 - 2.0 ** -24)
    got = _run(q, k, v, do, None)
    want = torch.softmax(q.double() @ k.double().transpose(-1, -2) * 0.125, -1) @ v.double()
    assert (got[0].double() - want).abs().max().item() <= 2e-5 * want.abs().max().item()
    assert not torch.equal(got[0][0, 0], _run(q, k, v, do, {"kernels": "general"})[0][0, 0])


@pytest.mark.parametrize("Sq,Skv", [(64, 64), (1, 1), (300, 64), (64, 65), (1, 65)])
def test_the_forward_up_to_one_tile_of_keys(Sq, Skv):
    """Up to 64 keys the forward is the fp32 kernel; the results agree on both sides (fp64, as in test_f32_tensor_core_gpu)."""
    q, k, v = (t.cuda() for t in qkv(2, 2, 2, Sq, Skv, 64))
    do = torch.randn(2, 2, Sq, 64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    got, general = _run(q, k, v, do, None), _run(q, k, v, do, {"kernels": "general"})
    assert torch.equal(got[0], general[0]) == (Skv <= 64)
    want = torch.softmax(q.double() @ k.double().transpose(-1, -2) * 0.125, -1) @ v.double()
    assert (got[0].double() - want).abs().max().item() <= 2e-5


@pytest.mark.parametrize("path", ["native", "python", "pipeline"])
def test_gradients_are_the_same_every_time_when_asked_for(path):
    import flaxattention_b200 as fa

    B, H, S = 2, 4, 1024
    q, k, v = (t.cuda() for t in qkv(B, H, H, S, S, 64))
    do = torch.randn(B, H, S, 64, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    if path == "pipeline":
        host = [t.cpu().pin_memory() for t in (q, k, v)]
        res = [torch.empty(B, H, S, 64).pin_memory() for _ in range(4)]
        hdo = do.cpu().pin_memory()
        pipe = fa.HostPipeline(B, H, H, S, S, 64, dtype=torch.float32)

        def grads():
            pipe.step(*host, *res, hdo)
            torch.cuda.synchronize()
            return [t.clone().cuda() for t in res[1:]]
    else:
        options = None if path == "native" else {}
        ts = [t.clone().requires_grad_(True) for t in (q, k, v)]
        for _ in range(2):
            out = fa.flax_attention_pallas(*ts) if path == "native" else fa.flax_attention(*ts, kernel_options=options)

        def grads():
            return torch.autograd.grad(out, ts, do, retain_graph=True)

    usual = grads()
    torch.use_deterministic_algorithms(True)
    try:
        several = [grads() for _ in range(6)]
    finally:
        torch.use_deterministic_algorithms(False)
    for g in several[1:]:
        assert all(torch.equal(a, b) for a, b in zip(g, several[0]))
    for a, b in zip(usual, several[0]):
        assert (a - b).abs().max().item() <= 2e-5 * max(1.0, b.abs().max().item())  # (as in test_f32_tensor_core_gpu)


@pytest.mark.parametrize("options", [None, {}])
def test_without_room_for_the_parts(options):
    """Forward and gradients fit where inputs and results do, as with the kernels that need no parts."""
    import flaxattention_b200 as fa

    H, S, MB = 8, 8192, 1 << 20  # 16 MiB a tensor; the parts take 72 and 96 MiB
    q, k, v, do = (torch.randn(1, H, S, 64, device="cuda") for _ in range(4))
    ts = [t.requires_grad_(True) for t in (q, k, v)]
    small = [t[:, :, :256].detach().requires_grad_(True) for t in ts]
    for o in (options, {"kernels": "general"}):
        for _ in range(2):  # (compiled, loaded and registered)
            torch.autograd.grad(fa.flax_attention(*small, kernel_options=o).sum(), small)
    total = torch.cuda.get_device_properties(0).total_memory

    def limit(room):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room * MB) / total)

    try:
        limit(40)
        out = fa.flax_attention(*ts, kernel_options=options)
        limit(80)
        got = torch.autograd.grad(out, ts, do)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    ref = fa.flax_attention(*ts, kernel_options={"kernels": "general"})
    assert torch.equal(out, ref)
    assert all(torch.equal(a, b) for a, b in zip(got, torch.autograd.grad(ref, ts, do)))
