"""The native host path of the entry points (csrc/host.cpp) against the Python layer: which calls it takes, and that
a call is answered alike on both.  The first call with a pair of mods goes through the Python layer, later ones are
taken natively; ``kernel_options={}`` always goes through Python."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(B=1, Hq=2, Hkv=2, S=256, dtype=torch.float16, layout="bhsd"):
    g = torch.Generator("cuda").manual_seed(3)

    def mk(H):
        shape = (B, H, S, 64) if layout == "bhsd" else (B, S, H, 64)
        return torch.randn(shape, device="cuda", generator=g).to(dtype)

    return mk(Hq), mk(Hkv), mk(Hkv), mk(Hq)


def _fresh_mod():
    return lambda score, b, h, q_idx, kv_idx: score * 1.5


@pytest.mark.parametrize("flag", [True, 1, np.True_, "yes", False, 0, np.False_, None, ""])
@pytest.mark.parametrize("entry", ["flax", "pallas"])
def test_return_lse_takes_any_truth_value(flag, entry):
    import flaxattention_b200 as fa

    q, k, v, _ = _inputs()
    f = fa.flax_attention if entry == "flax" else fa.flax_attention_pallas
    mod = _fresh_mod()
    first, second = (f(q, k, v, score_mod=mod, return_lse=flag) for _ in range(2))
    assert isinstance(first, tuple) == isinstance(second, tuple) == bool(flag)
    for a, b in zip(first, second) if flag else [(first, second)]:
        assert torch.equal(a, b)


@pytest.mark.parametrize("gqa", [True, 1, np.True_])
@pytest.mark.parametrize("layout", ["bhsd", "bshd"])
@pytest.mark.parametrize("strided", [False, True])
def test_both_layers_give_the_same(gqa, layout, strided):
    """Grouped heads, both layouts, strided inputs, with gradients: native call against the Python layer's first one."""
    import flaxattention_b200 as fa

    q, k, v, do = _inputs(2, 4, 2, 200, torch.bfloat16, layout)
    if strided:
        q, k, v = (torch.cat((t, t), -2)[..., :t.shape[-2], :] for t in (q, k, v))
        assert not q.is_contiguous()
    mod, res = _fresh_mod(), []
    for _ in range(2):
        ts = [t.detach().requires_grad_(True) for t in (q, k, v)]
        out, lse = fa.flax_attention_pallas(*ts, score_mod=mod, enable_gqa=gqa, bhln=layout == "bhsd", return_lse=True)
        res.append((out.detach(), lse, *torch.autograd.grad(out, ts, do)))
        assert not lse.requires_grad
    for i, (a, b) in enumerate(zip(*res)):
        if i == 2:  # dQ: no fixed order of the sums over the kv tiles
            assert (a.float() - b.float()).norm() <= 1e-2 * b.float().norm()
        else:
            assert torch.equal(a, b)


def _dual(f, q):
    import torch.autograd.forward_ad as ad

    with ad.dual_level():
        f(ad.make_dual(q.clone().requires_grad_(True), torch.ones_like(q)))


def _dispatch_mode(f, q):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Mode():
        f(q)


def _in_vmap(f, q):
    w = q.clone().requires_grad_(True)
    torch.func.vmap(lambda x: f(w).float().sum() + x)(torch.ones(3, device="cuda"))


@pytest.mark.parametrize("where,python,refused", [
    (lambda f, q: f(q), False, None),
    (_dual, True, NotImplementedError),
    (lambda f, q: torch.jit.trace(f, (q,), check_trace=False), True, Exception),  # (whether a trace of it succeeds is left open)
    (_dispatch_mode, True, None),
    (_in_vmap, True, RuntimeError),
    (lambda f, q: torch.func.grad(lambda x: f(x).float().sum())(q), True, RuntimeError),
    (lambda f, q: torch.func.vmap(f)(q[None]), True, RuntimeError),
], ids=["plain", "dual", "jit", "mode", "in_vmap", "func_grad", "vmap"])
@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
def test_calls_that_are_watched_go_through_the_python_layer(where, python, refused, monkeypatch):
    import flaxattention_b200 as fa
    from flaxattention_b200 import attention

    q, k, v, _ = _inputs()
    fa.flax_attention(q, k, v)
    seen, run = [], attention._run
    monkeypatch.setattr(attention, "_run", lambda *a: (seen.append(1), run(*a))[1])
    error = None
    try:
        where(lambda x: fa.flax_attention(x, k, v), q)
    except Exception as e:
        error = type(e)
    if refused is not Exception:
        assert error is refused
    assert bool(seen) == python


def test_the_backward_looks_at_the_status_word():
    """An error that an earlier launch reported is raised before the gradients are computed, once."""
    import flaxattention_b200 as fa
    from flaxattention_b200 import _cabi, attention

    q, k, v, do = _inputs()
    x = q.clone().requires_grad_(True)
    for options in (None, {}):
        for _ in range(2):
            out = fa.flax_attention(x, k, v, kernel_options=options)
        torch.cuda.synchronize()
        attention._status()[0] = 1
        with pytest.raises(_cabi.FlaxAttnError, match="status bits 0x1"):
            torch.autograd.grad(out, x, do, retain_graph=True)
        torch.autograd.grad(out, x, do)


def test_tensors_that_saved_tensor_hooks_give_back():
    """Moved to the host and back: the same gradients; with every second value of a row twice as long: refused, as
    such inputs are; with another type: refused."""
    import flaxattention_b200 as fa

    q, k, v, do = _inputs()
    fa.flax_attention(q, k, v)
    ts = [t.clone().requires_grad_(True) for t in (q, k, v)]
    want = torch.autograd.grad(fa.flax_attention(*ts), ts, do)

    def grads(pack, unpack):
        with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
            out = fa.flax_attention(*ts)
        return torch.autograd.grad(out, ts, do)

    got = grads(lambda t: t.cpu(), lambda t: t.cuda())
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    with pytest.raises(ValueError, match="head dimension must be contiguous"):
        grads(lambda t: t, lambda t: t if t.ndim == 3 else torch.stack((t, t), -1).flatten(-2)[..., ::2])
    with pytest.raises(RuntimeError, match="another shape, type or device"):
        grads(lambda t: t, lambda t: t.float())


def test_a_captured_tensor_elsewhere_after_a_build_that_failed():
    """create_block_mask reads a copy on the device; attention calls go on looking at the tensor itself."""
    import flaxattention_b200 as fa
    from flaxattention_b200 import _cabi

    S = 256
    limit = torch.full((S,), 200, dtype=torch.int32)

    def up_to_limit(b, h, q_idx, kv_idx):
        return kv_idx < limit[q_idx]

    q, k, v, _ = _inputs()
    bm = fa.create_block_mask(up_to_limit, None, None, S, S)
    fa.flax_attention(q, k, v, block_mask=bm)
    with pytest.raises(_cabi.FlaxAttnError):
        fa.create_block_mask(up_to_limit, 300, 300, S, S)  # more than 65535 heads
    for _ in range(2):
        before = fa.flax_attention(q, k, v, block_mask=bm)
    limit.fill_(150)
    now = fa.flax_attention(q, k, v, block_mask=bm)
    assert not torch.equal(now, before)
    assert torch.equal(now, fa.flax_attention(q, k, v, block_mask=fa.create_block_mask(up_to_limit, None, None, S, S)))


@pytest.mark.parametrize("dtype,D,S,block", [(torch.float32, 64, 256, 128), (torch.float32, 64, 48, 48), (torch.float32, 32, 128, 128),
                                             (torch.float16, 64, 256, 128), (torch.bfloat16, 128, 256, 128), (torch.float16, 64, 96, 96)])
def test_a_prepared_module_compiles_nothing_at_its_first_call(dtype, D, S, block):
    import random

    import flaxattention_b200 as fa
    from flaxattention_b200 import _cabi
    from flaxattention_b200.blockmask import module_for

    c = random.SystemRandom().random()  # (a text that no cache on disk holds)

    def score(s, b, h, q_idx, kv_idx):
        return s * c

    def mask(b, h, q_idx, kv_idx):
        return (q_idx >= kv_idx) | (q_idx * c > 1e9)

    q, k, v = (torch.randn(1, 2, S, D, device="cuda").to(dtype).requires_grad_(True) for _ in range(3))
    code = {torch.float16: _cabi.FA_F16, torch.bfloat16: _cabi.FA_BF16, torch.float32: _cabi.FA_F32}[dtype]
    module_for(None, mask).prepare(_cabi.KIND_BLOCKMASK, code, D, D)
    for kind in (_cabi.KIND_FWD, _cabi.KIND_BWD):
        module_for(score, mask).prepare(kind, code, D, D, S, S)
    before = _cabi.lib().fa_compile_count()
    fa.create_block_mask(mask, None, None, 96, 96, BLOCK_SIZE=24)  # not whole words
    bm = fa.create_block_mask(mask, None, None, S, S, BLOCK_SIZE=block)
    out = fa.flax_attention_pallas(q, k, v, score_mod=score, block_mask=bm)
    torch.autograd.grad(out.float().sum(), (q, k, v))
    torch.cuda.synchronize()
    assert _cabi.lib().fa_compile_count() == before
