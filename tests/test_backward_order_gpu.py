"""GPU parity of the backward where the order of its work items matters: enough heads for several chunks (the last
one smaller than the others), grouped heads, a ragged last kv tile, one kv tile only, and every (kv tile, head)
item written exactly once (dK, dV of all heads are compared).

Tolerance: gradients <= 5e-2 relative to an fp32 reference of the same inputs, the bar of the other backward tests."""
import pytest
import torch

from _util import DTYPES, rel_err

pytestmark = pytest.mark.gpu


def _reference(q, k, v, do, mask):
    """fp32 gradients, one query head at a time."""
    B, Hq, S, D = q.shape
    G = Hq // k.shape[1]
    dq, dk, dv = torch.empty_like(q, dtype=torch.float32), torch.zeros_like(k, dtype=torch.float32), torch.zeros_like(v, dtype=torch.float32)
    for b in range(B):
        for h in range(Hq):
            qf, kf, vf, df = (t[b, h // g].float() for t, g in ((q, 1), (k, G), (v, G), (do, 1)))
            s = qf @ kf.T * D ** -0.5
            if mask is not None:
                s.masked_fill_(~mask, float("-inf"))
            p = torch.softmax(s, -1)
            ds = p * (df @ vf.T - (df * (p @ vf)).sum(-1, keepdim=True)) * D ** -0.5
            dq[b, h] = ds @ kf
            dk[b, h // G] += ds.T @ qf
            dv[b, h // G] += p.T @ df
    return dq, dk, dv


# dense: chunks of 24 MB / (Sq * D * 8 bytes) heads; with tables: of 96 MB, when that leaves 3 items per SM
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,D,dt,sink", [
    (1, 9, 9, 4096, 4096, 128, "bf16", 0),     # chunks of 6 and 3
    (2, 10, 5, 1920, 3333, 128, "f16", 0),     # grouped: chunks of 6 and 4 (batch, kv head) pairs, ragged last kv tile
    (1, 13, 13, 4096, 2500, 64, "bf16", 0),    # head dim 64: chunks of 12 and 1
    (1, 14, 14, 8192, 8192, 128, "bf16", 512),  # with tables: chunks of 12 and 2, the first kv tile heavier
    (3, 5, 5, 700, 128, 64, "f16", 0),         # one kv tile
    (1, 2, 2, 130, 1000, 128, "f16", 0),       # q tiles fewer than kv tiles: starts that coincide
])
def test_backward_over_chunks_of_heads(B, Hq, Hkv, Sq, Skv, D, dt, sink):
    import flaxattention_b200 as fa
    from flaxattention_b200.masks import generate_attention_sink

    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = (torch.randn(B, h, s, D, generator=g, device="cuda").to(DTYPES[dt]) for h, s in
                   ((Hq, Sq), (Hkv, Skv), (Hkv, Skv), (Hq, Sq)))
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    bm = mask = None
    if sink:
        mod = generate_attention_sink(sink, 4)
        bm = fa.create_block_mask(mod, None, None, Sq, Skv)
        i, j = torch.arange(Sq, device="cuda")[:, None], torch.arange(Skv, device="cuda")[None]
        mask = mod(0, 0, i, j)
    out, _ = fa.flax_attention_pallas(q, k, v, block_mask=bm, enable_gqa=Hq != Hkv, return_lse=True)
    got = torch.autograd.grad(out, (q, k, v), do)
    with torch.no_grad():
        ref = _reference(q, k, v, do, mask)
    for name, a, r in zip(("dq", "dk", "dv"), got, ref):
        for b in range(B):
            for h in range(a.shape[1]):
                assert rel_err(a[b, h], r[b, h]) <= 5e-2, (name, b, h)
