"""score_mods that put a large negative number in the place of scores, in the tiles of keys that a row meets first: they are the row's
running maximum until others come, and the others must not be lost against them.

Tolerance: O <= 2e-2 of values around 1, the bar of the other forward tests.  LSE <= 3e-4: a quarter of the exponentials is
a cubic with a relative error of 1.0e-4, the scores (up to 8 in log2 units) are rounded to 2^-21, or to 2^-18 against a maximum of -64.
(Scores taken relative to -1e4 are rounded to 2^-11 in log2 units, 3.4e-4 per key, to -1e9 lost.)"""
import pytest
import torch

from _util import DTYPES, max_abs, qkv
from flaxattention_b200 import fnp
from flaxattention_b200.masks import causal_mask

pytestmark = pytest.mark.gpu

MODS = {  # affine in the score or not, and the bias of a line over the keys
    "where": (lambda n, low: (lambda s, b, h, q, kv: fnp.where((kv // n) % 2 == 0, low, s)),
              lambda n, low, s, kv: torch.where((kv // n) % 2 == 0, low, s)),
    "add": (lambda n, low: (lambda s, b, h, q, kv: s + fnp.where((kv // n) % 2 == 0, low, 0.0)),
            lambda n, low, s, kv: s + torch.where((kv // n) % 2 == 0, low, 0.0)),
    "softcap": (lambda n, low: (lambda s, b, h, q, kv: fnp.where((kv // n) % 2 == 0, low, 20 * fnp.tanh(s / 20))),
                lambda n, low, s, kv: torch.where((kv // n) % 2 == 0, low, 20 * torch.tanh(s / 20))),
}


def _reference(q, k, v, values, keep, low, n):
    q, k, v = q.double(), k.double(), v.double()
    kv = torch.arange(k.shape[2], device="cuda")
    s = values(n, torch.tensor(low, dtype=torch.float64, device="cuda"), q @ k.transpose(-1, -2) * q.shape[-1] ** -0.5, kv)
    if keep:
        s = s.masked_fill(kv > torch.arange(q.shape[2], device="cuda")[:, None], float("-inf"))
    return torch.softmax(s, -1) @ v, torch.logsumexp(s, -1)


def _check(out, lse, ref, ref_lse, name):
    low = ref_lse < -1e3  # (rows of nothing else: LSE relative; the sum of a score and -1e9 has no more than its multiples of 64 in fp32)
    seen = ~low if name == "add" else torch.ones_like(low)
    assert torch.isfinite(out).all() and max_abs(out[seen], ref[seen]) <= 2e-2
    assert max_abs(lse[~low], ref_lse[~low]) <= 3e-4
    assert max_abs(lse[low] / ref_lse[low], torch.ones_like(ref_lse[low])) <= 1e-6 if low.any() else True


@pytest.mark.parametrize("low", [-20.0, -40.0, -50.0, -1e4, -1e9, -1e30])
@pytest.mark.parametrize("name", list(MODS))
@pytest.mark.parametrize("B,H,Sq,Skv,D,dt,causal", [
    (1, 2, 128, 133, 64, "f16", False),     # one query tile per CTA; five keys that count
    (1, 2, 300, 900, 128, "bf16", False),
    (1, 3, 640, 640, 64, "bf16", True),
    (2, 26, 300, 300, 128, "f16", True),    # two query tiles: 156
    (2, 9, 1100, 2100, 64, "f16", False),   # 162
])
def test_forward(B, H, Sq, Skv, D, dt, causal, name, low):
    import flaxattention_b200 as fa

    make, values = MODS[name]
    q, k, v = (t.cuda() for t in qkv(B, H, H, Sq, Skv, D, dtype=DTYPES[dt]))
    bm = fa.create_block_mask(causal_mask, None, None, Sq, Skv) if causal else None
    out, lse = fa.flax_attention_pallas(q, k, v, score_mod=make(128, low), block_mask=bm, return_lse=True)
    _check(out, lse, *_reference(q, k, v, values, causal, low, 128), name)


@pytest.mark.parametrize("low", [-20.0, -50.0, -1e4, -1e9, -1e30])
@pytest.mark.parametrize("name", list(MODS))
@pytest.mark.parametrize("Sq", [1, 48])
def test_decode(Sq, name, low):
    """(48 rows: the tcgen05 decode kernel, whose warpgroups take the tiles in turn)"""
    import flaxattention_b200 as fa

    make, values = MODS[name]
    q, k, v = (t.cuda() for t in qkv(1, 2, 2, Sq, 2053, 64, dtype=torch.float16))
    out, lse = fa.flax_attention(q, k, v, score_mod=make(256, low), return_lse=True,
                                 kernel_options={"path": "decode", "num_splits": 2, "round_scores": False})
    _check(out, lse, *_reference(q, k, v, values, False, low, 256), name)
