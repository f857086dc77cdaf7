"""A large bias that grows towards the keys that count, in the general decode kernel: one that is linear over the keys (taken at a thread's
first key, the others by multiples of the slope) is rounded no more often than one that is evaluated per key."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 80])  # K and V by TMA, by cp.async
@pytest.mark.parametrize("form", ["linear", "per key"])
def test_rounding_of_a_large_bias(D, form):
    import flaxattention_b200 as fa
    from flaxattention_b200 import fnp

    H, Skv = 8, 4096
    B = Skv // D  # entry b of the batch shows the probabilities of keys D b .. D b + D - 1 as its output
    Skv = B * D

    def mod(score, b, h, q, kv):
        k = kv if form == "linear" else fnp.where(kv >= 0, kv, -kv)
        return score + (k * 2.0 ** -11 + (h * 1000 + 60000))

    q = torch.zeros(B, H, 1, D, dtype=torch.float16, device="cuda")
    q[..., 0] = 1
    raw = (torch.arange(Skv, device="cuda") * 37 % 509) / 256 - 1  # the scores before the mods, exact in fp16
    k = torch.zeros(B, H, Skv, D, dtype=torch.float16, device="cuda")
    k[..., 0] = raw
    v = torch.zeros_like(k)
    for b in range(B):
        v[b, :, D * b:D * b + D] = torch.eye(D, dtype=torch.float16, device="cuda")
    out = fa.flax_attention(q, k, v, score_mod=mod, kernel_options={"path": "decode", "kernels": "general"})
    got = out[:, :, 0].transpose(0, 1).reshape(H, Skv).double()  # [H, keys]
    want = torch.softmax(torch.arange(Skv, device="cuda", dtype=torch.float64) * 2.0 ** -11 + raw.double() * D ** -0.5, -1)
    err = got / want - 1
    # The bias is rounded twice, as c + k / 2048 and times log2(e), and its sum with the score once: errors of up to half a unit of fp32
    # there, evenly spread.  (Once more is 1.09 times the bound as measured; the output in fp16 adds 2e-4.)
    c = [60000 + 1000 * h for h in range(H)]
    units = [(2.0 ** (math.floor(math.log2(x)) - 23), 2.0 ** (math.floor(math.log2(x * math.log2(math.e))) - 23) * math.log(2)) for x in c]
    bound = math.sqrt(sum((a * a + 2 * b * b) / 12 for a, b in units) / H)
    assert err.square().mean().sqrt().item() <= 1.08 * bound
