"""A large bias that is linear over the keys, in the 16-bit forward: it is rounded where it is evaluated, and not again at every key.  In a
row's first tile of keys, in later ones, and far below 0 as well as above."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,Skv", [(64, 128), (64, 1024), (128, 128), (128, 1024)])
@pytest.mark.parametrize("sign", [1, -1])
def test_rounding_of_a_large_bias(D, Skv, sign):
    import flaxattention_b200 as fa

    H, Sq = 32, 128
    B = Skv // D  # entry b of the batch shows the probabilities of keys D b .. D b + D - 1 as its output
    q = torch.zeros(B, H, Sq, D, dtype=torch.float16, device="cuda")
    q[..., 0] = 1
    raw = (torch.arange(Skv, device="cuda") * 37 % 509) / 256 - 1  # the scores before the mods, exact in fp16
    k = torch.zeros(B, H, Skv, D, dtype=torch.float16, device="cuda")
    k[..., 0] = raw
    v = torch.zeros_like(k)
    for b in range(B):
        v[b, :, D * b:D * b + D] = torch.eye(D, dtype=torch.float16, device="cuda")
    out = fa.flax_attention_pallas(q, k, v, score_mod=lambda s, b, h, q, kv: s + (kv * 2.0 ** -11 + sign * (h * 200 + 60000)))
    got = out[:, :, 0].transpose(0, 1).reshape(H, Skv).double()  # [H, keys]
    want = torch.softmax(torch.arange(Skv, device="cuda", dtype=torch.float64) * 2.0 ** -11 + raw.double() * D ** -0.5, -1)
    err = got / want - 1
    # The bias is rounded twice, as c + k / 2048 and times log2(e): errors of up to half a unit of fp32 there, evenly spread.  Its sum with the
    # score would be a third, one more per key a fourth (1.18 of the bound); probabilities and output in fp16 add 2e-4 of 2.5e-3.
    c = [60000 + 200 * h for h in range(H)]
    units = [(2.0 ** (math.floor(math.log2(x)) - 23), 2.0 ** (math.floor(math.log2(x * math.log2(math.e))) - 23) * math.log(2)) for x in c]
    bound = math.sqrt(sum((a * a + 2 * b * b) / 12 for a, b in units) / H)
    assert err.square().mean().sqrt().item() <= bound
