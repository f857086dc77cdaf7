"""What a mask is over a rectangle by interval arithmetic (modtrace.to_cuda_range) against its values there: a rectangle said to be
all kept or all dropped has to be, whatever the mask is made of; and the masks that block-sparse attention lives on have to be
told apart at the rectangles that matter.  The generated text is plain C++ and runs on the host here."""
import ctypes
import subprocess

import numpy as np
import pytest
import torch

from flaxattention_b200 import fnp, modtrace
from flaxattention_b200.masks import causal_mask, generate_attention_sink, generate_causal_offset, generate_sliding_window

DOC = torch.arange(4096) // 300


def _masks():
    return {
        "causal": causal_mask,
        "offset": generate_causal_offset(-70),
        "window": generate_sliding_window(100),
        "sink": generate_attention_sink(64, 4),
        "document": lambda b, h, q, kv: (DOC[q] == DOC[kv]) & (q >= kv),
        "document_or": lambda b, h, q, kv: (DOC[q] == DOC[kv]) | (kv < 40),
        "dilated": lambda b, h, q, kv: ((q - kv) % 7 == 0) & (q >= kv),
        "tiles": lambda b, h, q, kv: q // 96 == kv // 96,
        "negative": lambda b, h, q, kv: (kv - q) // 50 >= -3,
        "by_head": lambda b, h, q, kv: q + 3 * h >= kv - 20 * b,
        "absolute": lambda b, h, q, kv: ~(fnp.abs(q - kv) > 90),
        "bounds": lambda b, h, q, kv: fnp.minimum(q, 200) >= fnp.maximum(kv, 60) - 10,
        "where": lambda b, h, q, kv: fnp.where(q > 150, kv, 2 * kv) < q,
        "float": lambda b, h, q, kv: (q * 0.5 > kv) | (q < 9),
        "wrap": lambda b, h, q, kv: (q * 70000 >= kv * 70001) | (kv != q),
        "shift": lambda b, h, q, kv: (q >> 5) != (kv >> 6),
        "all": lambda b, h, q, kv: (q >= 0) & (kv >= 0),
    }


# of 300 rectangles, at least so many are told to be dropped and kept: about half of what the rules give, so that one that has stopped
# to work is seen (remainders, quotients of negative numbers, minima, selects, shifts, one unknown operand of an or)
TOLD = {"causal": (60, 60), "offset": (85, 40), "window": (95, 11), "sink": (100, 8), "document": (60, 0), "document_or": (0, 7), "dilated": (65, 1),
        "tiles": (90, 18), "negative": (23, 105), "by_head": (50, 75), "absolute": (70, 35), "bounds": (85, 45), "where": (65, 55), "float": (0, 1),
        "wrap": (0, 120), "shift": (2, 125), "all": (0, 300)}


def test_values_that_may_wrap_are_not_told():
    """Products that leave int32 for indices within the bound: no range, in a mask of them alone no function."""
    assert modtrace.to_cuda_range(modtrace.lower_mods(None, lambda b, h, q, kv: q * 70000 >= kv * 70001).mask, "f") is None
    assert modtrace.to_cuda_range(modtrace.lower_mods(None, lambda b, h, q, kv: (q + 1) * (kv + 1) > 9).mask, "f") is None


def _range_function(mod, tmp_path):
    text = modtrace.to_cuda_range(mod, "fa_mask_range")
    if text is None:
        return None
    src = tmp_path / "r.cc"
    src.write_text("#include <algorithm>\n#include <cmath>\n#define __device__\n#define __forceinline__ inline\nusing std::min; using std::max;\n"
                   + "".join(modtrace._PRELUDE) + text +
                   'extern "C" int run(int b, int h, int a, int c, int d, int e) { return fa_mask_range(b, h, a, c, d, e); }\n')
    lib = tmp_path / "r.so"
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", str(src), "-o", str(lib)], check=True)
    return ctypes.CDLL(str(lib)).run


@pytest.mark.parametrize("name", list(_masks()))
def test_a_rectangle_that_is_known_is_right(name, tmp_path):
    ms = modtrace.lower_mods(None, _masks()[name])
    mod = ms.mask
    f = None if mod is None else _range_function(mod, tmp_path)
    assert f is not None
    rng = np.random.RandomState(1)
    told = [0, 0]  # dropped, kept
    for _ in range(300):
        hq, hk = rng.choice([1, 7, 32, 128], 2)
        q0, k0 = (int(x) for x in rng.randint(0, 400, 2))
        b, h = (int(x) for x in rng.randint(0, 4, 2))
        got = f(b, h, q0, q0 + int(hq) - 1, k0, k0 + int(hk) - 1)
        q, kv = np.arange(q0, q0 + hq, dtype=np.int32)[:, None], np.arange(k0, k0 + hk, dtype=np.int32)[None]
        want = np.broadcast_to(modtrace.evaluate(mod, None, np.int32(b), np.int32(h), q, kv), (hq, hk))
        if got != 1:
            told[got // 2] += 1
            assert want.all() if got == 2 else not want.any(), (name, got, b, h, q0, hq, k0, hk)
    assert told[0] >= TOLD[name][0] and told[1] >= TOLD[name][1], told
    assert f(0, 0, 0, 1 << 21, 0, 31) == 1 and f(0, 0, -1, 30, 0, 31) == 1  # beyond the indices the bounds are for
