"""The host's estimate of how many key tiles a mask leaves per query tile."""
import numpy as np
import pytest
import torch

from flaxattention_b200 import modtrace
from flaxattention_b200.masks import causal_mask, generate_attention_sink, generate_causal_offset, generate_sliding_window


def _listed(mask, Q, K):
    q, kv = np.arange(Q)[:, None], np.arange(K)[None]
    keep = np.broadcast_to(modtrace.evaluate(modtrace.lower_mods(None, mask).mask, None, 0, 0, q, kv), (Q, K))
    return keep.reshape(Q // 128, 128, K // 128, 128).any(axis=(1, 3)).sum(axis=1).mean()


@pytest.mark.parametrize("Q,K", [(128, 128), (128, 1024), (1024, 1024), (3072, 3072), (4096, 512)])
@pytest.mark.parametrize("mask", [causal_mask, generate_sliding_window(256), generate_attention_sink(300, 4), generate_causal_offset(100)],
                         ids=["causal", "window", "sink", "offset"])
def test_estimate_is_near_the_count(mask, Q, K):
    assert abs(modtrace.lower_mods(None, mask).kv_tiles(Q, K) - max(_listed(mask, Q, K), 1)) <= 1.5


def test_captured_tensors():
    ids, other = torch.zeros(256, dtype=torch.int32), torch.zeros(256, dtype=torch.int32)
    n = lambda mask: modtrace.lower_mods(None, mask).kv_tiles(256, 256)  # noqa: E731
    assert n(lambda b, h, q, kv: (ids[q] == ids[kv]) & (q >= kv)) > 0          # documents
    assert n(lambda b, h, q, kv: (q >= kv) & (ids[kv] == ids[q])) > 0
    assert n(lambda b, h, q, kv: ids[q] == other[kv]) == 0                     # anything else is not known
    assert n(lambda b, h, q, kv: (q >= kv) | (ids[q] == ids[kv])) == 0
    assert n(lambda b, h, q, kv: kv < ids[b]) == 0
    assert modtrace.lower_mods(None, None).kv_tiles(256, 256) == 0


def test_a_failure_is_no_failure_of_the_call(monkeypatch):
    ms = modtrace.lower_mods(None, generate_sliding_window(77))

    def fail(*_):
        raise MemoryError("no room")

    monkeypatch.setattr(modtrace.np, "linspace", fail)
    assert ms.kv_tiles(1024, 1024) == 0
