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


def test_masks_of_scattered_positions():
    """Every tile has some: a stride, one position per row, a band between the samples that a look at a few positions would take."""
    n = lambda mask: modtrace.lower_mods(None, mask).kv_tiles(8192, 8192)  # noqa: E731
    assert n(lambda b, h, q, kv: (kv % 128 == 5) | (q == kv)) == 64
    assert n(lambda b, h, q, kv: (kv // 16) % 8 == 3) == 64
    assert n(lambda b, h, q, kv: (q - kv >= 20) & (q - kv < 26)) == 2


@pytest.mark.parametrize("mask", [lambda b, h, q, kv: (q >= kv) & (b > 0), lambda b, h, q, kv: q + 1000 * h >= kv], ids=["batch", "head"])
def test_masks_that_differ_between_entries_are_not_known(mask):
    assert modtrace.lower_mods(None, mask).kv_tiles(8192, 8192) == 0


def test_documents_are_a_guess_bounded_by_the_rest_of_the_mask():
    ids = torch.arange(8192) // 700
    causal = modtrace.lower_mods(None, lambda b, h, q, kv: (ids[q] == ids[kv]) & (q >= kv))
    assert causal.kv_tiles(8192, 8192) == 8 and causal.kv_tiles(640, 640) == 3
    assert modtrace.lower_mods(None, lambda b, h, q, kv: ids[q] == ids[kv]).kv_tiles(8192, 8192) == 8
