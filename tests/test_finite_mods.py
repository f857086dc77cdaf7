"""What the tracer knows of a score_mod being finite (modtrace.always_finite) against its values: a function said to be finite has
to be, at the largest indices too; and the mods that matter have to be known."""
import numpy as np
import pytest

from flaxattention_b200 import fnp, modtrace
from flaxattention_b200.mods import checkerboard, generate_alibi_bias

TOP = modtrace._IDX_BOUND - 1
MODS = {  # the mod; whether its derivative is known to be finite
    "checkerboard": (checkerboard, True),
    "alibi": (generate_alibi_bias(8), True),
    "relative": (lambda s, b, h, q, kv: s + (q - kv), True),
    "scaled": (lambda s, b, h, q, kv: s * fnp.exp(-fnp.abs((q - kv) * 0.01)) + 1, True),
    "by_bool": (lambda s, b, h, q, kv: fnp.where(q >= kv, s * 2, s / 3), True),
    "product": (lambda s, b, h, q, kv: s * (q * 0.5) * (kv * 0.5), True),
    "over_position": (lambda s, b, h, q, kv: s / (200 - q), False),
    "over_distance": (lambda s, b, h, q, kv: s / (q - kv), False),
    "root": (lambda s, b, h, q, kv: s * fnp.sqrt((199 - q) * 1.0), False),
    "grows": (lambda s, b, h, q, kv: s * fnp.exp(q * 1.0), False),
    "huge": (lambda s, b, h, q, kv: s * (q * 1e20) * (kv * 1e20), False),
    "inf": (lambda s, b, h, q, kv: s * fnp.where(q >= kv, 1.0, float("-inf")), False),
    "square": (lambda s, b, h, q, kv: s * s, False),
    "softcap": (lambda s, b, h, q, kv: 20 * fnp.tanh(s / 20), False),
}


@pytest.mark.parametrize("name", list(MODS))
def test_a_derivative_said_to_be_finite_is(name):
    mod, known = MODS[name]
    ms = modtrace.lower_mods(mod, None)
    at_0 = "#define FA_SCORE_FINITE_AT_0" in ms.source  # value and derivative, at a score of 0
    assert at_0 == (known or name in ("square", "softcap"))
    assert ("#define FA_SCORE_GRAD_FINITE" in ms.source) == known
    if known or at_0:
        rng = np.random.RandomState(0)
        q, kv = (np.concatenate([rng.randint(0, TOP + 1, 500), [0, 0, TOP, TOP]]).astype(np.int32) for _ in range(2))
        q[-4:], kv[-4:] = [0, TOP, 0, TOP], [0, 0, TOP, TOP]
        for b, h in ((0, 0), (TOP, TOP)):
            if known:
                assert np.isfinite(modtrace.evaluate(ms.grad, np.float32(1e30), np.int32(b), np.int32(h), q, kv)).all()
            if at_0:
                assert all(np.isfinite(modtrace.evaluate(m, np.float32(0), np.int32(b), np.int32(h), q, kv)).all() for m in (ms.score, ms.grad))
