"""Lowering of user ``score_mod`` / ``mask_mod`` callables to CUDA device-function fragments.

The reference evaluates the mods by ``jax.vmap`` over (kv, q, h, b)
(flaxattention/core/common.py:41-81) on the dense score tensor, and inside its Pallas
kernel on (block_q, block_k) index spans (flaxattention/kernel/attention.py:83-93).
Here a mod is called ONCE with symbolic scalars; every operator applied to them is
recorded into a small SSA expression graph (int32 / float32 / bool scalars).  That
graph has three back ends:

* ``to_cuda``      - text of a ``__device__ __forceinline__`` function that the runtime
                     compiler splices into the attention kernel templates;
* ``evaluate``     - a numpy evaluator (used by the tests to check the tracer);
* ``derivative``   - the symbolic derivative with respect to the score argument, which
                     plays the role of ``jax.grad(score_mod)``
                     (flaxattention/core/attention.py:286).

Integer ``%`` and ``//`` follow Python / ``jnp.remainder`` / ``jnp.floor_divide``
semantics (result takes the sign of the divisor, division rounds toward -inf).
Python scalars are weakly typed the way JAX treats them: ``int32 * 8.0`` is float32,
``int32 + 1`` stays int32, ``/`` always gives float32.
"""
from __future__ import annotations

import builtins
import contextlib
import copy
import dis
import functools
import hashlib
import inspect
import math
import struct
import types
import weakref
from typing import Callable, Dict, List, Optional, Sequence, Tuple

import numpy as np
import torch
from torch.utils._python_dispatch import TorchDispatchMode

I32, F32, B1 = "i32", "f32", "b1"

_LEAVES = ("score", "b", "h", "q", "kv")
_UNARY_F = (
    "exp", "exp2", "log", "log2", "sqrt", "rsqrt", "tanh", "sigmoid", "sin", "cos",
    "floor", "ceil", "erf",
)


class Expr:
    """One node of the expression graph (hash-consed, immutable)."""

    __slots__ = ("op", "dtype", "args", "value", "_key")

    def __init__(self, op: str, dtype: str, args: Tuple["Expr", ...] = (), value=None):
        self.op = op
        self.dtype = dtype
        self.args = args
        self.value = value
        self._key = (op, dtype, tuple(id(a) for a in args), value if op in ("const", "load") else None)

    def __repr__(self):
        if self.op == "const":
            return f"{self.value!r}:{self.dtype}"
        if not self.args:
            return self.op
        return f"{self.op}({', '.join(map(repr, self.args))})"


class _Builder:
    """Hash-consing constructor with light algebraic simplification."""

    def __init__(self):
        self._table: Dict[tuple, Expr] = {}

    def _mk(self, op, dtype, args=(), value=None) -> Expr:
        if op == "const":
            if dtype == F32:
                v = float(np.float32(value))
                key = ("const", dtype, np.float32(v).tobytes())
            elif dtype == I32:
                v = int(np.int64(value).astype(np.int32)) if not isinstance(value, int) else _wrap_i32(value)
                key = ("const", dtype, v)
            else:
                v = bool(value)
                key = ("const", dtype, v)
            e = self._table.get(key)
            if e is None:
                e = Expr("const", dtype, (), v)
                self._table[key] = e
            return e
        key = (op, dtype, tuple(id(a) for a in args), value if op == "load" else None)
        e = self._table.get(key)
        if e is None:
            e = Expr(op, dtype, tuple(args), value if op == "load" else None)
            self._table[key] = e
        return e

    def const(self, value, dtype) -> Expr:
        return self._mk("const", dtype, value=value)

    def leaf(self, name) -> Expr:
        return self._mk(name, F32 if name == "score" else I32)


def _wrap_i32(v: int) -> int:
    v &= 0xFFFFFFFF
    return v - (1 << 32) if v & 0x80000000 else v


_B = _Builder()


def _depends_on_leaves(e: Expr, leaves, memo=None) -> bool:
    if memo is None:
        memo = {}
    r = memo.get(id(e))
    if r is None:
        r = e.op in leaves or any(_depends_on_leaves(a, leaves, memo) for a in e.args)
        memo[id(e)] = r
    return r


def _is_const(e: Expr, v=None) -> bool:
    if e.op != "const":
        return False
    return True if v is None else e.value == v


# --------------------------------------------------------------------------------------
# typed constructors
# --------------------------------------------------------------------------------------
def _is_bit(e: Expr) -> bool:
    """True when the int32 expression can only be 0 or 1."""
    if e.dtype != I32:
        return False
    if e.op == "const":
        return e.value in (0, 1)
    if e.op == "and":
        return _is_const(e.args[0], 1) or _is_const(e.args[1], 1) or (_is_bit(e.args[0]) and _is_bit(e.args[1]))
    if e.op in ("or", "xor"):
        return _is_bit(e.args[0]) and _is_bit(e.args[1])
    if e.op == "cast_i32":
        return e.args[0].dtype == B1
    return False


def _parity(e: Expr) -> Expr:
    """e & 1 with the mask pushed through +, -, negation: the low bit of a sum is the xor of
    the low bits.  This separates the q and kv contributions of expressions like
    (kv - q) % 2, so that a kernel can evaluate the kv part per column at compile time."""
    if e.op == "const":
        return _B.const(e.value & 1, I32)
    if e.op in ("add", "sub") and e.dtype == I32:
        a, b = _parity(e.args[0]), _parity(e.args[1])
        if _is_const(a, 0):
            return b
        if _is_const(b, 0):
            return a
        if a.op == "const" and b.op == "const":
            return _B.const(a.value ^ b.value, I32)
        return _B._mk("xor", I32, (a, b))
    if e.op == "neg" and e.dtype == I32:
        return _parity(e.args[0])
    if _is_bit(e):
        return e
    return _B._mk("and", I32, (e, _B.const(1, I32)))


_UNARY_OPS = ("neg", "not", "abs", "isneginf", "isinf", "isnan", "sign") + _UNARY_F
_BINARY_OPS = ("add", "sub", "mul", "div", "floordiv", "rem", "pow", "min", "max", "and", "or", "xor", "shl", "shr",
               "lt", "le", "gt", "ge", "eq", "ne")


def _rebuild(e: Expr, args) -> Expr:
    if e.op in _UNARY_OPS:
        return unary(e.op, args[0])
    if e.op in _BINARY_OPS:
        return binary(e.op, args[0], args[1])
    if e.op == "select":
        return select(args[0], args[1], args[2])
    if e.op.startswith("cast_"):
        return cast(args[0], e.dtype)
    if e.op == "load":
        return _B._mk("load", e.dtype, (args[0],), e.value)
    raise NotImplementedError(e.op)


def _assume(e: Expr, cond: Expr, value: bool, memo=None) -> Expr:
    """e with the boolean node `cond` replaced by a constant, re-simplified."""
    if memo is None:
        memo = {}
    if e is cond:
        return _B.const(value, B1)
    if not e.args:
        return e
    got = memo.get(id(e))
    if got is not None:
        return got
    new_args = tuple(_assume(a, cond, value, memo) for a in e.args)
    r = e if all(x is y for x, y in zip(new_args, e.args)) else _rebuild(e, new_args)
    memo[id(e)] = r
    return r


def cast(e: Expr, dtype: str) -> Expr:
    if e.dtype == dtype:
        return e
    if e.op == "const":
        if dtype == B1:
            return _B.const(e.value != 0, B1)
        if dtype == I32:
            return _B.const(int(e.value), I32)
        return _B.const(float(e.value), F32)
    return _B._mk("cast_" + dtype, dtype, (e,))


def _promote(a: Expr, b: Expr) -> Tuple[Expr, Expr, str]:
    """Result type of an arithmetic op on two typed operands."""
    if F32 in (a.dtype, b.dtype):
        t = F32
    elif I32 in (a.dtype, b.dtype):
        t = I32
    else:
        t = B1
    return cast(a, t), cast(b, t), t


def binary(op: str, a: Expr, b: Expr) -> Expr:
    if op in ("and", "or", "xor"):
        a, b, t = _promote(a, b)
        if t == F32:
            raise TypeError(f"bitwise '{op}' is not defined for float operands")
        if t == I32 and op == "and":
            if _is_const(b, 1) and a.op in ("add", "sub", "neg", "const"):
                return _parity(a)
            if _is_const(a, 1) and b.op in ("add", "sub", "neg", "const"):
                return _parity(b)
        if t == B1:
            if op == "and":
                if _is_const(a):
                    return b if a.value else a
                if _is_const(b):
                    return a if b.value else b
            if op == "or":
                if _is_const(a):
                    return a if a.value else b
                if _is_const(b):
                    return b if b.value else a
        return _B._mk(op, t, (a, b))
    if op in ("lt", "le", "gt", "ge", "eq", "ne"):
        a, b, t = _promote(a, b)
        if t == B1:
            a, b = cast(a, I32), cast(b, I32)
        if op in ("eq", "ne") and t == I32:
            if a.op == "const" and b.op != "const":
                a, b = b, a
            if b.op == "const" and _is_bit(a) and a.op != "const":
                # a is 0 or 1: every test against a constant is `a == 0`, its negation, or constant
                is_zero = _B._mk("eq", B1, (a, _B.const(0, I32)))
                if b.value not in (0, 1):
                    return _B.const(op == "ne", B1)
                if (op == "eq") == (b.value == 0):
                    return is_zero
                return unary("not", is_zero)
        return _B._mk(op, B1, (a, b))
    if op in ("shl", "shr"):
        a, b = cast(a, I32), cast(b, I32)
        return _B._mk(op, I32, (a, b))
    a, b, t = _promote(a, b)
    if t == B1:
        a, b, t = cast(a, I32), cast(b, I32), I32
    if op == "div":
        a, b, t = cast(a, F32), cast(b, F32), F32
    if op == "pow":
        a, b, t = cast(a, F32), cast(b, F32), F32
    # light simplification; keeps derivative graphs small
    if op == "add":
        if _is_const(a, 0):
            return b
        if _is_const(b, 0):
            return a
    elif op == "sub":
        if _is_const(b, 0):
            return a
    elif op == "mul":
        if t == F32:
            # (x * y) * c -> x * (y * c) when y does not vary along a score row (no score, no kv):
            # the kernels can then hoist y * c out of their per-element loops
            for u, c in ((a, b), (b, a)):
                if c.op == "const" and u.op == "mul" and u.dtype == F32:
                    for x, y in ((u.args[0], u.args[1]), (u.args[1], u.args[0])):
                        if y.op != "const" and not _depends_on_leaves(y, ("score", "kv")) and _depends_on_leaves(x, ("score", "kv")):
                            return binary("mul", x, binary("mul", y, c))
        if _is_const(a, 1):
            return b
        if _is_const(b, 1):
            return a
        if _is_const(a, 0) or _is_const(b, 0):
            return _B.const(0, t)
    elif op == "div":
        if _is_const(b, 1):
            return a
    if t == I32 and op in ("rem", "floordiv") and b.op == "const" and b.value > 0 and (b.value & (b.value - 1)) == 0:
        # Python semantics for a positive power-of-two divisor are exactly the two's-complement
        # mask / arithmetic shift: x % 2^k == x & (2^k - 1), x // 2^k == x >> k
        if b.value == 1:
            return _B.const(0, I32) if op == "rem" else a
        if op == "rem":
            return binary("and", a, _B.const(b.value - 1, I32))
        return _B._mk("shr", I32, (a, _B.const(b.value.bit_length() - 1, I32)))
    if a.op == "const" and b.op == "const":
        folded = _fold_binary(op, a.value, b.value, t)
        if folded is not None:
            return _B.const(folded, t)
    return _B._mk(op, t, (a, b))


def _fold_binary(op, x, y, t):
    try:
        if t == F32:
            x32, y32 = np.float32(x), np.float32(y)
            with np.errstate(all="ignore"):
                if op == "add":
                    return float(x32 + y32)
                if op == "sub":
                    return float(x32 - y32)
                if op == "mul":
                    return float(x32 * y32)
                if op == "div":
                    return float(x32 / y32)
                if op == "min":
                    return float(np.minimum(x32, y32))
                if op == "max":
                    return float(np.maximum(x32, y32))
            return None
        if op == "add":
            return _wrap_i32(x + y)
        if op == "sub":
            return _wrap_i32(x - y)
        if op == "mul":
            return _wrap_i32(x * y)
        if op == "floordiv" and y != 0:
            return _wrap_i32(x // y)
        if op == "rem" and y != 0:
            return _wrap_i32(x % y)
        if op == "min":
            return min(x, y)
        if op == "max":
            return max(x, y)
    except Exception:
        return None
    return None


def unary(op: str, a: Expr) -> Expr:
    if op == "neg":
        if a.dtype == B1:
            a = cast(a, I32)
        if a.op == "const":
            return _B.const(-a.value, a.dtype)
        return _B._mk("neg", a.dtype, (a,))
    if op == "not":
        if a.dtype == F32:
            raise TypeError("'~' is not defined for float operands")
        if a.op == "const" and a.dtype == B1:
            return _B.const(not a.value, B1)
        if a.op == "not" and a.dtype == B1:
            return a.args[0]
        return _B._mk("not", a.dtype, (a,))
    if op == "abs":
        if a.dtype == B1:
            return cast(a, I32)
        return _B._mk("abs", a.dtype, (a,))
    if op in ("isneginf", "isinf", "isnan"):
        return _B._mk(op, B1, (cast(a, F32),))
    if op == "sign":
        return _B._mk(op, a.dtype if a.dtype != B1 else I32, (a if a.dtype != B1 else cast(a, I32),))
    if op in _UNARY_F:
        a = cast(a, F32)
        if a.op == "const" and op in ("exp2", "exp", "log", "log2", "sqrt"):
            with np.errstate(all="ignore"):
                f = {"exp2": np.exp2, "exp": np.exp, "log": np.log, "log2": np.log2, "sqrt": np.sqrt}[op]
                return _B.const(float(f(np.float32(a.value))), F32)
        return _B._mk(op, F32, (a,))
    raise ValueError(f"unknown unary op {op}")


def select(c: Expr, a: Expr, b: Expr) -> Expr:
    c = cast(c, B1)
    a, b, t = _promote(a, b)
    if c.op == "const":
        return a if c.value else b
    if c.op == "not":
        c, a, b = c.args[0], b, a
    # inside the arms the condition is known
    a = _assume(a, c, True)
    b = _assume(b, c, False)
    a, b, t = _promote(a, b)
    if a is b:
        return a
    return _B._mk("select", t, (c, a, b))


# --------------------------------------------------------------------------------------
# the tracer value
# --------------------------------------------------------------------------------------
def _lift(x) -> Expr:
    if isinstance(x, Sym):
        return x.e
    if isinstance(x, Expr):
        return x
    if isinstance(x, (bool, np.bool_)):
        return _B.const(bool(x), B1)
    if isinstance(x, (int, np.integer)):
        return _B.const(int(x), I32)
    if isinstance(x, (float, np.floating)):
        return _B.const(float(x), F32)
    if isinstance(x, np.ndarray) and x.ndim == 0:
        return _lift(x.item())
    try:  # 0-d torch tensors captured as constants
        import torch

        if isinstance(x, torch.Tensor) and x.ndim == 0:
            return _lift(x.item())
    except ImportError:  # pragma: no cover
        pass
    raise TypeError(
        f"cannot use a value of type {type(x).__name__} inside a score_mod/mask_mod trace; "
        "only Python scalars and the traced arguments are supported"
    )


# --------------------------------------------------------------------------------------
# captured buffers: tensors a mod closes over and indexes with traced values
# (score_mod_other_buffers / mask_mod_other_buffers of flaxattention/core/attention.py:22-23,
#  :35-52; in the reference they are jaxpr constants, here the tensors the closure holds)
# --------------------------------------------------------------------------------------
MAX_MOD_BUFFERS = 8
_ELEM_TYPES = {
    "torch.int32": ("i32", I32), "torch.int64": ("i64", I32), "torch.uint8": ("u8", I32), "torch.bool": ("u8", B1),
    "torch.float32": ("f32", F32),
    "int32": ("i32", I32), "int64": ("i64", I32), "uint8": ("u8", I32), "bool": ("u8", B1), "float32": ("f32", F32),
}
_TRACE_BUFFERS: Optional[List[object]] = None  # buffers of the mod pair being traced


def _buffer_load(buf, index) -> "Sym":
    """``buf[index]`` with traced indices: registers the tensor and records a load node.  The
    linear index is built from the tensor's strides; out-of-range indices (rows and keys of the
    padding of a ragged tile reach the mods too) are clamped by the generated code."""
    if _TRACE_BUFFERS is None:
        raise TypeError("a tensor can only be indexed with a traced value while a mod is being lowered")
    et = _ELEM_TYPES.get(str(buf.dtype))
    if et is None:
        raise TypeError(f"captured buffers of dtype {buf.dtype} are not supported (int32, int64, uint8, bool, float32 are)")
    idx = index if isinstance(index, tuple) else (index,)
    shape = tuple(int(d) for d in buf.shape)
    if len(idx) != len(shape):
        raise TypeError(f"a captured buffer of {len(shape)} dimensions needs {len(shape)} indices, got {len(idx)}")
    if hasattr(buf, "stride") and callable(buf.stride):
        strides = tuple(int(x) for x in buf.stride())
    else:
        strides = tuple(int(x // buf.itemsize) for x in buf.strides)
    numel = 1
    for d in shape:
        numel *= d
    if numel == 0 or numel >= (1 << 31):
        raise TypeError("captured buffers must hold between 1 and 2^31-1 elements")
    span = 1 + sum((d - 1) * st for d, st in zip(shape, strides))
    k = None
    for i, b in enumerate(_TRACE_BUFFERS):
        if b is buf:
            k = i
    if k is None:
        if len(_TRACE_BUFFERS) >= MAX_MOD_BUFFERS:
            raise TypeError(f"at most {MAX_MOD_BUFFERS} captured buffers per (score_mod, mask_mod) pair")
        _TRACE_BUFFERS.append(buf)
        k = len(_TRACE_BUFFERS) - 1
    lin = _B.const(0, I32)
    for i, st in zip(idx, strides):
        e = cast(_lift(i), I32)
        lin = binary("add", lin, binary("mul", e, _B.const(st, I32)))
    return Sym(_B._mk("load", et[1], (lin,), (k, span, et[0])))


def _bin(op):
    def f(self, other):
        try:
            return Sym(binary(op, self.e, _lift(other)))
        except TypeError:
            return NotImplemented

    def r(self, other):
        try:
            return Sym(binary(op, _lift(other), self.e))
        except TypeError:
            return NotImplemented

    return f, r


class Sym:
    """Symbolic scalar handed to a mod while it is traced."""

    __slots__ = ("e",)
    __array_priority__ = 1000

    def __init__(self, e: Expr):
        self.e = e

    @property
    def dtype(self):
        return {I32: np.dtype("int32"), F32: np.dtype("float32"), B1: np.dtype("bool")}[self.e.dtype]

    shape = ()
    ndim = 0

    __add__, __radd__ = _bin("add")
    __sub__, __rsub__ = _bin("sub")
    __mul__, __rmul__ = _bin("mul")
    __truediv__, __rtruediv__ = _bin("div")
    __floordiv__, __rfloordiv__ = _bin("floordiv")
    __mod__, __rmod__ = _bin("rem")
    __pow__, __rpow__ = _bin("pow")
    __and__, __rand__ = _bin("and")
    __or__, __ror__ = _bin("or")
    __xor__, __rxor__ = _bin("xor")
    __lshift__, __rlshift__ = _bin("shl")
    __rshift__, __rrshift__ = _bin("shr")
    __lt__, _ = _bin("lt")
    __le__, _ = _bin("le")
    __gt__, _ = _bin("gt")
    __ge__, _ = _bin("ge")
    __eq__, _ = _bin("eq")  # type: ignore[assignment]
    __ne__, _ = _bin("ne")  # type: ignore[assignment]
    __hash__ = None  # type: ignore[assignment]

    def __neg__(self):
        return Sym(unary("neg", self.e))

    def __pos__(self):
        return self

    def __invert__(self):
        return Sym(unary("not", self.e))

    def __abs__(self):
        return Sym(unary("abs", self.e))

    def __bool__(self):
        raise TypeError(
            "the truth value of a traced value is not known while a score_mod/mask_mod is being "
            "lowered; use where(cond, a, b) and the &, |, ~ operators instead of if/and/or/not"
        )

    def astype(self, dtype):
        return Sym(cast(self.e, _dtype_name(dtype)))

    # numpy interop: np.exp2(sym), np.where(sym, a, b) ...
    def __array_ufunc__(self, ufunc, method, *inputs, **kwargs):
        if method != "__call__" or kwargs:
            return NotImplemented
        fn = _NP_UFUNCS.get(ufunc.__name__)
        if fn is None:
            return NotImplemented
        return fn(*inputs)

    def __array_function__(self, func, types, args, kwargs):
        if func is np.where and not kwargs and len(args) == 3:
            return where(*args)
        return NotImplemented

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        name = getattr(func, "__name__", "")
        if name == "__getitem__" and len(args) == 2 and not isinstance(args[0], Sym):
            return _buffer_load(args[0], args[1])
        fn = _TORCH_FUNCS.get(name)
        if fn is None or kwargs:
            return NotImplemented
        return fn(*args)


def _dtype_name(dtype) -> str:
    if dtype in (bool, np.bool_) or str(dtype) in ("bool", "torch.bool"):
        return B1
    s = str(dtype)
    if "int" in s:
        return I32
    if "float" in s or dtype is float:
        return F32
    if dtype is int:
        return I32
    raise TypeError(f"unsupported dtype {dtype!r} in a mod trace")


# --------------------------------------------------------------------------------------
# function namespace usable on Sym / numpy / torch values alike
# --------------------------------------------------------------------------------------
def _any_sym(*xs) -> bool:
    return any(isinstance(x, Sym) for x in xs)


def _is_torch(*xs) -> bool:
    for x in xs:
        if type(x).__module__.startswith("torch"):
            return True
    return False


def _mk_unary(op, np_fn, torch_name):
    def f(x):
        if isinstance(x, Sym):
            return Sym(unary(op, x.e))
        if _is_torch(x):
            import torch

            return getattr(torch, torch_name)(x)
        return np_fn(x)

    f.__name__ = op
    return f


def _np_sigmoid(x):
    return 1.0 / (1.0 + np.exp(-np.asarray(x, dtype=np.float32)))


def _np_rsqrt(x):
    return 1.0 / np.sqrt(x)


exp = _mk_unary("exp", np.exp, "exp")
exp2 = _mk_unary("exp2", np.exp2, "exp2")
log = _mk_unary("log", np.log, "log")
log2 = _mk_unary("log2", np.log2, "log2")
sqrt = _mk_unary("sqrt", np.sqrt, "sqrt")
rsqrt = _mk_unary("rsqrt", _np_rsqrt, "rsqrt")
tanh = _mk_unary("tanh", np.tanh, "tanh")
sigmoid = _mk_unary("sigmoid", _np_sigmoid, "sigmoid")
sin = _mk_unary("sin", np.sin, "sin")
cos = _mk_unary("cos", np.cos, "cos")
floor = _mk_unary("floor", np.floor, "floor")
ceil = _mk_unary("ceil", np.ceil, "ceil")
isneginf = _mk_unary("isneginf", np.isneginf, "isneginf")
isinf = _mk_unary("isinf", np.isinf, "isinf")
isnan = _mk_unary("isnan", np.isnan, "isnan")
sign = _mk_unary("sign", np.sign, "sign")


def abs(x):  # noqa: A001 - mirrors jnp.abs
    if isinstance(x, Sym):
        return Sym(unary("abs", x.e))
    if _is_torch(x):
        import torch

        return torch.abs(x)
    return np.abs(x)


def where(c, a, b):
    if _any_sym(c, a, b):
        return Sym(select(_lift(c), _lift(a), _lift(b)))
    if _is_torch(c, a, b):
        import torch

        if not isinstance(c, torch.Tensor):
            c = torch.as_tensor(c)
        return torch.where(c, a, b)
    return np.where(c, a, b)


def _mk_binary(op, np_fn, torch_name):
    def f(a, b):
        if _any_sym(a, b):
            return Sym(binary(op, _lift(a), _lift(b)))
        if _is_torch(a, b):
            import torch

            if not isinstance(a, torch.Tensor):
                a = torch.as_tensor(a)
            if not isinstance(b, torch.Tensor):
                b = torch.as_tensor(b)
            return getattr(torch, torch_name)(a, b)
        return np_fn(a, b)

    f.__name__ = op
    return f


minimum = _mk_binary("min", np.minimum, "minimum")
maximum = _mk_binary("max", np.maximum, "maximum")
remainder = _mk_binary("rem", np.remainder, "remainder")
floor_divide = _mk_binary("floordiv", np.floor_divide, "floor_divide")
power = _mk_binary("pow", np.power, "pow")


def logical_and(a, b):
    if _any_sym(a, b):
        return Sym(binary("and", cast(_lift(a), B1), cast(_lift(b), B1)))
    if _is_torch(a, b):
        import torch

        return torch.logical_and(a, b)
    return np.logical_and(a, b)


def logical_or(a, b):
    if _any_sym(a, b):
        return Sym(binary("or", cast(_lift(a), B1), cast(_lift(b), B1)))
    if _is_torch(a, b):
        import torch

        return torch.logical_or(a, b)
    return np.logical_or(a, b)


def logical_not(a):
    if isinstance(a, Sym):
        return Sym(unary("not", cast(a.e, B1)))
    if _is_torch(a):
        import torch

        return torch.logical_not(a)
    return np.logical_not(a)


def ones(shape=(), dtype=np.float32):
    """Scalar one of the given dtype (the reference's combinators start from
    ``jnp.ones((), dtype=bool)``, flaxattention/core/blockmask.py:392)."""
    if shape not in ((), []):
        raise ValueError("only scalar constants can be created inside a mod")
    return np.ones((), dtype=np.bool_ if dtype in (bool, np.bool_) else dtype)[()]


def zeros(shape=(), dtype=np.float32):
    if shape not in ((), []):
        raise ValueError("only scalar constants can be created inside a mod")
    return np.zeros((), dtype=np.bool_ if dtype in (bool, np.bool_) else dtype)[()]


def float32(x):
    if isinstance(x, Sym):
        return x.astype(np.float32)
    if _is_torch(x):
        import torch

        return x.to(torch.float32)
    return np.float32(x)


def int32(x):
    if isinstance(x, Sym):
        return x.astype(np.int32)
    if _is_torch(x):
        import torch

        return x.to(torch.int32)
    return np.int32(x)


inf = float("inf")

_NP_UFUNCS = {
    "add": lambda a, b: Sym(binary("add", _lift(a), _lift(b))),
    "subtract": lambda a, b: Sym(binary("sub", _lift(a), _lift(b))),
    "multiply": lambda a, b: Sym(binary("mul", _lift(a), _lift(b))),
    "true_divide": lambda a, b: Sym(binary("div", _lift(a), _lift(b))),
    "divide": lambda a, b: Sym(binary("div", _lift(a), _lift(b))),
    "floor_divide": lambda a, b: Sym(binary("floordiv", _lift(a), _lift(b))),
    "remainder": lambda a, b: Sym(binary("rem", _lift(a), _lift(b))),
    "mod": lambda a, b: Sym(binary("rem", _lift(a), _lift(b))),
    "power": lambda a, b: Sym(binary("pow", _lift(a), _lift(b))),
    "minimum": minimum,
    "maximum": maximum,
    "less": lambda a, b: Sym(binary("lt", _lift(a), _lift(b))),
    "less_equal": lambda a, b: Sym(binary("le", _lift(a), _lift(b))),
    "greater": lambda a, b: Sym(binary("gt", _lift(a), _lift(b))),
    "greater_equal": lambda a, b: Sym(binary("ge", _lift(a), _lift(b))),
    "equal": lambda a, b: Sym(binary("eq", _lift(a), _lift(b))),
    "not_equal": lambda a, b: Sym(binary("ne", _lift(a), _lift(b))),
    "logical_and": logical_and,
    "logical_or": logical_or,
    "logical_not": logical_not,
    "bitwise_and": lambda a, b: Sym(binary("and", _lift(a), _lift(b))),
    "bitwise_or": lambda a, b: Sym(binary("or", _lift(a), _lift(b))),
    "bitwise_xor": lambda a, b: Sym(binary("xor", _lift(a), _lift(b))),
    "negative": lambda a: Sym(unary("neg", _lift(a))),
    "absolute": abs,
    "exp": exp, "exp2": exp2, "log": log, "log2": log2, "sqrt": sqrt, "tanh": tanh,
    "sin": sin, "cos": cos, "floor": floor, "ceil": ceil, "sign": sign,
    "isinf": isinf, "isnan": isnan,
}

_TORCH_FUNCS = {
    "where": where, "exp": exp, "exp2": exp2, "log": log, "log2": log2, "sqrt": sqrt,
    "rsqrt": rsqrt, "tanh": tanh, "sigmoid": sigmoid, "sin": sin, "cos": cos, "abs": abs,
    "floor": floor, "ceil": ceil, "minimum": minimum, "maximum": maximum,
    "remainder": remainder, "logical_and": logical_and, "logical_or": logical_or,
    "logical_not": logical_not, "isneginf": isneginf, "isinf": isinf, "isnan": isnan,
    "sign": sign, "pow": power,
}


# --------------------------------------------------------------------------------------
# tracing entry points
# --------------------------------------------------------------------------------------
def mod_arity(fn: Callable) -> int:
    """Number of parameters without a default: 5 marks a score_mod, 4 a mask_mod
    (flaxattention/core/common.py:20-39)."""
    if type(fn) is types.FunctionType and not fn.__dict__:
        code = fn.__code__
        if not code.co_flags & (inspect.CO_VARARGS | inspect.CO_VARKEYWORDS) and not code.co_kwonlyargcount:
            return code.co_argcount - len(fn.__defaults__ or ())  # what inspect.signature takes 10 us to find
    return sum(
        1 for p in inspect.signature(fn).parameters.values() if p.default is inspect.Parameter.empty
    )


class TracedMod:
    """Result of tracing: ``kind`` is 'score' (float32 result) or 'mask' (bool result)."""

    def __init__(self, kind: str, root: Expr, buffers: Optional[List[object]] = None):
        self.kind = kind
        self.root = root
        self.buffers = buffers  # captured tensors the load nodes refer to (shared by a mod pair)

    @property
    def is_identity(self) -> bool:
        return self.kind == "score" and self.root.op == "score"

    @property
    def is_all_true(self) -> bool:
        return self.kind == "mask" and self.root.op == "const" and bool(self.root.value)

    def uses_score(self) -> bool:
        return _depends_on_score(self.root, {})


def _leaf_syms():
    return tuple(Sym(_B.leaf(n)) for n in _LEAVES)


def _traced(buffers: Optional[List[object]], run: Callable[[], Expr], kind: str) -> TracedMod:
    """Runs a trace with `buffers` as the registry that tensor[traced index] fills."""
    global _TRACE_BUFFERS
    bufs = [] if buffers is None else buffers
    prev, _TRACE_BUFFERS = _TRACE_BUFFERS, bufs
    try:
        root = run()
    finally:
        _TRACE_BUFFERS = prev
    return TracedMod(kind, root, bufs)


def trace_score_mod(fn: Callable, buffers: Optional[List[object]] = None) -> TracedMod:
    def run():
        s, b, h, q, kv = _leaf_syms()
        return cast(_lift(fn(s, b, h, q, kv)), F32)

    return _traced(buffers, run, "score")


def trace_mask_mod(fn: Callable, buffers: Optional[List[object]] = None) -> TracedMod:
    """Traces a mask_mod.  A 5-argument function is accepted as well and is then a
    score_mod evaluated on a zero score whose -inf results mark masked positions, the
    rule ``create_mask`` applies (flaxattention/core/blockmask.py:303-315)."""
    def run():
        s, b, h, q, kv = _leaf_syms()
        if mod_arity(fn) == 5:
            out = fn(Sym(_B.const(0.0, F32)), b, h, q, kv)
            return unary("not", unary("isneginf", cast(_lift(out), F32)))
        return cast(_lift(fn(b, h, q, kv)), B1)

    return _traced(buffers, run, "mask")


def _depends_on_score(e: Expr, memo) -> bool:
    r = memo.get(id(e))
    if r is None:
        r = e.op == "score" or any(_depends_on_score(a, memo) for a in e.args)
        memo[id(e)] = r
    return r


# --------------------------------------------------------------------------------------
# symbolic derivative with respect to the score
# --------------------------------------------------------------------------------------
def derivative(mod: TracedMod) -> TracedMod:
    if mod.kind != "score":
        raise ValueError("only a score_mod has a derivative")
    dep: Dict[int, bool] = {}
    memo: Dict[int, Expr] = {}
    zero, one = _B.const(0.0, F32), _B.const(1.0, F32)

    def d(e: Expr) -> Expr:
        if not _depends_on_score(e, dep):
            return zero
        got = memo.get(id(e))
        if got is not None:
            return got
        op, a = e.op, e.args
        if op == "score":
            r = one
        elif op == "add":
            r = binary("add", d(a[0]), d(a[1]))
        elif op == "sub":
            r = binary("sub", d(a[0]), d(a[1]))
        elif op == "neg":
            r = unary("neg", d(a[0]))
        elif op == "mul":
            r = binary("add", binary("mul", d(a[0]), a[1]), binary("mul", a[0], d(a[1])))
        elif op == "div":
            # (u/v)' = u'/v - u v'/v^2
            t1 = binary("div", d(a[0]), a[1])
            dv = d(a[1])
            if _is_const(dv, 0):
                r = t1
            else:
                r = binary("sub", t1, binary("div", binary("mul", a[0], dv), binary("mul", a[1], a[1])))
        elif op == "exp":
            r = binary("mul", e, d(a[0]))
        elif op == "exp2":
            r = binary("mul", binary("mul", e, _B.const(math.log(2.0), F32)), d(a[0]))
        elif op == "log":
            r = binary("div", d(a[0]), a[0])
        elif op == "log2":
            r = binary("div", d(a[0]), binary("mul", a[0], _B.const(math.log(2.0), F32)))
        elif op == "sqrt":
            r = binary("div", d(a[0]), binary("mul", _B.const(2.0, F32), e))
        elif op == "rsqrt":
            r = binary("mul", binary("mul", _B.const(-0.5, F32), binary("div", e, a[0])), d(a[0]))
        elif op == "tanh":
            r = binary("mul", binary("sub", one, binary("mul", e, e)), d(a[0]))
        elif op == "sigmoid":
            r = binary("mul", binary("mul", e, binary("sub", one, e)), d(a[0]))
        elif op == "sin":
            r = binary("mul", unary("cos", a[0]), d(a[0]))
        elif op == "cos":
            r = unary("neg", binary("mul", unary("sin", a[0]), d(a[0])))
        elif op == "erf":
            g = binary("mul", _B.const(2.0 / math.sqrt(math.pi), F32),
                       unary("exp", unary("neg", binary("mul", a[0], a[0]))))
            r = binary("mul", g, d(a[0]))
        elif op == "abs":
            r = binary("mul", unary("sign", a[0]), d(a[0]))
        elif op == "pow":
            if not _depends_on_score(a[1], dep):
                # u^c: c u^(c-1) u'
                r = binary("mul", binary("mul", a[1], binary("pow", a[0], binary("sub", a[1], one))), d(a[0]))
            else:
                # general: e * (v' ln u + v u'/u)
                r = binary("mul", e, binary("add", binary("mul", d(a[1]), unary("log", a[0])),
                                            binary("div", binary("mul", a[1], d(a[0])), a[0])))
        elif op == "min":
            r = select(binary("le", a[0], a[1]), d(a[0]), d(a[1]))
        elif op == "max":
            r = select(binary("ge", a[0], a[1]), d(a[0]), d(a[1]))
        elif op == "select":
            r = select(a[0], d(a[1]), d(a[2]))
        elif op == "rem":
            # float remainder u - floor(u / c) * c with a divisor that does not depend on the
            # score: piecewise u + const, so the derivative is u'; integer remainders are steps
            if e.dtype == F32 and not _depends_on_score(a[1], dep):
                r = d(a[0])
            else:
                r = zero
        elif op in ("floor", "ceil", "sign", "cast_i32", "cast_b1", "floordiv"):
            r = zero
        elif op == "cast_f32":
            r = zero  # the operand is an integer or bool: piecewise constant
        else:
            raise NotImplementedError(f"no derivative rule for '{op}'")
        memo[id(e)] = r
        return r

    return TracedMod("score", cast(d(mod.root), F32), mod.buffers)


# --------------------------------------------------------------------------------------
# affine decomposition:  score_mod(score, ...) == A(b,h,q,kv) * score + B(b,h,q,kv)
# --------------------------------------------------------------------------------------
def affine_parts(mod: TracedMod):
    """Returns (A, B) as index-only TracedMods when the score_mod is affine in the score
    (bias-type and scaling-type mods: ALiBi, relative biases, checkerboard ...), else None.
    Kernels use it to fold the softmax scale and the log2(e) factor into one FMA per score;
    A is also the derivative with respect to the score."""
    if mod.kind != "score":
        return None
    dep: Dict[int, bool] = {}
    memo: Dict[int, Optional[Tuple[Expr, Expr]]] = {}
    zero, one = _B.const(0.0, F32), _B.const(1.0, F32)
    fail = object()

    def go(e: Expr):
        if not _depends_on_score(e, dep):
            return (zero, cast(e, F32)) if e.dtype != B1 else None
        got = memo.get(id(e), fail)
        if got is not fail:
            return got
        op, a = e.op, e.args
        r = None
        if op == "score":
            r = (one, zero)
        elif op in ("add", "sub"):
            x, y = go(a[0]), go(a[1])
            if x and y:
                r = (binary(op, x[0], y[0]), binary(op, x[1], y[1]))
        elif op == "neg":
            x = go(a[0])
            if x:
                r = (unary("neg", x[0]), unary("neg", x[1]))
        elif op == "mul":
            for u, v in ((a[0], a[1]), (a[1], a[0])):
                if not _depends_on_score(v, dep):
                    x = go(u)
                    if x:
                        k = cast(v, F32)
                        r = (binary("mul", x[0], k), binary("mul", x[1], k))
                    break
        elif op == "div":
            if not _depends_on_score(a[1], dep):
                x = go(a[0])
                if x:
                    r = (binary("div", x[0], a[1]), binary("div", x[1], a[1]))
        elif op == "select":
            if not _depends_on_score(a[0], dep):
                x, y = go(a[1]), go(a[2])
                if x and y:
                    r = (select(a[0], x[0], y[0]), select(a[0], x[1], y[1]))
        memo[id(e)] = r
        return r

    res = go(mod.root)
    if res is None:
        return None
    return TracedMod("score", cast(res[0], F32), mod.buffers), TracedMod("score", cast(res[1], F32), mod.buffers)


# --------------------------------------------------------------------------------------
# index-linear biases:  B(b,h,q,kv) == B(.., x0) + (x - x0) * S(b,h,other index)   for x in {q, kv}
# --------------------------------------------------------------------------------------
def _depends_on(e: Expr, leaf: str, memo) -> bool:
    r = memo.get(id(e))
    if r is None:
        r = e.op == leaf or any(_depends_on(a, leaf, memo) for a in e.args)
        memo[id(e)] = r
    return r


def _int_bound(e: Expr, memo) -> float:
    """Upper bound of |value| of an integer expression made of indices (below 2^16 each), constants,
    +, - and *; infinity for anything else."""
    got = memo.get(id(e))
    if got is not None:
        return got
    if e.op in ("b", "h", "q", "kv"):
        r = float(1 << 16)
    elif e.op == "const" and e.dtype == I32:
        r = float(abs(int(e.value)))
    elif e.op in ("add", "sub") and e.dtype == I32:
        r = _int_bound(e.args[0], memo) + _int_bound(e.args[1], memo)
    elif e.op == "neg" and e.dtype == I32:
        r = _int_bound(e.args[0], memo)
    elif e.op == "mul" and e.dtype == I32:
        r = _int_bound(e.args[0], memo) * _int_bound(e.args[1], memo)
    else:
        r = float("inf")
    memo[id(e)] = r
    return r


def linear_slope(root: Expr, leaf: str) -> Optional[Expr]:
    """If the float expression ``root`` is linear in the index ``leaf`` ('q' or 'kv') - relative-position
    biases such as ALiBi are - returns its slope, an expression that does not read ``leaf``; else None.
    A kernel that walks along that index then evaluates the bias once per tile and adds multiples of
    the slope, instead of an integer subtraction, an int-to-float conversion (which shares the
    special-function unit with the exponentials) and a multiplication per element.
    Integer sub-expressions must stay below 2^24 in magnitude so that their conversion to float is
    exact term by term."""
    dep: Dict[int, bool] = {}
    bounds: Dict[int, float] = {}
    memo: Dict[int, object] = {}
    fail = object()

    def go(e: Expr):
        """slope of e (Expr of e's dtype, independent of leaf), or None when e is not linear in leaf"""
        if not _depends_on(e, leaf, dep):
            return _B.const(0, I32) if e.dtype == I32 else _B.const(0.0, F32)
        got = memo.get(id(e), fail)
        if got is not fail:
            return got
        op, a, r = e.op, e.args, None
        if e.dtype not in (I32, F32):
            r = None
        elif op == leaf:
            r = _B.const(1, I32)
        elif op in ("add", "sub"):
            x, y = go(a[0]), go(a[1])
            if x is not None and y is not None:
                r = binary(op, cast(x, e.dtype), cast(y, e.dtype))
        elif op == "neg":
            x = go(a[0])
            if x is not None:
                r = unary("neg", x)
        elif op == "mul":
            for u, v in ((a[0], a[1]), (a[1], a[0])):
                if not _depends_on(v, leaf, dep):
                    x = go(u)
                    if x is not None:
                        r = binary("mul", cast(x, e.dtype), v)
                    break
        elif op == "div" and e.dtype == F32:
            if not _depends_on(a[1], leaf, dep):
                x = go(a[0])
                if x is not None:
                    r = binary("div", cast(x, F32), a[1])
        elif op == "cast_f32" and a[0].dtype == I32:
            x = go(a[0])
            if x is not None and _int_bound(a[0], bounds) < float(1 << 24):
                r = cast(x, F32)
        memo[id(e)] = r
        return r

    res = go(root)
    if res is None:
        return None
    return cast(res, F32)


# --------------------------------------------------------------------------------------
# back ends
# --------------------------------------------------------------------------------------
def _topo(root: Expr) -> List[Expr]:
    order: List[Expr] = []
    seen = set()
    stack = [(root, False)]
    while stack:
        e, done = stack.pop()
        if done:
            order.append(e)
            continue
        if id(e) in seen:
            continue
        seen.add(id(e))
        stack.append((e, True))
        for a in reversed(e.args):
            if id(a) not in seen:
                stack.append((a, False))
    return order


import os as _os

_MAGIC_I2F = _os.environ.get("FLAXATTN_MAGIC_I2F", "0") == "1"
_IDX_BOUND = 1 << 21  # q, kv, b, h are taken to lie in [0, 2^21): sequences of up to 2M tokens


def _int_range(e: Expr, memo: Dict[int, Optional[Tuple[int, int]]]) -> Optional[Tuple[int, int]]:
    """Conservative value range of an int32 expression, or None when unknown."""
    got = memo.get(id(e), 0)
    if got != 0:
        return got
    r = None
    if e.dtype == I32:
        if e.op == "const":
            r = (e.value, e.value)
        elif e.op in ("q", "kv", "b", "h"):
            r = (0, _IDX_BOUND - 1)
        elif e.op in ("add", "sub"):
            a, b = _int_range(e.args[0], memo), _int_range(e.args[1], memo)
            if a and b:
                r = (a[0] + b[0], a[1] + b[1]) if e.op == "add" else (a[0] - b[1], a[1] - b[0])
        elif e.op == "neg":
            a = _int_range(e.args[0], memo)
            if a:
                r = (-a[1], -a[0])
        elif e.op == "and" and (_is_bit(e) or (e.args[1].op == "const" and e.args[1].value >= 0)):
            r = (0, 1) if _is_bit(e) else (0, e.args[1].value)
        elif e.op in ("xor", "or") and _is_bit(e):
            r = (0, 1)
        elif e.op == "cast_i32" and e.args[0].dtype == B1:
            r = (0, 1)
        elif e.op in ("min", "max"):
            a, b = _int_range(e.args[0], memo), _int_range(e.args[1], memo)
            if a and b:
                f = min if e.op == "min" else max
                r = (f(a[0], b[0]), f(a[1], b[1]))
        elif e.op == "abs":
            a = _int_range(e.args[0], memo)
            if a:
                r = (0, max(abs(a[0]), abs(a[1])))
    memo[id(e)] = r
    return r


def _float_range(e: Expr, memo: Dict[int, Optional[Tuple[float, float]]], ints: Dict[int, Optional[Tuple[int, int]]]) -> Optional[Tuple[float, float]]:
    """Conservative value range of an fp32 expression that is neither infinite nor NaN at any position (indices below
    ``_IDX_BOUND``), or None when that is not known.  A range in ``memo`` for the score leaf counts for it."""
    got = memo.get(id(e), 0)
    if got != 0:
        return got
    r = None
    if e.op == "const":
        r = (float(e.value), float(e.value))
    elif e.op == "cast_f32":
        a = e.args[0]
        r = (0.0, 1.0) if a.dtype == B1 else (_int_range(a, ints) or (-2.0 ** 31, 2.0 ** 31)) if a.dtype == I32 else None
    elif e.op == "select":
        a, b = (_float_range(x, memo, ints) for x in e.args[1:])
        if a and b:
            r = (min(a[0], b[0]), max(a[1], b[1]))
    elif e.op in ("add", "sub", "mul", "div", "min", "max", "neg", "abs", "exp", "exp2", "tanh", "sigmoid", "sin", "cos"):
        x = [_float_range(a, memo, ints) if a.dtype == F32 else None for a in e.args]
        if all(x):
            (lo, hi), (lo2, hi2) = x[0], x[-1]
            if e.op == "add":
                r = (lo + lo2, hi + hi2)
            elif e.op == "sub":
                r = (lo - hi2, hi - lo2)
            elif e.op == "mul":
                p = (lo * lo2, lo * hi2, hi * lo2, hi * hi2)
                r = (min(p), max(p))
            elif e.op == "div":
                if lo2 > 1e-30 or hi2 < -1e-30:
                    p = (lo / lo2, lo / hi2, hi / lo2, hi / hi2)
                    r = (min(p), max(p))
            elif e.op in ("min", "max"):
                f = min if e.op == "min" else max
                r = (f(lo, lo2), f(hi, hi2))
            elif e.op == "neg":
                r = (-hi, -lo)
            elif e.op == "abs":
                r = (0.0, max(abs(lo), abs(hi)))
            elif e.op in ("exp", "exp2"):
                r = (0.0, 2.0 ** (1.5 * max(hi, 0.0))) if hi < 60 else None
            elif e.op == "sigmoid":
                r = (0.0, 1.0) if lo > -80 else None
            else:
                r = (-1.0, 1.0)
    if r is not None and not max(abs(r[0]), abs(r[1])) <= 1e30:
        r = None
    memo[id(e)] = r
    return r


def always_finite(roots, score_is_zero: bool) -> bool:
    """Whether the fp32 expressions are finite at every position: for any score, or for a score of zero."""
    for root in roots:
        memo = {id(x): (0.0, 0.0) for x in _topo(root) if x.op == "score"} if score_is_zero else {}
        if _float_range(root, memo, {}) is None:
            return False
    return True


_CTYPE = {I32: "int", F32: "float", B1: "bool"}


def _f32_literal(v: float) -> str:
    if math.isnan(v):
        return "__int_as_float(0x7fc00000)"
    if math.isinf(v):
        return "__int_as_float(0x7f800000)" if v > 0 else "__int_as_float(0xff800000)"
    return float(np.float32(v)).hex() + "f"


_CUDA_BIN = {
    "add": "({0} + {1})", "sub": "({0} - {1})", "mul": "({0} * {1})",
    "lt": "({0} < {1})", "le": "({0} <= {1})", "gt": "({0} > {1})", "ge": "({0} >= {1})",
    "eq": "({0} == {1})", "ne": "({0} != {1})",
}
_CUDA_UN_F = {
    "exp": "expf({0})", "exp2": "exp2f({0})", "log": "logf({0})", "log2": "log2f({0})",
    "sqrt": "sqrtf({0})", "rsqrt": "(1.0f / sqrtf({0}))", "tanh": "tanhf({0})",
    "sigmoid": "(1.0f / (1.0f + expf(-({0}))))", "sin": "sinf({0})", "cos": "cosf({0})",
    "floor": "floorf({0})", "ceil": "ceilf({0})", "erf": "erff({0})",
}


def to_cuda(mod: TracedMod, name: str) -> str:
    """Device function text.  Signature:
    ``float name(float score, int b, int h, int q, int kv)`` for a score mod (and its
    derivative), ``bool name(int b, int h, int q, int kv)`` for a mask mod."""
    lines: List[str] = []
    names: Dict[int, str] = {}
    ranges: Dict[int, Optional[Tuple[int, int]]] = {}
    n = 0
    for e in _topo(mod.root):
        if e.op in _LEAVES:
            names[id(e)] = e.op
            continue
        if e.op == "const":
            if e.dtype == F32:
                names[id(e)] = _f32_literal(e.value)
            elif e.dtype == I32:
                names[id(e)] = f"({e.value})" if e.value != -(1 << 31) else "(-2147483647 - 1)"
            else:
                names[id(e)] = "true" if e.value else "false"
            continue
        a = [names[id(x)] for x in e.args]
        t = e.dtype
        op = e.op
        if op in _CUDA_BIN:
            if t == I32 and op in ("add", "sub", "mul"):
                # wrap-around int32 arithmetic without signed-overflow UB
                sym = {"add": "+", "sub": "-", "mul": "*"}[op]
                rhs = f"(int)((unsigned){a[0]} {sym} (unsigned){a[1]})"
            else:
                rhs = _CUDA_BIN[op].format(*a)
        elif op == "div":
            rhs = f"({a[0]} / {a[1]})"
        elif op == "floordiv":
            rhs = f"fa_floordiv_i32({a[0]}, {a[1]})" if t == I32 else f"floorf({a[0]} / {a[1]})"
        elif op == "rem":
            rhs = f"fa_pymod_i32({a[0]}, {a[1]})" if t == I32 else f"fa_pymod_f32({a[0]}, {a[1]})"
        elif op == "pow":
            rhs = f"powf({a[0]}, {a[1]})"
        elif op == "min":
            rhs = f"min({a[0]}, {a[1]})" if t == I32 else f"fminf({a[0]}, {a[1]})"
        elif op == "max":
            rhs = f"max({a[0]}, {a[1]})" if t == I32 else f"fmaxf({a[0]}, {a[1]})"
        elif op == "and":
            rhs = f"({a[0]} && {a[1]})" if t == B1 else f"({a[0]} & {a[1]})"
        elif op == "or":
            rhs = f"({a[0]} || {a[1]})" if t == B1 else f"({a[0]} | {a[1]})"
        elif op == "xor":
            rhs = f"({a[0]} != {a[1]})" if t == B1 else f"({a[0]} ^ {a[1]})"
        elif op == "shl":
            rhs = f"(int)((unsigned){a[0]} << ({a[1]} & 31))"
        elif op == "shr":
            rhs = f"({a[0]} >> ({a[1]} & 31))"
        elif op == "neg":
            rhs = f"(-{a[0]})" if t == F32 else f"(int)(0u - (unsigned){a[0]})"
        elif op == "not":
            rhs = f"(!{a[0]})" if t == B1 else f"(~{a[0]})"
        elif op == "abs":
            rhs = f"fabsf({a[0]})" if t == F32 else f"abs({a[0]})"
        elif op == "sign":
            if t == F32:
                rhs = f"(({a[0]} > 0.0f) ? 1.0f : (({a[0]} < 0.0f) ? -1.0f : {a[0]}))"
            else:
                rhs = f"(({a[0]} > 0) - ({a[0]} < 0))"
        elif op == "isneginf":
            rhs = f"({a[0]} == __int_as_float(0xff800000))"
        elif op == "isinf":
            rhs = f"(fabsf({a[0]}) == __int_as_float(0x7f800000))"
        elif op == "isnan":
            rhs = f"({a[0]} != {a[0]})"
        elif op in _CUDA_UN_F:
            rhs = _CUDA_UN_F[op].format(*a)
        elif op == "select":
            rhs = f"({a[0]} ? {a[1]} : {a[2]})"
        elif op == "cast_f32":
            if e.args[0].dtype == I32:
                rg = _int_range(e.args[0], ranges)
                if _MAGIC_I2F and rg is not None and -(1 << 22) < rg[0] and rg[1] < (1 << 22):
                    # exact int -> float for |x| < 2^22 with an integer add and a float subtract
                    # (1.5 * 2^23 has the integer x in its low mantissa bits): keeps the
                    # conversion off the special-function unit the softmax exponentials need
                    rhs = f"(__int_as_float(0x4B400000 + {a[0]}) - 12582912.0f)"
                else:
                    rhs = f"(float)({a[0]})"
            else:
                rhs = f"({a[0]} ? 1.0f : 0.0f)"
        elif op == "cast_i32":
            rhs = f"(int)({a[0]})" if e.args[0].dtype == F32 else f"({a[0]} ? 1 : 0)"
        elif op == "cast_b1":
            rhs = f"({a[0]} != 0)" if e.args[0].dtype == I32 else f"({a[0]} != 0.0f)"
        elif op == "load":
            k, span, elem = e.value
            rhs = f"fa_ld_{elem}({k}, min(max({a[0]}, 0), {span - 1}))"
            if t == B1:
                rhs = f"({rhs} != 0)"
        else:
            raise NotImplementedError(op)
        var = f"t{n}"
        n += 1
        lines.append(f"  const {_CTYPE[t]} {var} = {rhs};")
        names[id(e)] = var
    ret = names[id(mod.root)]
    if mod.kind == "score":
        head = f"__device__ __forceinline__ float {name}(float score, int b, int h, int q, int kv) {{"
    else:
        head = f"__device__ __forceinline__ bool {name}(int b, int h, int q, int kv) {{"
    return "\n".join([head] + lines + [f"  return {ret};", "}"]) + "\n"


class _RangeText:
    """What ``_range_walk`` builds from: C++ text, a line for each pair of bounds."""

    true, false = "true", "false"

    def __init__(self):
        self.lines: List[str] = []

    def keep(self, pair, ctype):
        i = len(self.lines)
        a, b = f"a{i}", f"z{i}"
        self.lines.append(f"  const {ctype} {a} = {pair[0]}, {b} = {pair[1]};")
        return a, b

    def index(self, name):
        return (name + "0", name + "1") if name in ("q", "kv") else (name, name)

    def const(self, v):
        return f"({v})" if v != -(1 << 31) else "(-2147483647 - 1)"

    def op(self, sign, u, v):
        return f"{u} {sign} {v}"

    def neg(self, u):
        return f"-{u}"

    def min(self, u, v):
        return f"min({u}, {v})"

    def max(self, u, v):
        return f"max({u}, {v})"

    def floordiv(self, u, c):
        return f"fa_floordiv_i32({u}, {c})"

    def pymod(self, u, c):
        return f"fa_pymod_i32({u}, {c})"

    def where(self, c, u, v):
        return f"{c} ? {u} : {v}"

    def all(self, *x):
        return " && ".join(x)

    def any(self, *x):
        return " || ".join(x)

    def par(self, u):
        return f"({u})"


class _RangeNumpy:
    """The same on arrays of rectangles (bounds in int64: nothing that is kept leaves int32)."""

    true, false = np.bool_(True), np.bool_(False)
    _OPS = {"+": np.add, "-": np.subtract, "*": np.multiply, ">>": np.right_shift, "<": np.less, "<=": np.less_equal,
            ">": np.greater, ">=": np.greater_equal, "==": np.equal}
    neg, min, max, const = staticmethod(np.negative), staticmethod(np.minimum), staticmethod(np.maximum), staticmethod(np.int64)
    floordiv, pymod, where = staticmethod(np.floor_divide), staticmethod(np.remainder), staticmethod(np.where)

    def __init__(self, q, kv):
        self._index = {"q": q, "kv": kv}

    def keep(self, pair, ctype):
        return pair

    def index(self, name):
        return self._index[name]

    def op(self, sign, u, v):
        return self._OPS[sign](u, v)

    def all(self, *x):
        return functools.reduce(np.logical_and, x)

    def any(self, *x):
        return functools.reduce(np.logical_or, x)

    def par(self, u):
        return u


def _range_walk(mod: TracedMod, K):
    """What a mask is over a rectangle of positions, by interval arithmetic on its graph: the pair (certainly true, certainly false)
    in the terms of K, None if it would never be told.

    An integer node is a pair of bounds, a boolean one a pair (certainly true, certainly false); floats, loads from
    captured tensors and whatever else has no rule here (a remainder by a power of two is a bitwise and) is unknown.  A node whose values could leave int32 for indices below
    ``_IDX_BOUND`` is unknown too (the arithmetic of the mask wraps there)."""
    env: Dict[int, Optional[tuple]] = {}  # int: (lo, hi, static lo, static hi); bool: (true, false)

    def integer(lo, hi, slo, shi):
        if slo < -(1 << 31) or shi >= 1 << 31:
            return None
        return K.keep((lo, hi), "int") + (slo, shi)

    for e in _topo(mod.root):
        x = [env.get(id(a)) for a in e.args]
        known = all(v is not None for v in x)
        ints = known and all(a.dtype == I32 for a in e.args)
        c = e.args[1].value if len(e.args) == 2 and e.args[1].op == "const" and e.args[1].dtype == I32 else None
        r = None
        op = e.op
        if op in ("q", "kv", "b", "h"):
            r = tuple(K.index(op)) + (0, _IDX_BOUND - 1)
        elif op == "const":
            if e.dtype == I32:
                r = (K.const(e.value), K.const(e.value), e.value, e.value)
            elif e.dtype == B1:
                r = (K.true, K.false) if e.value else (K.false, K.true)
        elif e.dtype == I32 and ints:
            if op == "add":
                r = integer(K.op("+", x[0][0], x[1][0]), K.op("+", x[0][1], x[1][1]), x[0][2] + x[1][2], x[0][3] + x[1][3])
            elif op == "sub":
                r = integer(K.op("-", x[0][0], x[1][1]), K.op("-", x[0][1], x[1][0]), x[0][2] - x[1][3], x[0][3] - x[1][2])
            elif op == "neg":
                r = integer(K.neg(x[0][1]), K.neg(x[0][0]), -x[0][3], -x[0][2])
            elif op in ("min", "max"):
                f, g = (min, K.min) if op == "min" else (max, K.max)
                r = integer(g(x[0][0], x[1][0]), g(x[0][1], x[1][1]), f(x[0][2], x[1][2]), f(x[0][3], x[1][3]))
            elif op == "abs":
                m = max(abs(x[0][2]), abs(x[0][3]))
                lo, hi = x[0][:2]
                least = K.par(K.where(K.op(">", lo, 0), lo, K.par(K.where(K.op("<", hi, 0), K.neg(hi), 0))))
                r = integer(least, K.max(K.neg(lo), hi), 0, m) if m < 1 << 31 else None
            elif op == "mul" and (c is not None or (e.args[0].op == "const")):
                k, y = (c, x[0]) if c is not None else (e.args[0].value, x[1])
                lo, hi = (y[0], y[1]) if k >= 0 else (y[1], y[0])
                r = integer(K.op("*", lo, K.const(k)), K.op("*", hi, K.const(k)), min(y[2] * k, y[3] * k), max(y[2] * k, y[3] * k)) if k != -(1 << 31) else None
            elif op == "floordiv" and c is not None and c > 0:
                r = integer(K.floordiv(x[0][0], c), K.floordiv(x[0][1], c), x[0][2] // c, x[0][3] // c)
            elif op == "rem" and c is not None and c > 0:
                same = K.par(K.op("==", K.floordiv(x[0][0], c), K.floordiv(x[0][1], c)))
                r = integer(K.where(same, K.pymod(x[0][0], c), 0), K.where(same, K.pymod(x[0][1], c), c - 1), 0, c - 1)
            elif op == "shr" and c is not None and 0 <= c < 32:
                r = integer(K.op(">>", x[0][0], c), K.op(">>", x[0][1], c), x[0][2] >> c, x[0][3] >> c)
        elif e.dtype == I32 and op == "select" and known and e.args[0].dtype == B1:
            (t, f), u, v = x
            r = integer(K.where(t, u[0], K.par(K.where(f, v[0], K.min(u[0], v[0])))), K.where(t, u[1], K.par(K.where(f, v[1], K.max(u[1], v[1])))),
                        min(u[2], v[2]), max(u[3], v[3]))
        elif e.dtype == B1 and op in ("lt", "le", "gt", "ge", "eq", "ne") and ints:
            u, v = (x[1], x[0]) if op in ("gt", "ge") else (x[0], x[1])
            if op in ("lt", "gt"):
                r = K.keep((K.op("<", u[1], v[0]), K.op(">=", u[0], v[1])), "bool")
            elif op in ("le", "ge"):
                r = K.keep((K.op("<=", u[1], v[0]), K.op(">", u[0], v[1])), "bool")
            else:
                same = K.all(K.op("==", u[0], v[1]), K.op("==", u[1], v[0]))
                apart = K.any(K.op("<", u[1], v[0]), K.op("<", v[1], u[0]))
                r = K.keep((same, apart) if op == "eq" else (apart, same), "bool")
        elif e.dtype == B1 and op in ("and", "or"):
            u, v = (y if y is not None else (K.false, K.false) for y in x)
            if x[0] is not None or x[1] is not None:
                j, k = (K.all, K.any) if op == "and" else (K.any, K.all)
                r = K.keep((j(u[0], v[0]), k(u[1], v[1])), "bool")
        elif e.dtype == B1 and op == "not" and known:
            r = (x[0][1], x[0][0])
        elif e.dtype == B1 and op == "select" and known and all(a.dtype == B1 for a in e.args):
            (t, f), u, v = x
            r = K.keep(tuple(K.any(K.par(K.all(t, u[i])), K.par(K.all(f, v[i])), K.par(K.all(u[i], v[i]))) for i in (0, 1)), "bool")
        elif op == "cast_b1" and ints:
            r = K.keep((K.any(K.op(">", x[0][0], 0), K.op("<", x[0][1], 0)), K.all(K.op("==", x[0][0], 0), K.op("==", x[0][1], 0))), "bool")
        elif op == "cast_i32" and known and e.args[0].dtype == B1:
            r = integer(K.where(x[0][0], 1, 0), K.where(x[0][1], 0, 1), 0, 1)
        env[id(e)] = r
    return env[id(mod.root)]


def to_cuda_range(mod: TracedMod, name: str) -> Optional[str]:
    """Device function text of ``_range_walk``: ``int name(int b, int h, int q0, int q1, int kv0, int kv1)`` (bounds inclusive)
    gives 0 where the mask is false for every position, 2 where it is true for every one, 1 where the intervals do not tell
    and for rectangles beyond ``_IDX_BOUND``.  None if they never would."""
    K = _RangeText()
    root = _range_walk(mod, K)
    if root is None:
        return None
    bound = " || ".join(f"(unsigned){v} >= {_IDX_BOUND}u" for v in ("b", "h", "q0", "q1", "kv0", "kv1"))
    return "\n".join([f"__device__ __forceinline__ int {name}(int b, int h, int q0, int q1, int kv0, int kv1) {{",
                      f"  if ({bound}) return 1;"] + K.lines + [f"  return {root[0]} ? 2 : ({root[1]} ? 0 : 1);", "}"]) + "\n"


def _buffer_storage(buf, span: int) -> np.ndarray:
    """The first `span` elements of the storage behind a captured tensor (strided view undone)."""
    try:
        import torch

        if isinstance(buf, torch.Tensor):
            return torch.as_strided(buf.detach().cpu(), (span,), (1,)).numpy()
    except ImportError:  # pragma: no cover
        pass
    a = np.asarray(buf)
    return np.lib.stride_tricks.as_strided(a, (span,), (a.itemsize,))


def evaluate(mod: TracedMod, score, b, h, q, kv):
    """Numpy evaluation of the graph on broadcastable arrays (int32 indices, float32 score)."""
    env: Dict[int, np.ndarray] = {}
    leaves = {
        "score": None if score is None else np.asarray(score, dtype=np.float32),
        "b": np.asarray(b, dtype=np.int32), "h": np.asarray(h, dtype=np.int32),
        "q": np.asarray(q, dtype=np.int32), "kv": np.asarray(kv, dtype=np.int32),
    }
    npdt = {I32: np.int32, F32: np.float32, B1: np.bool_}
    with np.errstate(all="ignore"):
        for e in _topo(mod.root):
            op = e.op
            if op in _LEAVES:
                env[id(e)] = leaves[op]
                continue
            if op == "const":
                env[id(e)] = npdt[e.dtype](e.value)
                continue
            a = [env[id(x)] for x in e.args]
            t = npdt[e.dtype]
            if op == "add":
                r = a[0] + a[1]
            elif op == "sub":
                r = a[0] - a[1]
            elif op == "mul":
                r = a[0] * a[1]
            elif op == "div":
                r = np.float32(a[0]) / np.float32(a[1]) if np.ndim(a[0]) == 0 and np.ndim(a[1]) == 0 else a[0] / a[1]
            elif op == "floordiv":
                r = np.floor_divide(a[0], a[1])
            elif op == "rem":
                r = np.remainder(a[0], a[1])
            elif op == "pow":
                r = np.power(a[0], a[1])
            elif op == "min":
                r = np.minimum(a[0], a[1])
            elif op == "max":
                r = np.maximum(a[0], a[1])
            elif op == "and":
                r = np.logical_and(a[0], a[1]) if e.dtype == B1 else a[0] & a[1]
            elif op == "or":
                r = np.logical_or(a[0], a[1]) if e.dtype == B1 else a[0] | a[1]
            elif op == "xor":
                r = np.logical_xor(a[0], a[1]) if e.dtype == B1 else a[0] ^ a[1]
            elif op == "shl":
                r = a[0] << (a[1] & 31)
            elif op == "shr":
                r = a[0] >> (a[1] & 31)
            elif op in ("lt", "le", "gt", "ge", "eq", "ne"):
                r = {"lt": np.less, "le": np.less_equal, "gt": np.greater, "ge": np.greater_equal,
                     "eq": np.equal, "ne": np.not_equal}[op](a[0], a[1])
            elif op == "neg":
                r = -a[0]
            elif op == "not":
                r = np.logical_not(a[0]) if e.dtype == B1 else ~a[0]
            elif op == "abs":
                r = np.abs(a[0])
            elif op == "sign":
                r = np.sign(a[0])
            elif op == "isneginf":
                r = np.isneginf(a[0])
            elif op == "isinf":
                r = np.isinf(a[0])
            elif op == "isnan":
                r = np.isnan(a[0])
            elif op == "sigmoid":
                r = 1.0 / (1.0 + np.exp(-a[0]))
            elif op == "rsqrt":
                r = 1.0 / np.sqrt(a[0])
            elif op == "erf":
                from scipy.special import erf as _erf

                r = _erf(a[0])
            elif op in _UNARY_F:
                r = getattr(np, op)(a[0])
            elif op == "select":
                r = np.where(a[0], a[1], a[2])
            elif op.startswith("cast_"):
                r = a[0] != 0 if e.dtype == B1 else a[0]
            elif op == "load":
                k, span, _elem = e.value
                if mod.buffers is None:
                    raise ValueError("this mod reads captured buffers; evaluate a mod obtained from lower_mods")
                r = _buffer_storage(mod.buffers[k], span)[np.clip(np.asarray(a[0], dtype=np.int64), 0, span - 1)]
            else:
                raise NotImplementedError(op)
            env[id(e)] = np.asarray(r).astype(t, copy=False)
    return env[id(mod.root)]


_PRELUDE = r"""
__device__ __forceinline__ int fa_pymod_i32(int a, int b) {
  if (b == 0) return 0;
  if (b == -1) return 0;
  int r = a % b;
  return (r != 0 && ((r ^ b) < 0)) ? r + b : r;
}
__device__ __forceinline__ int fa_floordiv_i32(int a, int b) {
  if (b == 0) return 0;
  if (b == -1) return (int)(0u - (unsigned)a);
  int q = a / b;
  int r = a - q * b;
  return (r != 0 && ((r ^ b) < 0)) ? q - 1 : q;
}
__device__ __forceinline__ float fa_pymod_f32(float a, float b) {
  float r = fmodf(a, b);
  return (r != 0.0f && ((r < 0.0f) != (b < 0.0f))) ? r + b : r;
}
"""


_BUFFER_PRELUDE = r"""
// Captured buffers: every kernel fills this table from its parameters (FA_MOD_BUFS_INIT).
__shared__ const void* fa_mod_buf[FA_NUM_MOD_BUFS];
__device__ __forceinline__ int fa_ld_i32(int k, int i) { return __ldg((const int*)fa_mod_buf[k] + i); }
__device__ __forceinline__ int fa_ld_i64(int k, int i) { return (int)__ldg((const long long*)fa_mod_buf[k] + i); }
__device__ __forceinline__ int fa_ld_u8(int k, int i) { return (int)__ldg((const unsigned char*)fa_mod_buf[k] + i); }
__device__ __forceinline__ float fa_ld_f32(int k, int i) { return __ldg((const float*)fa_mod_buf[k] + i); }
"""


class ModSet:
    """The (score_mod, mask_mod) pair of one attention call, lowered.

    ``source`` is the device-code fragment: helper functions plus ``fa_score_mod``,
    ``fa_score_mod_grad`` and ``fa_mask_mod`` together with the ``FA_HAS_*`` macros the
    kernel templates test.  ``key`` is a SHA-256 of that text, used as the cache key of
    compiled kernels and of this object.
    """

    def __init__(self, score: Optional[TracedMod], mask: Optional[TracedMod], buffers: Optional[List[object]] = None):
        self.score = score if (score is not None and not score.is_identity) else None
        self.mask = mask if (mask is not None and not mask.is_all_true) else None
        # tensors the mods close over and index (document ids, learned biases ...); the load
        # nodes of both mods number them in this list
        self.buffers: List[object] = list(buffers) if buffers else []
        parts = [_PRELUDE]
        if self.buffers:
            parts.append(f"#define FA_NUM_MOD_BUFS {len(self.buffers)}\n")
            parts.append(_BUFFER_PRELUDE)
        parts.append(f"#define FA_HAS_SCORE_MOD {1 if self.score is not None else 0}\n")
        parts.append(f"#define FA_HAS_MASK_MOD {1 if self.mask is not None else 0}\n")
        self.affine = None
        if self.score is not None:
            self.grad = derivative(self.score)
            parts.append(to_cuda(self.score, "fa_score_mod"))
            parts.append(to_cuda(self.grad, "fa_score_mod_grad"))
            self.affine = affine_parts(self.score)
            if always_finite([self.affine[0].root if self.affine is not None else self.grad.root], False):
                parts.append("#define FA_SCORE_GRAD_FINITE 1\n")  # (0 times it is 0)
            whole = [t.root for t in self.affine] if self.affine is not None else [self.score.root, self.grad.root]
            if always_finite(whole, True):
                parts.append("#define FA_SCORE_FINITE_AT_0 1\n")  # value and derivative, at a score of 0
            if self.affine is not None:
                # score_mod(s) == fa_score_mul(...) * s + fa_score_add(...); both ignore `score`
                parts.append("#define FA_SCORE_AFFINE 1\n")
                if _is_const(self.affine[0].root, 1):
                    parts.append("#define FA_SCORE_MUL_ONE 1\n")  # nothing but an additive part
                if _is_const(self.affine[1].root, 0):
                    parts.append("#define FA_SCORE_MUL_ONLY 1\n")  # no additive part
                n_ops = sum(1 for t in self.affine for e in _topo(t.root) if e.args)
                if n_ops <= 10:
                    # cheap enough to evaluate twice (row maximum pass and exponent pass) instead of
                    # writing the modified scores back between the passes
                    parts.append("#define FA_SCORE_AFFINE_CHEAP 1\n")
                parts.append(to_cuda(self.affine[0], "fa_score_mul"))
                parts.append(to_cuda(self.affine[1], "fa_score_add"))
                # B already multiplied by log2(e), with the constant folded into row-invariant factors
                b2 = TracedMod("score", binary("mul", self.affine[1].root, _B.const(math.log2(math.e), F32)), self.affine[1].buffers)
                parts.append(to_cuda(b2, "fa_score_add2"))
                # A bias that is linear in kv (q) under a multiplier that does not read kv (q): the kernels
                # take the bias at the first column of a chunk and add multiples of the slope
                self.linear = {}
                for leaf, tag in (("kv", "KV"), ("q", "Q")):
                    slope = linear_slope(b2.root, leaf)
                    if slope is not None and not _depends_on(self.affine[0].root, leaf, {}):
                        self.linear[leaf] = slope
                        parts.append(f"#define FA_SCORE_LINEAR_{tag} 1\n")
                        parts.append(to_cuda(TracedMod("score", slope, b2.buffers), f"fa_score_add2_d{leaf}"))
        else:
            self.grad = None
            parts.append(
                "__device__ __forceinline__ float fa_score_mod(float score, int, int, int, int) { return score; }\n"
                "__device__ __forceinline__ float fa_score_mod_grad(float, int, int, int, int) { return 1.0f; }\n"
            )
        # whether the mask differs between batch entries / heads
        self.mask_reads_b = self.mask is not None and _depends_on(self.mask.root, "b", {})
        self.mask_reads_h = self.mask is not None and _depends_on(self.mask.root, "h", {})
        self._documents = self.mask is not None and bool(self.buffers) and _same_ids(self.mask.root)
        self._kv_tiles: Dict[Tuple[int, int], int] = {}
        if self.mask is not None:
            parts.append(to_cuda(self.mask, "fa_mask_mod"))
            over_range = to_cuda_range(self.mask, "fa_mask_range")
            if over_range is not None:
                parts.append("#define FA_HAS_MASK_RANGE 1\n" + over_range)
        else:
            parts.append("__device__ __forceinline__ bool fa_mask_mod(int, int, int, int) { return true; }\n")
        self.source = "".join(parts)
        self.key = hashlib.sha256(self.source.encode()).hexdigest()

    def kv_tiles(self, Q_LEN: int, KV_LEN: int) -> int:
        """A guess at how many 128-key tiles the mask leaves of the keys per 128 query rows, 0 where there is none: what
        interval arithmetic does not rule out (``_range_walk``), the average over up to eight query tiles.  Masks over captured
        tensors have none, but for document masks: at most eight, as many documents leave.  (Forward, us, two query tiles per
        CTA against the one that eight asks for, head dim 128, B2 H8 S8192: 12 documents 75 / 67, 4 121 / 114, 3 148 / 133, 2 158 / 172.)"""
        if self.mask is None or self.mask_reads_b or self.mask_reads_h or (self.buffers and not self._documents):
            return 0
        n = self._kv_tiles.get((Q_LEN, KV_LEN))
        if n is None:
            try:
                n = self._count_kv_tiles(Q_LEN, KV_LEN)
            except Exception:  # (whatever it is, no result needs the guess)
                n = 0
            if self._documents:
                n = min(n, 8)
            if len(self._kv_tiles) >= 64:
                self._kv_tiles.clear()
            self._kv_tiles[(Q_LEN, KV_LEN)] = n
        return n

    def _count_kv_tiles(self, Q_LEN: int, KV_LEN: int) -> int:
        if not 0 < min(Q_LEN, KV_LEN) <= max(Q_LEN, KV_LEN) <= _IDX_BOUND:
            return 0
        nq, nkv = (Q_LEN + 127) // 128, (KV_LEN + 127) // 128
        q = 128 * np.linspace(0, nq - 1, min(nq, 8)).round().astype(np.int64)[:, None]
        kv = 128 * np.arange(nkv, dtype=np.int64)[None]
        told = _range_walk(self.mask, _RangeNumpy((q, np.minimum(q + 127, Q_LEN - 1)), (kv, np.minimum(kv + 127, KV_LEN - 1))))
        dropped = _RangeNumpy.false if told is None else told[1]
        listed = ~np.broadcast_to(dropped, (len(q), nkv))
        return min(max(int(round(float(listed.sum(axis=1).mean()))), 1), 65535)


def _trace_any(fn: Callable, kind: str, bufs: List[object]) -> TracedMod:
    """Symbolic call first; a mod written with jax.numpy rejects the symbols and is traced through
    its jaxpr instead (jax_frontend), when JAX is installed."""
    try:
        return trace_score_mod(fn, bufs) if kind == "score" else trace_mask_mod(fn, bufs)
    except Exception as first:
        try:
            import jax  # noqa: F401
        except ImportError:
            raise first from None
        from .jax_frontend import trace_with_jax

        try:
            return trace_with_jax(fn, kind)
        except Exception:
            raise first from None


# --------------------------------------------------------------------------------------
# what a mod's trace depends on
# --------------------------------------------------------------------------------------
# A training loop over packed documents makes a new mask_mod for every batch, the same code over
# another tensor.  Tracing and lowering it takes 100-200 us; what the trace can depend on (the code, the
# constants it closes over, shape, strides and type of its tensors) is gone through in about 10, and a pair
# of mods with equal fingerprints shares the lowered text and only brings its own tensors.
# What counts as known is kept narrow, because a miss is silent: names are followed to their values through
# the globals and through modules, functions found there are gone through like the mod itself, and whatever
# is not one of the types below, a function of this module or one of a fixed list of pure functions of
# torch, numpy and math makes the pair one that is traced every time.
@functools.lru_cache(maxsize=1024)
def _code_facts(code):
    """(chains of names the code and the code nested in it look up: a global and the attributes taken of it
    right away, whether it branches on a value, whether it does anything else that reaches outside)."""
    chains, branches, opaque = set(), False, False
    ins = list(dis.get_instructions(code))
    i = 0
    while i < len(ins):
        op, arg = ins[i].opname, ins[i].argval
        i += 1
        if op in ("LOAD_GLOBAL", "LOAD_NAME"):
            chain = [arg]
            while i < len(ins) and ins[i].opname in ("LOAD_ATTR", "LOAD_METHOD"):
                chain.append(ins[i].argval)
                i += 1
            chains.add(tuple(chain))
        elif "JUMP_IF" in op:
            branches = True
        elif op in ("LOAD_ATTR", "LOAD_METHOD", "LOAD_SUPER_ATTR", "IMPORT_NAME", "IMPORT_FROM", "STORE_GLOBAL",
                    "DELETE_GLOBAL", "STORE_ATTR", "DELETE_ATTR", "STORE_NAME", "LOAD_BUILD_CLASS"):
            opaque = True  # a method or an attribute of a value, or state that changes
        elif op == "STORE_DEREF" and arg in code.co_freevars:
            opaque = True
    for c in code.co_consts:
        if isinstance(c, types.CodeType):
            n, br, o = _code_facts(c)
            chains |= set(n)
            branches, opaque = branches or br, opaque or o
    return tuple(sorted(chains)), branches, opaque


class _Unknown(Exception):
    """The trace may depend on something a fingerprint does not cover."""


# functions of numpy and torch that give the same for the same arguments and read nothing else
_PURE = {"torch": frozenset(_TORCH_FUNCS), "numpy": frozenset(_NP_UFUNCS) | {"where", "float32", "int32"}}


class _Fingerprint:
    """What the trace of a mod pair can depend on, gathered in ``parts``, apart from the contents of the
    tensors found on the way (``tensors``); raises ``_Unknown`` where that cannot be said."""

    def __init__(self, *fns):
        self.tensors: List[object] = []
        self.parts: List[object] = []
        self.host_math = False  # calls functions that could turn a tensor into a number
        for fn in fns:
            self.parts.append("|")
            if fn is not None:
                if type(fn) is not types.FunctionType:
                    raise _Unknown
                self.function(fn, 0)
        if self.host_math and self.tensors:
            raise _Unknown
        self.key = tuple(self.parts)

    def value(self, x, depth: int) -> None:
        t = type(x)
        if t is float:
            self.parts.append((t, struct.pack("<d", x)))  # (0.0 == -0.0, and nan != nan)
        elif x is None or t in (bool, int, str, torch.dtype):
            self.parts.append((t, x))
        elif t is types.FunctionType:
            if x.__module__ == __name__:
                self.parts.append(x)  # (by identity, and kept alive by the key)
            else:
                self.function(x, depth + 1)
        elif t in (tuple, list):
            self.parts.append((t, len(x)))
            for y in x:
                self.value(y, depth + 1)
        elif t is torch.Tensor:
            k = next((i for i, y in enumerate(self.tensors) if y is x), len(self.tensors))
            if k == len(self.tensors):
                self.tensors.append(x)
            self.parts.append(("tensor", k, x.dtype, tuple(x.shape), x.stride()))
        else:
            raise _Unknown

    def chain(self, g, names, depth: int) -> None:
        """The value of ``names[0]`` in the globals ``g``, or of an attribute of the module it is."""
        self.parts.append(names)
        if names[0] not in g:
            if names != ("abs",):  # int(tensor), len(...) and the like
                raise _Unknown
            self.parts.append(getattr(builtins, "abs"))
            return
        x, parent, rest = g[names[0]], None, list(names[1:])
        while isinstance(x, types.ModuleType):
            if not rest or rest[0] not in vars(x):
                raise _Unknown
            parent, x = x, vars(x)[rest[0]]
            last = rest.pop(0)
        if rest:
            raise _Unknown  # an attribute of a value
        if parent is not None and (parent is math or last in _PURE.get(parent.__name__, ())) and callable(x):
            self.host_math = self.host_math or parent.__name__ != "torch"
            self.parts.append(x)
        else:
            self.value(x, depth)

    def function(self, fn, depth: int) -> None:
        chains, branches, opaque = _code_facts(fn.__code__)
        if depth > 8 or opaque:
            raise _Unknown
        self.parts.append(fn.__code__)
        before = len(self.tensors)
        for cell in fn.__closure__ or ():
            try:
                self.value(cell.cell_contents, depth)
            except ValueError:  # an empty cell
                raise _Unknown from None
        for d in (fn.__defaults__, tuple(sorted((fn.__kwdefaults__ or {}).items()))):
            self.value(d, depth)
        for names in chains:
            self.chain(fn.__globals__, names, depth)
        if branches and len(self.tensors) > before:
            raise _Unknown  # may branch on the contents of a tensor


class _TensorWatch(TorchDispatchMode):
    """Notices every operation on a tensor.  A trace in which there was none has read no tensor (indexing one
    with a traced value is not an operation on it), so its text holds for other tensors of the same form."""

    used = False

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.used = True
        return func(*args, **(kwargs or {}))


def _same_ids(e: Expr) -> bool:
    """Whether a mask keeps only pairs whose query and key read the same value of a captured tensor (document ids)."""
    if e.op == "and":
        return any(_same_ids(x) for x in e.args)
    if e.op != "eq" or any(x.op != "load" for x in e.args):
        return False
    x, y = e.args
    reads = [(_depends_on(z, "q", {}), _depends_on(z, "kv", {})) for z in (x, y)]
    return x.value == y.value and sorted(reads) == [(False, True), (True, False)]


class _Template:
    """A lowered pair of mods without its tensors."""

    def __init__(self, ms: ModSet, which: List[int]):
        self.ms = copy.copy(ms)
        self.ms.buffers = []
        if ms.buffers:  # the graphs stay, the tensors they were traced over do not
            for name in ("score", "mask"):
                m = getattr(ms, name)
                setattr(self.ms, name, None if m is None else TracedMod(m.kind, m.root))
        self.which = which  # per buffer, its place among the fingerprint's tensors

    def bind(self, tensors: List[object]) -> ModSet:
        ms = copy.copy(self.ms)
        ms.buffers = [tensors[k] for k in self.which]
        return ms


_TEMPLATES: Dict[object, _Template] = {}
# per pair of callables (by identity, 0: no mod), as long as both exist: what keeps track of them, and the lowered pair
_MODSET_CACHE: Dict[Tuple[int, int], Tuple[object, object, ModSet]] = {}
_ON_FORGET: List[Callable[[int, int], None]] = []  # told when a pair leaves the cache


def _forget(key: Tuple[int, int]) -> None:
    _MODSET_CACHE.pop(key, None)
    for f in _ON_FORGET:
        f(*key)


def _hold(fn, key):
    """A callable that gives ``fn``, and that lets the pair's entry go with ``fn``."""
    if fn is None:
        return lambda: None
    try:
        return weakref.ref(fn, lambda _: _forget(key))
    except TypeError:  # no weak references to this type of callable: it stays
        return lambda: fn


def lower_mods(score_mod: Optional[Callable], mask_mod: Optional[Callable]) -> ModSet:
    """Traces and lowers a pair of mods; cached on the identity of the callables (the
    reference keys its jit cache the same way: mods are static arguments,
    flaxattention/core/attention.py:169) for as long as they exist."""
    key = (0 if score_mod is None else id(score_mod), 0 if mask_mod is None else id(mask_mod))
    hit = _MODSET_CACHE.get(key)
    if hit is not None and hit[0]() is score_mod and hit[1]() is mask_mod:
        return hit[2]
    try:
        fp = _Fingerprint(score_mod, mask_mod)
    except _Unknown:
        fp = None
    tpl = _TEMPLATES.get(fp.key) if fp is not None else None
    if tpl is not None:
        ms = tpl.bind(fp.tensors)
    else:
        bufs: List[object] = []
        watch = _TensorWatch()
        with watch if fp is not None else contextlib.nullcontext():
            s = _trace_any(score_mod, "score", bufs) if score_mod is not None else None
            m = _trace_any(mask_mod, "mask", bufs) if mask_mod is not None else None
        ms = ModSet(s, m, bufs)
        if fp is not None and not watch.used:
            which = [next((i for i, t in enumerate(fp.tensors) if t is b), -1) for b in ms.buffers]
            if -1 not in which and len(set(which)) == len(fp.tensors):
                if len(_TEMPLATES) >= 1024:
                    _TEMPLATES.clear()
                _TEMPLATES[fp.key] = _Template(ms, which)
    if len(_MODSET_CACHE) > 4096:
        for k in list(_MODSET_CACHE):
            _forget(k)
    _MODSET_CACHE[key] = (_hold(score_mod, key), _hold(mask_mod, key), ms)
    return ms
