"""BlockMask container and its construction on the GPU.

Mirrors flaxattention/core/blockmask.py: ``BlockMask`` (:72-237), ``create_block_mask``
(:419-455), ``and_masks`` / ``or_masks`` (:372-397), ``noop_mask`` (:20-27).  The dense
``[B,H,Q,KV]`` boolean mask the reference materialises (:277-322) is never built: a CUDA
kernel classifies every block directly from the lowered ``mask_mod`` and a second one
writes the ordered tables.

Table layout (all int32, on the CUDA device):
    kv_num_blocks [B,H,nQ], kv_indices [B,H,nQ,nKV]        blocks that need mask_mod
    full_kv_num_blocks, full_kv_indices                     blocks kept entirely
    q_num_blocks [B,H,nKV], q_indices [B,H,nKV,nQ], full_q_*   the same grid by kv block
Row order is the reference's (stable descending argsort of the 0/1 grid, :57-64): listed
blocks ascending, then the remaining block ids ascending.

Two deliberate differences from the reference, both on fields its own code never reads:
``BLOCK_SIZE`` holds the block sizes actually used (the reference always stores
(128, 128), :452-454), and the q-tables are the true transpose of the kv-tables (the
reference's ``_ordered_to_dense`` drops its scatter result, :46, so its q tables are
always ``num = 0, indices = arange``).  ``reference_q_tables`` reproduces those values.
"""
from __future__ import annotations

import collections
import functools
import operator
from typing import Callable, Optional, Tuple, Union

import torch

from . import _cabi, modtrace
from .modtrace import lower_mods, mod_arity

_DEFAULT_SPARSE_BLOCK_SIZE = 128
_LARGE_SPARSE_BLOCK_SIZE = 1 << 30


def noop_mask(batch, head, token_q, token_kv):
    """Returns a noop mask_mod (everything visible)."""
    return True


def or_masks(*mask_mods: Callable) -> Callable:
    """Returns a mask_mod that's the union of provided mask_mods"""
    if not all(callable(arg) for arg in mask_mods):
        raise RuntimeError(f"All inputs should be callable mask_mods: {mask_mods}")

    def or_mask(b, h, q_idx, kv_idx):
        result = False
        for mask in mask_mods:
            result = result | mask(b, h, q_idx, kv_idx)
        return result

    return or_mask


def and_masks(*mask_mods: Callable) -> Callable:
    """Returns a mask_mod that's the intersection of provided mask_mods"""
    if not all(callable(arg) for arg in mask_mods):
        raise RuntimeError(f"All inputs should be callable mask_mods: {mask_mods}")

    def and_mask(b, h, q_idx, kv_idx):
        result = True
        for mask in mask_mods:
            result = result & mask(b, h, q_idx, kv_idx)
        return result

    return and_mask


def _dense_to_ordered(dense: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    dense = dense.to(torch.int32)
    num = dense.sum(dim=-1).to(torch.int32)
    idx = torch.argsort(dense, dim=-1, descending=True, stable=True).to(torch.int32)
    return num, idx


def _ordered_to_dense(num: torch.Tensor, idx: torch.Tensor) -> torch.Tensor:
    rows, cols = idx.shape[-2], idx.shape[-1]
    dense = torch.zeros(*idx.shape[:-1], cols + 1, dtype=torch.int32, device=idx.device)
    valid = torch.arange(cols, device=idx.device) < num[..., None]
    tgt = torch.where(valid, idx.to(torch.int64), torch.full_like(idx, cols, dtype=torch.int64))
    dense.scatter_(-1, tgt, torch.ones_like(tgt, dtype=torch.int32))
    return dense[..., :cols]


def _transpose_ordered(num: torch.Tensor, idx: torch.Tensor):
    dense = _ordered_to_dense(num, idx)
    return _dense_to_ordered(dense.transpose(-1, -2).contiguous())


def reference_q_tables(kv_indices: torch.Tensor):
    """The q-table values the reference produces for any kv-tables of this shape:
    ``q_num_blocks = 0`` and ``q_indices = arange(nQ)`` (its scatter result is discarded,
    flaxattention/core/blockmask.py:46)."""
    *lead, n_q, n_kv = kv_indices.shape
    num = torch.zeros(*lead, n_kv, dtype=torch.int32, device=kv_indices.device)
    idx = torch.arange(n_q, dtype=torch.int32, device=kv_indices.device).expand(*lead, n_kv, n_q).contiguous()
    return num, idx


class BlockMask:
    kv_num_blocks: torch.Tensor
    kv_indices: torch.Tensor
    full_kv_num_blocks: Optional[torch.Tensor]
    full_kv_indices: Optional[torch.Tensor]
    q_num_blocks: Optional[torch.Tensor]
    q_indices: Optional[torch.Tensor]
    full_q_num_blocks: Optional[torch.Tensor]
    full_q_indices: Optional[torch.Tensor]
    BLOCK_SIZE: Tuple[int, int]
    mask_mod: Callable
    # mask_mod of every position as a bit matrix [1 or B, 1 or H, Q_LEN, words] (int32), or None;
    # not part of the reference's BlockMask: the kernels read it on partial tiles instead of
    # evaluating mask_mod there
    mask_bits: Optional[torch.Tensor] = None
    # the same matrix transposed [1 or B, 1 or H, KV_LEN, words], or None
    mask_bits_t: Optional[torch.Tensor] = None
    _bits_at = (None, None)  # (of objects that were saved without it)
    # a guess at how many 128-key tiles the tables list per 128 query rows, 0 where there is none: a hint for the choice
    # of a kernel variant, no result depends on it
    _kv_tiles = 0

    def __init__(self, kv_num_blocks, kv_indices, full_kv_num_blocks, full_kv_indices, q_num_blocks, q_indices,
                 full_q_num_blocks, full_q_indices, BLOCK_SIZE, mask_mod, mask_bits=None, mask_bits_t=None,
                 _bits_sources=(), _bits_snapshot=None, _bits_at=(None, None)):
        if kv_indices.ndim < 2:
            raise RuntimeError("BlockMask must have at least 2 dimensions")
        assert kv_num_blocks is not None, "kv_num_blocks must be provided"
        assert kv_indices is not None, "kv_indices must be provided"
        assert q_num_blocks is not None, "q_num_blocks must be provided"
        assert q_indices is not None, "q_indices must be provided"
        assert (full_kv_num_blocks is None) == (
            full_kv_indices is None
        ), "full_kv_num_blocks and full_kv_indices must be both provided or omitted"
        assert (full_q_num_blocks is None) == (
            full_q_indices is None
        ), "full_q_num_blocks and full_q_indices must be both provided or omitted"
        self.kv_num_blocks = kv_num_blocks
        self.kv_indices = kv_indices
        self.full_kv_num_blocks = full_kv_num_blocks
        self.full_kv_indices = full_kv_indices
        self.q_num_blocks = q_num_blocks
        self.q_indices = q_indices
        self.full_q_num_blocks = full_q_num_blocks
        self.full_q_indices = full_q_indices
        self.BLOCK_SIZE = BLOCK_SIZE
        self.mask_mod = mask_mod
        self.mask_bits = mask_bits
        self.mask_bits_t = mask_bits_t
        # The bit matrices hold for this mask_mod, and while the tensors it captures are what they were: at
        # these versions, and, because a version does not move with every write (`.data`, other
        # libraries, a replayed graph), byte for byte the same as this copy of them, which every
        # launch that would use the matrices looks at on the device.
        self._bits_mod = mask_mod
        self._bits_sources = _bits_sources
        self._bits_snapshot = _bits_snapshot
        # For batch and heads: the index the first entry of the matrices was made for, None where mask_mod does not
        # read it.  A call with other entries (a broadcast mask over several heads, another offset) evaluates mask_mod.
        self._bits_at = _bits_at

    def bits_hold(self) -> bool:
        """Whether ``mask_bits`` is still what ``mask_mod`` gives, as far as the host can see."""
        return (self.mask_bits is not None and self.mask_mod is self._bits_mod
                and all(t is None or t._version == v for t, v in self._bits_sources))

    def bits_cover(self, B: int, H: int, b_offset: int, h_offset: int) -> bool:
        """Whether the entries of ``mask_bits`` are those of a call over these batch entries and heads."""
        return all(n in (1, size) if at is None else (n == size and at == offset)
                   for n, size, offset, at in zip(self.mask_bits.shape[:2], (B, H), (b_offset, h_offset), self._bits_at))

    def launch_check(self, buffers, stream) -> torch.Tensor:
        """Queues the comparison of the captured tensors (``buffers``, on the device) with the copy taken when
        the bit matrices were built; returns the device word it writes."""
        hold = torch.empty(1, dtype=torch.int32, device=self.mask_bits.device)
        addr, size, n = _cabi.ranges(buffers)
        L = _cabi.lib()
        if int(L.fa_snapshot_bytes(size, n)) == self._bits_snapshot.numel():
            _cabi.check(L.fa_snapshot_holds(addr, size, n, self._bits_snapshot.data_ptr(), hold.data_ptr(), stream))
        else:
            hold.zero_()
        return hold

    @classmethod
    def from_kv_blocks(cls, kv_num_blocks, kv_indices, full_kv_num_blocks=None, full_kv_indices=None,
                       BLOCK_SIZE: Union[int, Tuple[int, int]] = _DEFAULT_SPARSE_BLOCK_SIZE,
                       mask_mod: Optional[Callable] = None):
        if kv_indices.ndim < 2:
            raise RuntimeError("BlockMask must have at least 2 dimensions")
        assert (full_kv_num_blocks is None) == (
            full_kv_indices is None
        ), "full_kv_num_blocks and full_kv_indices must be both provided or omitted"
        q_num_blocks, q_indices = _transpose_ordered(kv_num_blocks, kv_indices)
        if full_kv_num_blocks is not None:
            full_q_num_blocks, full_q_indices = _transpose_ordered(full_kv_num_blocks, full_kv_indices)
        else:
            full_q_num_blocks, full_q_indices = None, None
        if isinstance(BLOCK_SIZE, int):
            BLOCK_SIZE = (BLOCK_SIZE, BLOCK_SIZE)
        mask_mod = mask_mod if mask_mod is not None else noop_mask
        return cls(kv_num_blocks, kv_indices, full_kv_num_blocks, full_kv_indices, q_num_blocks, q_indices,
                   full_q_num_blocks, full_q_indices, BLOCK_SIZE, mask_mod)

    def as_tuple(self, flatten: bool = True):
        """Returns a tuple of the attributes of the BlockMask (mask_mod last).

        Args:
            flatten (bool): If True, the (Q_BLOCK_SIZE, KV_BLOCK_SIZE) pair is flattened.
        """
        block_size = (self.BLOCK_SIZE[0], self.BLOCK_SIZE[1]) if flatten else (self.BLOCK_SIZE,)
        return (
            self.kv_num_blocks, self.kv_indices, self.full_kv_num_blocks, self.full_kv_indices,
            self.q_num_blocks, self.q_indices, self.full_q_num_blocks, self.full_q_indices,
            *block_size, self.mask_mod,
        )

    @property
    def shape(self):
        """Returns the shape of the mask."""
        *batch_dims, _, _ = self.kv_indices.shape
        q_length = self.kv_indices.shape[-2] * self.BLOCK_SIZE[0]
        kv_length = self.kv_indices.shape[-1] * self.BLOCK_SIZE[1]
        return tuple(list(batch_dims) + [q_length, kv_length])

    def numel(self):
        """Returns the number of elements (not accounting for sparsity) in the mask."""
        return functools.reduce(operator.mul, self.shape, 1)

    def sparsity(self) -> float:
        """Computes the percentage of blocks that are sparse (i.e. not computed)"""
        total_size = self.numel()
        computed_blocks = int(self.kv_num_blocks.sum().item())
        if self.full_kv_num_blocks is not None:
            computed_blocks += int(self.full_kv_num_blocks.sum().item())
        computed_size = computed_blocks * self.BLOCK_SIZE[0] * self.BLOCK_SIZE[1]
        return 100 * (1 - computed_size / total_size)

    def computed_blocks(self) -> int:
        """Number of (q block, kv block) pairs an attention call visits."""
        n = int(self.kv_num_blocks.sum().item())
        if self.full_kv_num_blocks is not None:
            n += int(self.full_kv_num_blocks.sum().item())
        return n

    def to(self, device):
        mv = lambda t: None if t is None else t.to(device)  # noqa: E731
        moved = BlockMask(mv(self.kv_num_blocks), mv(self.kv_indices), mv(self.full_kv_num_blocks),
                          mv(self.full_kv_indices), mv(self.q_num_blocks), mv(self.q_indices),
                          mv(self.full_q_num_blocks), mv(self.full_q_indices), self.BLOCK_SIZE, self.mask_mod,
                          *self._moved_bits(mv))
        moved._kv_tiles = self._kv_tiles
        return moved

    def _moved_bits(self, fn):
        """(mask_bits, mask_bits_t, sources, snapshot, first entries) of a copy whose tensors went through ``fn``."""
        if not self.bits_hold():
            return None, None, (), None, (None, None)
        bits, snapshot = fn(self.mask_bits), self._bits_snapshot
        if snapshot is not None and snapshot.device != bits.device:
            snapshot = snapshot.to(bits.device)
        return bits, fn(self.mask_bits_t), self._bits_sources, snapshot, self._bits_at

    def shard(self, b_slice: slice, h_slice: slice) -> "BlockMask":
        """Tables of one batch x heads shard (broadcast axes are kept whole)."""
        def cut(t):
            if t is None:
                return None
            bs = b_slice if t.shape[0] != 1 else slice(None)
            hs = h_slice if t.shape[1] != 1 else slice(None)
            return t[bs, hs].contiguous()
        part = BlockMask(cut(self.kv_num_blocks), cut(self.kv_indices), cut(self.full_kv_num_blocks),
                         cut(self.full_kv_indices), cut(self.q_num_blocks), cut(self.q_indices),
                         cut(self.full_q_num_blocks), cut(self.full_q_indices), self.BLOCK_SIZE, self.mask_mod,
                         *self._moved_bits(cut))
        part._kv_tiles = self._kv_tiles
        if part.mask_bits is not None:
            part._bits_at = tuple(at if at is None or n == 1 else at + range(n)[sl].start
                                  for at, n, sl in zip(self._bits_at, self.mask_bits.shape[:2], (b_slice, h_slice)))
        return part

    def __repr__(self):
        def shape_or_none(x):
            return tuple(x.shape) if x is not None else None

        return (
            f"BlockMask(\n"
            f"    kv_num_blocks={shape_or_none(self.kv_num_blocks)},\n"
            f"    kv_indices={shape_or_none(self.kv_indices)},\n"
            f"    full_kv_num_blocks={shape_or_none(self.full_kv_num_blocks)},\n"
            f"    full_kv_indices={shape_or_none(self.full_kv_indices)},\n"
            f"    q_num_blocks={shape_or_none(self.q_num_blocks)},\n"
            f"    q_indices={shape_or_none(self.q_indices)},\n"
            f"    full_q_num_blocks={shape_or_none(self.full_q_num_blocks)},\n"
            f"    full_q_indices={shape_or_none(self.full_q_indices)},\n"
            f"    BLOCK_SIZE={self.BLOCK_SIZE},\n"
            f"    shape={self.shape},\n"
            f"    sparsity={self.sparsity():.2f}%,\n"
            f"    mask_mod={self.mask_mod.__name__ if hasattr(self.mask_mod, '__name__') else self.mask_mod}\n"
            f")"
        )


def _create_empty_block_mask(query, key) -> BlockMask:
    """Default block mask: one block that spans the whole query and key range
    (flaxattention/core/blockmask.py:240-250)."""
    dev = query.device
    return BlockMask.from_kv_blocks(
        kv_num_blocks=torch.ones([1, 1, 1], dtype=torch.int32, device=dev),
        kv_indices=torch.zeros([1, 1, 1, 1], dtype=torch.int32, device=dev),
        BLOCK_SIZE=_LARGE_SPARSE_BLOCK_SIZE,
    )


def _round_up_to_multiple(x, multiple):
    return (x + multiple - 1) // multiple * multiple


_MODULES = {}


def module_for(score_mod: Optional[Callable], mask_mod: Optional[Callable]):
    """Lowered mods -> compiled-kernel module, cached per generated source.  The pair is also made
    known to the native host path, which then takes calls with it."""
    if mask_mod is noop_mask:
        mask_mod = None
    if score_mod is identity_score:
        score_mod = None
    ms = lower_mods(score_mod, mask_mod)
    m = _MODULES.get(ms.key)
    if m is None:
        m = _cabi.Module(ms.source)
        _MODULES[ms.key] = m
    if all(isinstance(t, torch.Tensor) for t in ms.buffers):
        _cabi.host().register(score_mod, mask_mod, m, m.handle.value, tuple(ms.buffers))
    return m


def identity_score(score, batch, head, token_q, token_kv):
    """The score_mod of a call without one."""
    return score


def _forget_pair(score_id: int, mask_id: int) -> None:
    if _cabi._host is not None:
        _cabi._host.forget(score_id, mask_id)


modtrace._ON_FORGET.append(_forget_pair)


_DEVICE_BUFFERS = {}


def bind_mod_buffers(module, score_mod: Optional[Callable], mask_mod: Optional[Callable], device) -> None:
    """Hands the module the device addresses of the tensors the mods close over and index
    (the reference's score_mod_other_buffers / mask_mod_other_buffers,
    flaxattention/core/attention.py:22-23).  Tensors that live elsewhere (CPU, another GPU) are
    copied to `device` once per tensor version; the copies are kept while the mods are cached."""
    if mask_mod is noop_mask:
        mask_mod = None
    if score_mod is identity_score:
        score_mod = None
    ms = lower_mods(score_mod, mask_mod)
    if not ms.buffers:
        return
    keep = device_buffers(ms, device)
    module.set_buffers([t.data_ptr() for t in keep])
    module._bound_buffers = keep  # the addresses stay valid at least until the next binding


def device_buffers(ms, device):
    """The captured tensors of a lowered pair on ``device``."""
    keep = []
    for t in ms.buffers:
        if not isinstance(t, torch.Tensor):
            t = torch.as_tensor(t)
        if t.device != device:
            key = (id(t), t._version, str(device))
            hit = _DEVICE_BUFFERS.get(key)
            if hit is None or hit[0] is not t:
                if len(_DEVICE_BUFFERS) > 256:
                    _DEVICE_BUFFERS.clear()
                # same strides as the original: the load indices were built from them
                span = 1 + sum((d - 1) * st for d, st in zip(t.shape, t.stride()))
                flat = torch.as_strided(t, (span,), (1,)).to(device)
                hit = (t, flat)
                _DEVICE_BUFFERS[key] = hit
            t = hit[1]
        keep.append(t)
    return keep


# finished tables of create_block_mask(..., _compile=True), least recently used first
_TABLE_CACHE: "collections.OrderedDict" = collections.OrderedDict()
_TABLE_CACHE_MAX = 64


_CUDA_DEVICES = {}


def _require_cuda(device) -> torch.device:
    if device is None and torch.cuda.is_initialized():
        index = torch.cuda.current_device()
        dev = _CUDA_DEVICES.get(index)
        if dev is None:
            dev = _CUDA_DEVICES[index] = torch.device("cuda", index)
        return dev
    if not torch.cuda.is_available():
        raise RuntimeError("flaxattention_b200 needs a CUDA device (B200, sm_100a); there is no CPU path")
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    if dev.type == "cuda" and dev.index is None:
        dev = torch.device("cuda", torch.cuda.current_device())
    if dev.type != "cuda":
        raise RuntimeError(f"flaxattention_b200 tensors must live on a CUDA device, got {dev}")
    return dev


_MASK_BITS_MAX_BYTES = 64 << 20
_SNAPSHOT_MAX_BYTES = 256 << 10  # (one CTA compares the copy at every launch that uses the matrices)


def _wants_bits(ms, dev, nb, nh, Q_LEN, KV_LEN, Q_BLOCK_SIZE, KV_BLOCK_SIZE, force) -> int:
    """Bit matrices built beside the tables of a mask: 0 none, 1 the matrix, 2 the transposed one too."""
    if force is False or ms.mask is None:
        return 0
    row_major = nb * nh * Q_LEN * ((KV_LEN + 127) // 128) * 16
    transposed = nb * nh * KV_LEN * ((Q_LEN + 127) // 128) * 16
    both = 2 if row_major + transposed <= _MASK_BITS_MAX_BYTES else 1
    if force is True:
        return both
    if (Q_LEN > Q_BLOCK_SIZE and Q_BLOCK_SIZE % 32) or (KV_LEN > KV_BLOCK_SIZE and KV_BLOCK_SIZE % 32):
        return 0  # (no kernel that takes such blocks reads the matrix)
    if any(not isinstance(t, torch.Tensor) or t.is_inference() or t.device != dev for t in ms.buffers):
        return 0
    if sum(_cabi.span_bytes(t) for t in ms.buffers) > _SNAPSHOT_MAX_BYTES:
        return 0
    return both if row_major <= _MASK_BITS_MAX_BYTES else 0


def create_block_mask(
    mask_mod: Callable,
    B: Optional[int],
    H: Optional[int],
    Q_LEN: int,
    KV_LEN: int,
    BLOCK_SIZE: Union[int, Tuple[int, int]] = _DEFAULT_SPARSE_BLOCK_SIZE,
    _compile=False,
    device=None,
    b_offset: int = 0,
    h_offset: int = 0,
    _mask_bits: Optional[bool] = None,
) -> BlockMask:
    """Builds the BlockMask of ``mask_mod`` on the GPU.

    Same arguments as the reference.  The kernels are always compiled; ``_compile=True`` (the
    reference jits the construction so that repeated calls are cheap,
    flaxattention/core/blockmask.py:445-448) additionally keeps the finished tables, keyed by the
    lowered mask source, the shape, the block sizes, the offsets and the device, so a repeated
    call launches nothing.  Masks that read captured tensors are not kept (their contents may
    change between calls).  ``b_offset`` / ``h_offset`` give the global index of the first batch
    / head when the tables of one batch x heads shard are built.  A 5-argument function is
    treated as a score_mod whose ``-inf`` results mark masked positions.

    Next to the tables the mask itself is kept as a bit matrix (``BlockMask.mask_bits``, 1 bit per
    position where the reference's ``create_mask`` materialises a boolean,
    flaxattention/core/blockmask.py:277-322), one entry along batch / heads when ``mask_mod`` does
    not read ``b`` / ``h``: on the partial tiles the attention kernels read a row's words instead of
    evaluating ``mask_mod`` 128 times per row.  It is built when it takes at most 64 MiB, and transposed too
    (for the backward) when both together do
    (``_mask_bits=True`` / ``False`` forces it on or off), from the same evaluation as the tables.  A mask
    that reads captured tensors gets one when these are on the device and take at most 256 KiB; the
    attention calls then compare them, on the device, with a copy taken here, and evaluate ``mask_mod``
    if anything in them has changed since.
    """
    if mod_arity(mask_mod) not in (4, 5):
        raise AssertionError("mask_mod must take (b, h, q_idx, kv_idx) or (score, b, h, q_idx, kv_idx)")
    if B is None:
        B = 1
    if H is None:
        H = 1
    if isinstance(BLOCK_SIZE, int):
        Q_BLOCK_SIZE = BLOCK_SIZE
        KV_BLOCK_SIZE = BLOCK_SIZE
    else:
        Q_BLOCK_SIZE, KV_BLOCK_SIZE = BLOCK_SIZE
    if Q_LEN < 128:
        Q_BLOCK_SIZE = Q_LEN
    else:
        Q_LEN = _round_up_to_multiple(Q_LEN, Q_BLOCK_SIZE)
    KV_LEN = _round_up_to_multiple(KV_LEN, KV_BLOCK_SIZE)
    dev = _require_cuda(device)
    nq, nkv = Q_LEN // Q_BLOCK_SIZE, KV_LEN // KV_BLOCK_SIZE
    mask = None if mask_mod is noop_mask else mask_mod
    host = _cabi.host()
    module = module_for(None, mask)
    ms = lower_mods(None, mask)
    b0, h0 = (int(b_offset) if ms.mask_reads_b else 0), (int(h_offset) if ms.mask_reads_h else 0)
    bits_at = (b0 if ms.mask_reads_b else None, h0 if ms.mask_reads_h else None)
    cache_key = None
    if _compile and not ms.buffers:
        cache_key = (ms.key, B, H, Q_LEN, KV_LEN, Q_BLOCK_SIZE, KV_BLOCK_SIZE, int(b_offset), int(h_offset), str(dev))
        hit = _TABLE_CACHE.get(cache_key)
        if hit is not None:
            _TABLE_CACHE.move_to_end(cache_key)
            bm = BlockMask(*hit[:8], (Q_BLOCK_SIZE, KV_BLOCK_SIZE), mask_mod, hit[8], hit[9], _bits_at=bits_at)
            bm._kv_tiles = ms.kv_tiles(Q_LEN, KV_LEN)
            return bm
    # a mask that does not read the batch (head) index is evaluated once for all of them
    nb, nh = (B if ms.mask_reads_b else 1), (H if ms.mask_reads_h else 1)
    want_bits = _wants_bits(ms, dev, nb, nh, Q_LEN, KV_LEN, Q_BLOCK_SIZE, KV_BLOCK_SIZE, _mask_bits)
    buffers = device_buffers(ms, dev)
    sources = ()
    if want_bits and buffers:
        # (an inference tensor has no version, the copy alone tells)
        sources = tuple((t, t._version) if isinstance(t, torch.Tensor) and not t.is_inference() else (None, 0) for t in ms.buffers)
    tables = host.build_block_mask(module.handle.value, tuple(buffers), dev.index, B, H, nb, nh, Q_LEN, KV_LEN, Q_BLOCK_SIZE,
                                   KV_BLOCK_SIZE, b0, h0, want_bits)
    if cache_key is not None:
        _TABLE_CACHE[cache_key] = tables
        while len(_TABLE_CACHE) > _TABLE_CACHE_MAX:
            _TABLE_CACHE.popitem(last=False)
    bm = BlockMask(*tables[:8], (Q_BLOCK_SIZE, KV_BLOCK_SIZE), mask_mod, tables[8], tables[9], sources, tables[10],
                   bits_at)
    bm._kv_tiles = ms.kv_tiles(Q_LEN, KV_LEN)
    return bm
