"""DeltaAdaptive key codec on the device as a stand-alone call.

The reference's live key encoder (binary/DeltaAdaptiveEncoder.java:23-146): an adaptive
variable-width bit code for sorted keys. The training step does not come through here: with
``key_encoder="delta_adaptive"`` the fused compress and decode kernels write and read this format
themselves, chunk by chunk, without leaving the device (csrc/cuda/compress_kernels.cu,
decode_common.cuh). This module is the library form of the codec, `encode(keys) -> AdaptiveKeys`
and back, bit for bit equal to the CPU oracle (`oracle.delta_adaptive_encode`). It returns tensors
of exactly the encoded size, which depends on the data, so `encode` waits once, for the mode and the
two bit counts (they come through a pinned host word while the streams are written, in the order of
the calling stream). The tensors are views of one buffer, at most twice as long as they are (or 256 KB
longer): the room that a list of this length may need, or a copy of what was used of it.
csrc/cuda/keys_kernels.cu has the kernels.
"""
from __future__ import annotations

import ctypes as C
import threading
from dataclasses import dataclass
from typing import Optional

import torch

from . import lib as L
from .codec import DoneWords


BAD_INPUT = 5            # SkmlStatus
TILE = 8192              # keys of a block where a list is decoded by one launch
SPARE_WORDS = 1 << 15    # 256 KB: the copy takes 4 us of 77 at 100,000 keys, 3 of 87 at 1M
ROOM_WORDS = 1 << 22     # 32 MB: from here on the length is found first, by a launch of its own, and no room is allocated unused


@dataclass
class AdaptiveKeys:
    size: int
    num_intervals: int
    flag_kind: int            # 0 = fixed-width flags, 1 = unary flags
    flag_bits: int
    delta_bits: int
    flag_words: torch.Tensor  # int64 on the device: java.util.BitSet words, ceil(flag_bits / 64) of them
    delta_words: torch.Tensor

    def to_oracle_dict(self) -> dict:
        import numpy as np
        return {"size": self.size, "num_intervals": self.num_intervals, "flag_kind": self.flag_kind,
                "flag_words": self.flag_words.cpu().numpy().view(np.uint64), "flag_bits": self.flag_bits,
                "delta_words": self.delta_words.cpu().numpy().view(np.uint64), "delta_bits": self.delta_bits}

    def nbytes_wire(self) -> int:
        """Bytes of the reference's field layout: 3 ints + flag + 2 counted word arrays."""
        return 4 + 4 + 1 + 4 + 8 * self.flag_words.numel() + 4 + 8 * self.delta_words.numel()


class _CallState:
    """What one thread's calls need: the pinned words a plan comes back in. They go back when the thread ends, with this
    object (the thread-local around it is one object for all threads and outlives them)."""

    def __init__(self):
        self.words = DoneWords.take(self)
        self.status = C.c_uint(0)
        self.status_ref = C.byref(self.status)


_call = threading.local()
_workspace_bytes = 0


def _workspace(device) -> torch.Tensor:
    global _workspace_bytes
    if not _workspace_bytes:
        _workspace_bytes = int(L.lib().skml_da_workspace_bytes())
    return torch.empty(_workspace_bytes, dtype=torch.uint8, device=device)


def _call_state() -> _CallState:
    state: Optional[_CallState] = getattr(_call, "state", None)
    if state is None:
        state = _call.state = _CallState()
    return state


def encode(keys: torch.Tensor) -> AdaptiveKeys:
    """keys: strictly increasing non-negative int32 on the device (synchronises to size the outputs)."""
    if keys.dtype != torch.int32 or not keys.is_cuda:
        raise ValueError("keys must be a CUDA int32 tensor")
    keys = keys.contiguous()
    n, dev, lib, cs = keys.numel(), keys.device, L.lib(), _call_state()
    stream = L.stream()
    work = _workspace(dev)
    room = lib.skml_da_words(n)

    def run(words: Optional[torch.Tensor], planned: bool = False):
        L.check(lib.skml_da_encode(keys.data_ptr(), n, work.data_ptr(), L.ptr(words), 0 if words is None else words.numel(), planned,
                                   cs.words.data_ptr(), cs.status_ref, stream), "skml_da_encode")
        L.count_launches(1)
        if cs.status.value & 0xFF == BAD_INPUT:
            raise ValueError("keys must be non-negative and strictly increasing")
        if cs.status.value:
            raise RuntimeError(f"skml_da_encode reported status {cs.status.value:#x}")

    known = room > ROOM_WORDS
    words = None if known else torch.empty(room, dtype=torch.int64, device=dev)
    run(words)
    _, mode, flag_bits, delta_bits = cs.words[:4].tolist()
    nf, nd = (flag_bits + 63) // 64, (delta_bits + 63) // 64
    if known:
        words = torch.empty(nf + nd, dtype=torch.int64, device=dev)
        run(words, True)
    elif room - (nf + nd) > max(nf + nd, SPARE_WORDS):
        words = words[:nf + nd].clone()
    fw, dw = words[:nf], words[nf:nf + nd]
    return AdaptiveKeys(n, mode & 0xFFFFFFFF, mode >> 32, flag_bits, delta_bits, fw, dw)


def decode(e: AdaptiveKeys) -> torch.Tensor:
    """Returns the int32 keys on the device."""
    dev, lib, n = e.delta_words.device, L.lib(), e.size
    if n == 0:
        return torch.zeros(0, dtype=torch.int32, device=dev)
    fw, dw = e.flag_words.to(torch.int64).contiguous(), e.delta_words.to(torch.int64).contiguous()
    keys = torch.empty(n, dtype=torch.int32, device=dev)
    work = _workspace(dev)
    pos = torch.empty(n, dtype=torch.int64, device=dev) if e.flag_kind else None
    L.check(lib.skml_da_decode(fw.data_ptr(), fw.numel(), dw.data_ptr(), dw.numel(), n, e.num_intervals, e.flag_kind, e.flag_bits,
                               work.data_ptr(), L.ptr(pos), keys.data_ptr(), 0, L.stream()), "skml_da_decode")
    L.count_launches((1 if n <= (TILE if e.flag_kind else 148 * TILE) else 3) + (2 if e.flag_kind else 0))
    return keys
