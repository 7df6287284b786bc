"""Room for the intermediates of one layer call.

The layers allocate their results between two kernels with `empty`.  Outside a `Scratch` block that is torch.empty.  Inside one, small arrays are cut from a
single allocation instead: a torch tensor costs the host 2.3 to 2.7 µs, a layer over few tokens has up to ten of them, and they are only ever handed to the next
kernel as an address, a shape and a pitch.  The room belongs to the call: it is an ordinary allocation on the current stream and lives as long as an array in
it does.  What a layer returns is allocated outside the block and is a torch tensor.

Only the classes that come with this package compute in such a block (`room_of`): a mixer or feed-forward derived elsewhere may do with its intermediates what a torch tensor
allows, and gets torch tensors.
"""
from __future__ import annotations

import contextlib
import threading
from typing import Any, ContextManager, Optional, Tuple, Union

import torch

CHUNK = 8 << 20                # bytes of the room; larger arrays than LARGEST are torch tensors (a call that has them is not bound by the host)
LARGEST = 2 << 20
ALIGN = 256
SIZES = {torch.float32: 4, torch.bfloat16: 2, torch.int32: 4, torch.uint8: 1}

_local = threading.local()


class Array:
    """Address, shape and row pitch of an array of one or two dimensions, with the few methods of a tensor that the kernel front-ends ask for."""

    __slots__ = ("ptr", "shape", "pitch", "dtype", "device", "room")
    is_cuda = True

    def __init__(self, ptr: int, shape: Tuple[int, ...], pitch: int, dtype: torch.dtype, device: torch.device, room: torch.Tensor):
        self.ptr, self.shape, self.pitch, self.dtype, self.device, self.room = ptr, shape, pitch, dtype, device, room

    def __getattr__(self, name: str) -> Any:
        raise AttributeError(f"{name!r}: an intermediate inside a layer of this package is an address with a shape (ops/scratch.py), not a torch tensor; a class derived "
                             "from the layer's outside the package gets tensors")

    def data_ptr(self) -> int:
        return self.ptr

    def stride(self, dim: int) -> int:
        return self.pitch if dim == 0 and len(self.shape) == 2 else 1

    def dim(self) -> int:
        return len(self.shape)

    def numel(self) -> int:
        return self.shape[0] * self.shape[1] if len(self.shape) == 2 else self.shape[0]

    def is_contiguous(self) -> bool:
        return len(self.shape) == 1 or self.pitch == self.shape[1] or self.shape[0] <= 1

    def view(self, *shape: int) -> "Array":
        n = self.numel()
        if not self.is_contiguous() or not 1 <= len(shape) <= 2:
            raise ValueError(f"no view {shape} of {self.shape} with pitch {self.pitch}")
        if -1 in shape:
            rest = 1
            for v in shape:
                rest *= v if v != -1 else 1
            shape = tuple(n // rest if v == -1 else v for v in shape)
        if (shape[0] * shape[1] if len(shape) == 2 else shape[0]) != n:
            raise ValueError(f"no view {shape} of {n} elements")
        return Array(self.ptr, shape, shape[-1] if len(shape) == 2 else 1, self.dtype, self.device, self.room)

    def __getitem__(self, key: Any) -> "Array":
        """Columns [:, a:b] of all rows."""
        rows, cols = key
        if len(self.shape) != 2 or rows != slice(None) or cols.step is not None:
            raise IndexError(f"{key} of an array of shape {self.shape}")
        a, b, _ = cols.indices(self.shape[1])
        return Array(self.ptr + a * SIZES[self.dtype], (self.shape[0], max(b - a, 0)), self.pitch, self.dtype, self.device, self.room)


class Scratch:
    """with Scratch(): arrays of `empty` come from one allocation (per thread; blocks may be nested)."""

    __slots__ = ("room", "base", "used", "before")

    def __init__(self) -> None:
        self.room: Optional[torch.Tensor] = None
        self.base = self.used = 0

    def __enter__(self) -> "Scratch":
        self.before = getattr(_local, "scratch", None)
        _local.scratch = self
        return self

    def __exit__(self, *exc: Any) -> None:
        _local.scratch = self.before

    def take(self, shape: Tuple[int, ...], pitch: int, nbytes: int, dtype: torch.dtype, device: torch.device) -> Union[Array, torch.Tensor]:
        if self.room is None or self.used + nbytes > CHUNK:
            self.room = torch.empty(CHUNK, dtype=torch.uint8, device=device)
            self.base, self.used = self.room.data_ptr(), 0
        elif self.room.device != device:
            return torch.empty(shape, dtype=dtype, device=device)
        at = self.base + self.used
        self.used += (nbytes + ALIGN - 1) // ALIGN * ALIGN
        return Array(at, shape, pitch, dtype, device, self.room)


_PACKAGE = __name__.partition(".")[0] + "."


def room_of(layer: object) -> ContextManager:
    """A Scratch block for what `layer` computes, if its class is one of this package's; else a block in which `empty` is torch.empty as outside."""
    return Scratch() if type(layer).__module__.startswith(_PACKAGE) else contextlib.nullcontext()


def empty(shape: Union[int, Tuple[int, ...]], *, dtype: torch.dtype, device: torch.device) -> Union[Array, torch.Tensor]:
    """torch.empty; inside a Scratch block an array of at most LARGEST bytes of its room."""
    scratch = getattr(_local, "scratch", None)
    if scratch is None:
        return torch.empty(shape, dtype=dtype, device=device)
    if isinstance(shape, int):
        shape = (shape,)
    size = SIZES.get(dtype)
    n = shape[0] * shape[1] if len(shape) == 2 else shape[0]
    if size is None or n * size > LARGEST or n == 0 or len(shape) > 2:
        return torch.empty(shape, dtype=dtype, device=device)
    return scratch.take(shape, shape[1] if len(shape) == 2 else 1, n * size, dtype, device)
