"""Host runtime above the backend ABI: context, arenas, tensors, step scopes and the tape.

This mirrors the part of the reference's core that the gpt_lm path exercises
(src/core/memory.c: params / state arenas, per-step scratch and data slots, one fence per
step, :1350-1474; src/core/tensor.c descriptors; src/autograd/autograd.c:128,943-1135 tape
and gradient slots) with the same names and call order, so that the op capsules in ops.py
read like the reference's core_*.c files. It holds no numerics: every byte of tensor data is
produced by a gd_backend_* call.
"""
from __future__ import annotations

import ctypes as C
import math
from typing import Callable, Optional, Sequence

import numpy as np

from . import abi
from .abi import BackendError, DTYPE_SIZE, F16, BF16, F32, I32, U8

ALIGN = 256

NP_DTYPES = {F16: np.float16, F32: np.float32, I32: np.int32, U8: np.uint8, BF16: np.uint16, abi.U16: np.uint16}


def bf16_bits_from_f32(a: np.ndarray) -> np.ndarray:
    """Round-to-nearest-even FP32 -> BF16 bit patterns (uint16)."""
    u = np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)
    lsb = (u >> 16) & 1
    return ((u + 0x7FFF + lsb) >> 16).astype(np.uint16)


def f32_from_bf16_bits(b: np.ndarray) -> np.ndarray:
    return (b.astype(np.uint32) << 16).view(np.float32)


class Arena:
    """One backend buffer with bump allocation (reference gd_arena, src/core/memory.c:214-258)."""

    def __init__(self, ctx: "Context", name: str, nbytes: int):
        self.ctx, self.name, self.capacity = ctx, name, int(nbytes)
        out = C.c_void_p()
        st = ctx.lib.gd_backend_buffer_create(ctx.backend, self.capacity, C.byref(out))
        if st != abi.GD_OK:
            raise BackendError(st, f"buffer_create({name}, {nbytes})", ctx.last_error())
        self.buffer = out
        self.top = 0
        self.high_water = 0
        self._views: dict = {}   # (dtype, shape) -> image of a tensor view without its offset

    def alloc(self, nbytes: int, align: int = ALIGN) -> int:
        off = (self.top + align - 1) & ~(align - 1)
        if off + nbytes > self.capacity:
            raise MemoryError(f"arena {self.name}: need {off + nbytes} bytes, capacity {self.capacity}")
        self.top = top = off + int(nbytes)
        if top > self.high_water:
            self.high_water = top
        return off

    def reset(self) -> None:
        self.top = 0

    def view(self, offset: int, dtype: int, shape: tuple, count: int) -> abi.TensorView:
        """gd_backend_tensor_view of contiguous bytes of this arena. The image of a (dtype, shape) is kept and copied: filling the
        sixteen array fields of a new structure was a quarter of the host time of a small attention call."""
        image = self._views.get((dtype, shape))
        if image is None:
            v = abi.TensorView()
            v.buffer, v.count, v.dtype, v.rank = self.buffer, count, dtype, len(shape)
            stride = 1
            for d in range(len(shape) - 1, -1, -1):
                v.shape[d] = shape[d]
                v.strides[d] = stride
                stride *= shape[d]
            if len(self._views) >= 1024:   # shapes follow the batch: bounded
                self._views.clear()
            image = self._views[(dtype, shape)] = bytes(v)
        v = abi.TensorView.from_buffer_copy(image)
        v.offset = offset
        return v

    def destroy(self) -> None:
        if self.buffer:
            self.ctx.lib.gd_backend_buffer_destroy(self.buffer)
            self.buffer = None
            self._views.clear()


class Tensor:
    """Descriptor of contiguous tensor bytes inside an arena (reference gd_tensor)."""

    # what most tensors never set
    requires_grad = False
    grad: Optional["Tensor"] = None
    is_leaf = False
    _count = _tv = _ref = None

    def __init__(self, ctx: "Context", arena: Arena, offset: int, dtype: int, shape: Sequence[int], name: str = ""):
        self.ctx, self.arena, self.dtype, self.name = ctx, arena, dtype, name
        self.offset = offset if type(offset) is int else int(offset)
        if type(shape) is not tuple:
            shape = tuple(map(int, shape))
        for d in shape:   # (a copy of every shape would cost as much as the rest of this)
            if type(d) is not int:
                shape = tuple(map(int, shape))
                break
        self.shape = shape

    @property
    def count(self) -> int:
        if self._count is None:
            self._count = math.prod(self.shape)
        return self._count

    @property
    def nbytes(self) -> int:
        return self.count * DTYPE_SIZE[self.dtype]

    @property
    def buffer(self):
        return self.arena.buffer

    def tv(self) -> abi.TensorView:
        """gd_backend_tensor_view of the whole tensor (cached; descriptors are immutable)."""
        if self._tv is None:
            self._tv = self.arena.view(self.offset, self.dtype, self.shape, self.count)
        return self._tv

    def ref(self):
        """Pointer argument to tv() (cached with it)."""
        r = self._ref
        if r is None:
            r = self._ref = C.byref(self.tv())
        return r

    def mv(self, rows: int, cols: int, row_offset: int = 0, row_bytes: Optional[int] = None) -> abi.MatrixView:
        es = DTYPE_SIZE[self.dtype]
        rb = cols * es if row_bytes is None else row_bytes
        return abi.MatrixView(self.arena.buffer, self.offset + row_offset * rb, rows, cols, rb, self.dtype)

    def vv(self, start: int = 0, length: Optional[int] = None) -> abi.VectorView:
        return abi.VectorView(self.arena.buffer, self.offset + start * DTYPE_SIZE[self.dtype], self.count - start if length is None else length, self.dtype)

    def reshape(self, shape: Sequence[int]) -> "Tensor":
        t = Tensor(self.ctx, self.arena, self.offset, self.dtype, shape, self.name)
        assert t.count == self.count
        return t

    def rows(self, start: int, n: int) -> "Tensor":
        """View of n leading-dimension rows starting at `start`."""
        inner = self.count // self.shape[0]
        return Tensor(self.ctx, self.arena, self.offset + start * inner * DTYPE_SIZE[self.dtype], self.dtype,
                      (n,) + self.shape[1:], self.name)

    # ---- transfers (gd_tensor_write / gd_tensor_read: flush + synchronous copy) ----
    def write(self, host: np.ndarray) -> None:
        if self.dtype == BF16 and host.dtype != np.uint16:
            host = bf16_bits_from_f32(host)
        a = np.ascontiguousarray(host, dtype=NP_DTYPES[self.dtype])
        assert a.size == self.count, (a.shape, self.shape)
        self.ctx.check(self.ctx.lib.gd_backend_upload(self.ctx.backend, self.buffer, self.offset,
                                                      a.ctypes.data_as(C.c_void_p), a.nbytes), "upload")

    def write_async(self, pinned: np.ndarray) -> None:
        """Stream-ordered upload from page-locked memory (Context.pinned_copy); not waited for. `pinned` must
        keep its contents until a fence recorded after this call has completed."""
        assert pinned.dtype == NP_DTYPES[self.dtype] and pinned.size == self.count and pinned.flags.c_contiguous
        self.ctx.check(self.ctx.lib.gdb200_upload_async(self.ctx.backend, self.buffer, self.offset,
                                                        pinned.ctypes.data, pinned.nbytes), "upload_async")

    def read_async(self, pinned_out: np.ndarray) -> None:
        """Stream-ordered download into page-locked memory; valid once a later fence has completed."""
        assert pinned_out.dtype == NP_DTYPES[self.dtype] and pinned_out.size == self.count and pinned_out.flags.c_contiguous
        self.ctx.check(self.ctx.lib.gdb200_download_async(self.ctx.backend, self.buffer, self.offset,
                                                          pinned_out.ctypes.data, pinned_out.nbytes), "download_async")

    def read(self) -> np.ndarray:
        out = np.empty(self.shape, dtype=NP_DTYPES[self.dtype])
        self.ctx.check(self.ctx.lib.gd_backend_download(self.ctx.backend, self.buffer, self.offset,
                                                        out.ctypes.data_as(C.c_void_p), out.nbytes), "download")
        return out

    def read_f32(self) -> np.ndarray:
        a = self.read()
        return f32_from_bf16_bits(a) if self.dtype == BF16 else a.astype(np.float32)


class Context:
    """gd_context: one backend, params/state arenas, one scratch slot and one data slot.

    The reference keeps `scratch_slots` ring buffers and waits on the slot's fence before
    reuse (memory.c:701); with one slot that is a wait for the previous step's fence at
    begin_step, which is what this class does by default (`run_ahead` 0). With `run_ahead` = n the
    host may enqueue up to n steps beyond the one the device is executing: begin_step then waits
    only for the fence of step k - n. Of the device arenas only the data slot needs two places for
    that (upload_beside copies a batch while the step before it runs): every kernel and every other
    copy of step k + 1 is queued behind step k; host memory handed to write_async / read_async must
    be rotated by the caller.
    """

    def __init__(self, params_bytes: int = 256 << 20, state_bytes: int = 512 << 20,
                 scratch_bytes: int = 6 << 30, data_bytes: int = 64 << 20):
        self.lib = abi.load_library()
        be = C.c_void_p()
        st = self.lib.gd_backend_create_default(C.byref(be))
        if st != abi.GD_OK:
            raise BackendError(st, "gd_backend_create_default", "no sm_100a CUDA device or library mismatch")
        self.backend = be
        self.params = Arena(self, "params", params_bytes)
        self.state = Arena(self, "state", state_bytes)
        self.scratch = Arena(self, "scratch", scratch_bytes)
        self._make_data_slot(data_bytes)
        self.tape: list[Callable[[], None]] = []
        self.grad_enabled = True
        self._fences: list[abi.Fence] = []
        self.run_ahead = 0
        self.in_step = False
        self.grad_ready_hook: Optional[Callable[[Tensor], None]] = None

    def _make_data_slot(self, nbytes: int) -> None:
        """The data arena: twice what was asked for, because batches copied beside the running step alternate between its halves."""
        self.data = Arena(self, "data", 2 * ((nbytes + ALIGN - 1) & ~(ALIGN - 1)))
        self._data_before, self._data_base = (0, 0), 0

    # ---- plumbing ----
    def last_error(self) -> str:
        s = self.lib.gdb200_last_error(self.backend) if getattr(self, "backend", None) else b""
        return (s or b"").decode()

    def check(self, status: int, what: str) -> None:
        if status != abi.GD_OK:
            raise BackendError(status, what, self.last_error())

    def destroy(self) -> None:
        if getattr(self, "backend", None):
            self.flush()
            for f in self._fences:
                self.lib.gd_backend_fence_destroy(C.byref(f))
            self._fences = []
            for a in (self.params, self.state, self.scratch, self.data):
                a.destroy()
            self.lib.gd_backend_destroy(self.backend)
            self.backend = None

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.destroy()

    def flush(self) -> None:
        self.check(self.lib.gd_backend_flush(self.backend), "flush")

    def launch_count(self) -> int:
        return int(self.lib.gdb200_launch_count(self.backend))

    def pinned_copy(self, a: np.ndarray) -> np.ndarray:
        """Copy of `a` in page-locked host memory (kept alive by the context)."""
        a = np.ascontiguousarray(a)
        ptr = self.lib.gdb200_pinned_alloc(max(a.nbytes, 1))
        if not ptr:
            raise MemoryError("pinned host allocation failed")
        self._pinned = getattr(self, "_pinned", [])
        self._pinned.append(ptr)
        buf = (C.c_byte * a.nbytes).from_address(ptr)
        out = np.frombuffer(buf, dtype=a.dtype).reshape(a.shape)
        out[...] = a
        return out

    # ---- step scope (reference gd_begin_step / gd_end_step) ----
    def begin_step(self) -> None:
        assert not self.in_step
        self.wait_steps(self.run_ahead)
        self.scratch.reset()
        self._data_before, self._data_base = (self._data_base, self.data.top), 0   # range of the data slot the step before uses
        self.data.reset()
        self.tape.clear()
        self.check(self.lib.gd_backend_scope_begin(self.backend), "scope_begin")
        self.in_step = True

    def end_step(self) -> None:
        assert self.in_step
        f = abi.Fence()
        self.check(self.lib.gd_backend_record_fence(self.backend, C.byref(f)), "record_fence")
        self._fences.append(f)
        self.tape.clear()
        self.in_step = False

    def wait_steps(self, keep: int = 0) -> None:
        """Waits until at most `keep` recorded steps are still in flight (oldest first)."""
        while len(self._fences) > keep:
            f = self._fences.pop(0)
            st = self.lib.gd_backend_fence_wait(C.byref(f))
            self.lib.gd_backend_fence_destroy(C.byref(f))
            self.check(st, "fence_wait")

    # ---- tensors ----
    def empty(self, arena: Arena, dtype: int, shape: Sequence[int], name: str = "") -> Tensor:
        t = Tensor(self, arena, 0, dtype, shape, name)
        t._count = n = math.prod(t.shape)
        t.offset = arena.alloc((n or 1) * DTYPE_SIZE[dtype])
        return t

    def scratch_empty(self, dtype: int, shape: Sequence[int], name: str = "") -> Tensor:
        return self.empty(self.scratch, dtype, shape, name)

    def fill(self, t: Tensor, pattern: int) -> None:
        self.check(self.lib.gd_backend_fill(self.backend, t.buffer, t.offset, t.count, DTYPE_SIZE[t.dtype], pattern), "fill")

    def zeros(self, arena: Arena, dtype: int, shape: Sequence[int], name: str = "") -> Tensor:
        t = self.empty(arena, dtype, shape, name)
        self.fill(t, 0)
        return t

    def from_numpy(self, arena: Arena, dtype: int, host: np.ndarray, name: str = "") -> Tensor:
        t = self.empty(arena, dtype, host.shape, name)
        t.write(host)
        return t

    def upload_beside(self, arrays: Sequence[np.ndarray]) -> Optional[list[Tensor]]:
        """I32 tensors of a step's page-locked arrays in the half of the data slot that the step before does not use, copied while that step
        still runs. None when there is no such half: more steps may be in flight, or the slot is used otherwise or too small."""
        half = self.data.capacity // 2 & ~(ALIGN - 1)
        lo, hi = self._data_before
        base = half if hi <= half else 0
        if self.run_ahead > 1 or self.data.top != 0 or (base == 0 and lo < half) or sum(a.nbytes + ALIGN for a in arrays) > half:
            return None
        self.data.top = self._data_base = base
        ts = [self.empty(self.data, I32, a.shape) for a in arrays]
        n = len(ts)
        assert all(a.dtype == np.int32 and a.flags.c_contiguous for a in arrays)
        self.check(self.lib.gdb200_upload_beside(self.backend, self.data.buffer, n, (C.c_size_t * n)(*[t.offset for t in ts]),
                                                 (C.c_void_p * n)(*[a.ctypes.data for a in arrays]), (C.c_size_t * n)(*[a.nbytes for a in arrays])),
                   "upload_beside")
        return ts

    # ---- tape (reference gd_autograd_record + reverse walk) ----
    def record(self, backward: Callable[[], None]) -> None:
        if self.grad_enabled:
            self.tape.append(backward)

    def accumulate_grad(self, t: Tensor, g: Tensor) -> None:
        """First contribution is adopted, later ones are added with gd_backend_accumulate
        (16-bit storage rounds after every add), as src/autograd/autograd.c:517-685 does."""
        if not t.requires_grad:
            return
        if t.grad is None:
            t.grad = g
        else:
            assert t.grad.count == g.count and t.grad.dtype == g.dtype
            self.check(self.lib.gd_backend_accumulate(self.backend, t.grad.buffer, t.grad.offset, g.buffer, g.offset,
                                                      g.count, g.dtype), "accumulate")

    def run_backward(self) -> None:
        for fn in reversed(self.tape):
            fn()
        self.tape.clear()
