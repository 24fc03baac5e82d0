"""``torch.library`` custom ops over the C ABI (CUDA only, no fallback).

``ternel::tq1_linear``, ``ternel::tq1_embedding`` and ``ternel::tq1_validate``
take the packed weight as canonical blocks ``uint8[N, K/128, 28]`` resident on
the GPU. PyTorch is only used for device memory and the current stream; the
work happens in ``libternel_b200.so``. The ops are registered for the CUDA
dispatch key alone, so a CPU tensor is refused by the dispatcher instead of
being served by some other path.

Eager calls do not pass through the dispatcher: the wrappers first offer the call to
the C function of csrc/torch_binding.cpp, which takes the plain case in one step and
declines everything else (wrong arguments, gradients, tensor subclasses, tracing).

The Python wrappers below (`tq1_matmul`, `tq1_gemm`, `tq1_get_rows`) keep the
names and the pre-launch checks of the reference's kernel wrappers
(src/ternel_mlx/kernels.py:1191-1284,1360-1398).
"""

from __future__ import annotations

import ctypes
import threading

import torch

from . import _native
from .format import BLOCK_BYTES, BLOCK_SIZE, FormatError, check
from .layout import out_of_range_message

ACTIVATION_DTYPES = (torch.float16,)
OUTPUT_DTYPES = (torch.float16, torch.float32)

# Scratch buffers: one per device for calls on its default stream and for captured ones, which hold it for good, and one for
# each of the last few other streams that have called. Buffers that a larger one has taken over from stay alive.
MAX_STREAM_WORKSPACES = 8
_workspaces: dict[int, torch.Tensor] = {}
_stream_workspaces: dict[tuple[int, int], torch.Tensor] = {}
_replaced: dict[int, list[torch.Tensor]] = {}
_workspace_lock = threading.Lock()


def _stream_ptr(device: torch.device) -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream(device).cuda_stream)


def _new_workspace(device: torch.device, nbytes: int) -> torch.Tensor:
    """A zero-filled buffer (slots and counters start at zero) of a power of two bytes, at least 1 MiB."""
    return torch.zeros(1 << max(20, (nbytes - 1).bit_length()), dtype=torch.uint8, device=device)


def _workspace(device: torch.device, nbytes: int) -> torch.Tensor | None:
    """A scratch buffer for a call on the current stream, grown on demand and reused across calls.

    Calls that may overlap need separate buffers, so every stream has its own. Only the last ``MAX_STREAM_WORKSPACES`` streams
    of a device that asked for one keep it; a buffer that is let go returns to the allocator in the order of its stream.

    A captured graph keeps the address it was captured with, and its replays expect the buffer as the last call left it.
    Captured calls therefore take the default stream's buffer, which is at least as large as any other (a warm-up on a side
    stream has grown it) and is never given back when a larger one replaces it: sizes are powers of two, so all replaced
    ones together are smaller than the one in use. A captured call that needs more than there is brings a buffer of its own,
    which belongs to the graph's memory and is zero-filled by each replay. Replays count as calls on the default stream.
    """
    if nbytes == 0:
        return None
    index = device.index if device.index is not None else torch.cuda.current_device()
    stream = torch.cuda.current_stream(device).cuda_stream
    with torch.cuda.device(index):
        capturing = torch.cuda.is_current_stream_capturing()
    with _workspace_lock:
        shared = _workspaces.get(index)
        if shared is None or shared.numel() < nbytes:
            if capturing:
                return torch.zeros(nbytes, dtype=torch.uint8, device=device)
            if shared is not None:
                _replaced.setdefault(index, []).append(shared)
            with torch.cuda.stream(torch.cuda.default_stream(device)):
                shared = _workspaces[index] = _new_workspace(device, nbytes)
            _native.binding().set_workspace(index, 0, shared)
        if capturing or stream == 0:
            return shared
        own = _stream_workspaces.pop((index, stream), None)
        if own is None or own.numel() < nbytes:
            own = _new_workspace(device, nbytes)
            _native.binding().set_workspace(index, stream, own)
        _stream_workspaces[index, stream] = own                 # the last one used stands last
        others = [key for key in _stream_workspaces if key[0] == index]
        if len(others) > MAX_STREAM_WORKSPACES:
            del _stream_workspaces[others[0]]
            _native.binding().set_workspace(index, others[0][1], None)
        return own


def check_status(device=None) -> None:
    """Read the status words of the device's workspaces (synchronises the device).

    Zero: every bounded wait inside the kernels was met. 7: results are good but the sequence tags are about
    to wrap, so the workspace is zeroed here. Anything else raises: a wait ran out (the results of the calls
    since the last check are not to be trusted) and the workspace is zeroed so that later calls start clean.
    """
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    index = device.index if device.index is not None else torch.cuda.current_device()
    if index not in _workspaces:
        return
    torch.cuda.synchronize(device)
    buffers = [_workspaces[index], *_replaced.get(index, ()), *(b for k, b in _stream_workspaces.items() if k[0] == index)]
    failed = 0
    for buf in buffers:
        status = int(buf[:4].view(torch.int32)[0].item())
        if status:
            buf.zero_()
            torch.cuda.synchronize(device)      # the buffer may be another stream's
            failed = status if status != 7 else failed
    if failed:
        raise RuntimeError(f"a bounded wait inside a packed ternary kernel ran out (status {failed}); "
                           "the workspace has been reset")


def _check_blocks(blocks: torch.Tensor) -> tuple[int, int]:
    if blocks.dtype != torch.uint8:
        raise FormatError(f"canonical blocks must be uint8, got {blocks.dtype}")
    if blocks.dim() != 3 or blocks.shape[2] != BLOCK_BYTES:
        raise FormatError(f"blocks must have shape (rows, groups, 28), got {tuple(blocks.shape)}")
    if blocks.shape[0] <= 0 or blocks.shape[1] <= 0:
        raise FormatError("packed tensor has no rows or no groups")
    if not blocks.is_contiguous():
        raise FormatError("blocks must be contiguous")
    return blocks.shape[0], blocks.shape[1]


@torch.library.custom_op("ternel::tq1_linear", mutates_args=(), device_types="cuda")
def _tq1_linear_op(blocks: torch.Tensor, x: torch.Tensor, out_f32: bool) -> torch.Tensor:
    rows, groups = blocks.shape[0], blocks.shape[1]
    batch, columns = x.shape
    out = torch.empty((batch, rows), dtype=torch.float32 if out_f32 else torch.float16, device=x.device)
    lib = _native.lib()
    need = lib.tq1_linear_workspace_bytes(batch, rows, columns)
    ws = _workspace(x.device, need)
    with torch.cuda.device(x.device):
        check(lib.tq1_linear_f16(blocks.data_ptr(), x.data_ptr(), out.data_ptr(), int(out_f32),
                                 batch, rows, columns,
                                 ws.data_ptr() if ws is not None else None,
                                 ws.numel() if ws is not None else 0,
                                 _stream_ptr(x.device)))
    return out


@_tq1_linear_op.register_fake
def _(blocks, x, out_f32):
    return x.new_empty((x.shape[0], blocks.shape[0]), dtype=torch.float32 if out_f32 else torch.float16)


@torch.library.custom_op("ternel::tq1_linear_swiglu", mutates_args=(), device_types="cuda")
def _tq1_linear_swiglu_op(blocks: torch.Tensor, x: torch.Tensor, out_f32: bool) -> torch.Tensor:
    rows = blocks.shape[0]
    batch, columns = x.shape
    out = torch.empty((batch, rows // 2), dtype=torch.float32 if out_f32 else torch.float16, device=x.device)
    lib = _native.lib()
    need = lib.tq1_linear_workspace_bytes(batch, rows, columns)
    ws = _workspace(x.device, need)
    with torch.cuda.device(x.device):
        check(lib.tq1_linear_swiglu_f16(blocks.data_ptr(), x.data_ptr(), out.data_ptr(), int(out_f32),
                                        batch, rows // 2, columns,
                                        ws.data_ptr() if ws is not None else None,
                                        ws.numel() if ws is not None else 0, _stream_ptr(x.device)))
    return out


@_tq1_linear_swiglu_op.register_fake
def _(blocks, x, out_f32):
    return x.new_empty((x.shape[0], blocks.shape[0] // 2), dtype=torch.float32 if out_f32 else torch.float16)


@torch.library.custom_op("ternel::tq1_embedding", mutates_args=(), device_types="cuda")
def _tq1_embedding_op(blocks: torch.Tensor, ids: torch.Tensor, out_f32: bool) -> torch.Tensor:
    rows, groups = blocks.shape[0], blocks.shape[1]
    columns = groups * BLOCK_SIZE
    out = torch.empty((ids.numel(), columns), dtype=torch.float32 if out_f32 else torch.float16,
                      device=blocks.device)
    with torch.cuda.device(blocks.device):
        check(_native.lib().tq1_embedding_f16(blocks.data_ptr(), ids.data_ptr(), out.data_ptr(),
                                              int(out_f32), ids.numel(), rows, columns,
                                              _stream_ptr(blocks.device)))
    return out


@_tq1_embedding_op.register_fake
def _(blocks, ids, out_f32):
    return blocks.new_empty((ids.numel(), blocks.shape[1] * BLOCK_SIZE),
                            dtype=torch.float32 if out_f32 else torch.float16)


@torch.library.custom_op("ternel::tq1_validate", mutates_args=(), device_types="cuda")
def _tq1_validate_op(blocks: torch.Tensor) -> torch.Tensor:
    counts = torch.empty(2, dtype=torch.int64, device=blocks.device)
    groups = blocks.numel() // BLOCK_BYTES
    with torch.cuda.device(blocks.device):
        check(_native.lib().tq1_validate_blocks_device(blocks.data_ptr(), groups, counts.data_ptr(),
                                                       _stream_ptr(blocks.device)))
    return counts


@_tq1_validate_op.register_fake
def _(blocks):
    return blocks.new_empty(2, dtype=torch.int64)


def eager_linear(blocks, x, out_dtype, swiglu: bool, flat: bool):
    """The product through the eager call path, or None where that path does not apply. ``flat``: ``x`` must be
    two-dimensional; otherwise its leading dimensions carry over to the result."""
    if torch.compiler.is_compiling():
        return None
    return (_fast or _load_fast()).linear(blocks, x, out_dtype, swiglu, flat)


def eager_embedding(blocks, ids, dtype, flat: bool):
    """The row gather through the eager call path, or None where that path does not apply."""
    if torch.compiler.is_compiling():
        return None
    return (_fast or _load_fast()).embedding(blocks, ids, dtype, flat)


_fast = None


class _NoFastPath:
    """Stands in where there is no GPU: every call is left to the ordinary path, which says so."""

    linear = embedding = staticmethod(lambda *args: None)


def _load_fast():
    global _fast
    _fast = _native.binding() if torch.cuda.is_available() else _NoFastPath
    return _fast


def _require_cuda(tensor: torch.Tensor, name: str) -> None:
    if not tensor.is_cuda:
        raise RuntimeError(
            f"{name} is on {tensor.device}: the packed ternary kernels run on CUDA only "
            "(there is no CPU fallback)")


def validate_device_blocks(blocks: torch.Tensor) -> None:
    """Load-time scan on the GPU; raises FormatError with both counts (fail closed)."""
    _check_blocks(blocks)
    _require_cuda(blocks, "blocks")
    bad_full, bad_tail = (int(v) for v in _tq1_validate_op(blocks).tolist())
    if bad_full or bad_tail:
        raise FormatError(f"invalid base-3 bytes: regular={bad_full}, tail={bad_tail}")


_STAGING_BYTES = 8 << 20            # pinned memory of an upload at most
_STAGED_FROM = 64 << 10             # smaller arrays the driver takes along: 11 KB 72 us, staged 78; 54 KB 77.5 both ways; 115 KB 84 and 81


def _upload(first: torch.Tensor, second: torch.Tensor, device: torch.device) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor | None]:
    """Contiguous copies of both on the current device, complete in the order of its current stream. Ordinary host memory goes
    through pinned staging, filled by several threads while the transfer runs (``tq1_upload_pair``). The third result is that
    staging: the transfers out of it are not known to torch's pool, so the caller holds it until the stream has been waited for."""
    arrays = [array.contiguous() for array in (first, second)]
    sizes = [array.numel() * array.element_size() for array in arrays]
    plain = sum(sizes) < _STAGED_FROM or any(array.device.type != "cpu" or array.is_pinned() for array in arrays)
    if not plain:
        try:
            staging = torch.empty(min(sum(sizes) + (1 << 20), _STAGING_BYTES), dtype=torch.uint8, device="cpu", pin_memory=True)
        except RuntimeError:            # no pinned memory to be had: the driver's own way
            plain = True
    if plain:
        return *(array.to(device) for array in arrays), None
    copies = [torch.empty(array.shape, dtype=array.dtype, device=device) for array in arrays]
    check(_native.lib().tq1_upload_pair(copies[0].data_ptr(), arrays[0].data_ptr(), sizes[0],
                                        copies[1].data_ptr(), arrays[1].data_ptr(), sizes[1],
                                        staging.data_ptr(), staging.numel(), _stream_ptr(device)))
    return *copies, staging


def load_tiled_device(blocks: torch.Tensor, codes: torch.Tensor, scales: torch.Tensor, tile: int) -> None:
    """Fill canonical ``blocks`` on the GPU from the tiled pair (``uint8[tiles, groups, 26, tile]`` and 16-bit
    ``[tiles, groups, tile]``, on the host or the GPU): the arrays are uploaded as they are, scanned there, and
    converted only if every byte is legal (fail closed, as ``validate_packed_codes``). The blocks are there when the call
    returns, on whatever stream they are used next."""
    rows, groups = _check_blocks(blocks)
    with torch.cuda.device(blocks.device):
        codes, scales, staging = _upload(codes, scales, blocks.device)
        try:
            counts = torch.empty(2, dtype=torch.int64, device=blocks.device)
            # scanned and, where nothing was found, converted: one wait for both, by reading the counts
            check(_native.lib().tq1_load_tiled_device(codes.data_ptr(), scales.data_ptr(), blocks.data_ptr(), rows, groups, tile,
                                                      counts.data_ptr(), _stream_ptr(blocks.device)))
            bad_full, bad_tail = counts.tolist()
        except BaseException:
            torch.cuda.current_stream().synchronize()       # nothing is read from the staging any more
            raise
        del staging
    if bad_full or bad_tail:
        raise FormatError(out_of_range_message(bad_full, bad_tail))


def _check_activations(x: torch.Tensor, groups_per_row: int) -> int:
    if x.dtype not in ACTIVATION_DTYPES:
        raise FormatError(f"activations must be one of {ACTIVATION_DTYPES}, got {x.dtype}")
    if x.dim() != 2:
        raise FormatError(f"activations must be 2-D (batch, columns), got shape {tuple(x.shape)}")
    columns = groups_per_row * BLOCK_SIZE
    if x.shape[1] != columns:
        raise FormatError(f"activations have {x.shape[1]} columns, expected {columns}")
    if x.shape[0] <= 0:
        raise FormatError("activations have an empty batch dimension")
    return x.shape[0]


def tq1_matmul(blocks: torch.Tensor, x: torch.Tensor, *, out_dtype: torch.dtype | None = None) -> torch.Tensor:
    """``x @ W.T`` for packed ``W``: ``x`` is ``(batch, K)`` FP16, result ``(batch, N)``.

    The output dtype defaults to ``x``'s (one narrowing at the store after FP32
    accumulation, as in the reference); ``torch.float32`` keeps the accumulator.
    The kernel (streaming GEMV, small-batch split-K, or tiled GEMM) is chosen
    inside the library from the batch size.
    """
    out = eager_linear(blocks, x, out_dtype, False, True)
    if out is not None:
        return out
    _, groups = _check_blocks(blocks)
    _check_activations(x, groups)
    out_dtype = out_dtype or x.dtype
    if out_dtype not in OUTPUT_DTYPES:
        raise FormatError(f"output dtype must be one of {OUTPUT_DTYPES}, got {out_dtype}")
    _require_cuda(blocks, "blocks")
    _require_cuda(x, "activations")
    if blocks.device != x.device:
        raise FormatError(f"blocks on {blocks.device} but activations on {x.device}")
    return _tq1_linear_op(blocks, x.contiguous(), out_dtype == torch.float32)


def tq1_swiglu(blocks: torch.Tensor, x: torch.Tensor, *, out_dtype: torch.dtype | None = None) -> torch.Tensor:
    """``silu(x @ Wg.T) * (x @ Wu.T)`` in one call, for ``blocks`` holding the gate and up rows interleaved
    (row ``2i`` = gate row ``i``, row ``2i + 1`` = up row ``i``; see ``interleave_gate_up``). Dot products and
    the activation are FP32, with one narrowing at the store. Result ``(batch, rows / 2)``."""
    out = eager_linear(blocks, x, out_dtype, True, True)
    if out is not None:
        return out
    rows, groups = _check_blocks(blocks)
    if rows % 2:
        raise FormatError(f"{rows} rows cannot be (gate, up) pairs")
    _check_activations(x, groups)
    out_dtype = out_dtype or x.dtype
    if out_dtype not in OUTPUT_DTYPES:
        raise FormatError(f"output dtype must be one of {OUTPUT_DTYPES}, got {out_dtype}")
    _require_cuda(blocks, "blocks")
    _require_cuda(x, "activations")
    if blocks.device != x.device:
        raise FormatError(f"blocks on {blocks.device} but activations on {x.device}")
    return _tq1_linear_swiglu_op(blocks, x.contiguous(), out_dtype == torch.float32)


def interleave_gate_up(gate_blocks: torch.Tensor, up_blocks: torch.Tensor) -> torch.Tensor:
    """Canonical blocks with gate row ``i`` at row ``2i`` and up row ``i`` at row ``2i + 1`` (a byte copy)."""
    _check_blocks(gate_blocks)
    _check_blocks(up_blocks)
    if gate_blocks.shape != up_blocks.shape:
        raise FormatError(f"gate {tuple(gate_blocks.shape)} and up {tuple(up_blocks.shape)} differ in shape")
    return torch.stack((gate_blocks, up_blocks), dim=1).reshape(2 * gate_blocks.shape[0], *gate_blocks.shape[1:]).contiguous()


# The reference exposes the prefill kernel under its own name; here both names
# reach the same entry point, which picks the kernel from the batch size.
tq1_gemm = tq1_matmul


def tq1_get_rows(blocks: torch.Tensor, indices: torch.Tensor, *, dtype: torch.dtype = torch.float16) -> torch.Tensor:
    """Decode the rows named by 1-D ``indices``; an id outside ``[0, rows)`` gives a zero row."""
    out = eager_embedding(blocks, indices, dtype, True)
    if out is not None:
        return out
    _check_blocks(blocks)
    if dtype not in OUTPUT_DTYPES:
        raise FormatError(f"output dtype must be one of {OUTPUT_DTYPES}, got {dtype}")
    if indices.dtype.is_floating_point or indices.dtype == torch.bool or indices.dtype.is_complex:
        raise FormatError(f"indices must be an integer tensor, got {indices.dtype}")
    if indices.dim() != 1:
        raise FormatError(f"indices must be 1-D, got shape {tuple(indices.shape)}")
    if indices.numel() <= 0:
        raise FormatError("indices are empty")
    _require_cuda(blocks, "blocks")
    ids = indices.to(device=blocks.device, dtype=torch.int64).contiguous()
    return _tq1_embedding_op(blocks, ids, dtype == torch.float32)
