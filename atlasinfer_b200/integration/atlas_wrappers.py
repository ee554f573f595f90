"""``QuantizedLinear`` with the reference's surface, computed by the B200 kernels.

Mirrors ``integration/atlas_wrappers.py:21-83`` of AtlasInfer: a module that
keeps a ``QuantizedTensor`` and an optional bias as plain attributes
(``quantized_weights``, ``bias``, ``original_shape`` -- readable and
re-assignable, absent from ``state_dict``), moves them lazily to the
activations' device, and returns ``x @ W^T + bias``.  Where the reference
dequantizes the whole weight to a cached fp16 copy and calls ``F.linear``
(:56, :67), this module keeps a tile-major uint8 image of the codes beside the
canonical streams and calls the fused dequant GEMV / GEMM of
``libatlas_b200.so``; no fp16 weight is ever materialised.
"""
from __future__ import annotations

import os
import threading
from typing import NamedTuple, Optional

import torch
import torch.nn as nn

from .. import _capi
from ..quant.adaptive_quantizer import QuantizedTensor

# rows of x up to which the per-strip streaming kernel is used (16 rows per pass over the weight); above it the tcgen05
# kernels.  At 16 fp16 rows the per-strip kernel is ahead on small weights (1024 x 1024 3.3 against 4.6 us, 4096 x 4096
# 8.3 against 10.6), even on 12288 x 4096 (21.5, 22.4) and 57344 x 8192 (151, 151) and behind where its strips end in a
# poorly filled wave or K is long (10240 x 8192 36.8 against 30.8, 8192 x 28672 81.5 against 72.1); at 9 rows it is behind
# in three of twelve shapes, by 6 % at most.  The persistent streaming kernel takes up to STREAM_MAX_ROWS rows in one pass; it is what the
# column-parallel linear with the fused gather runs on and can be asked for with force="stream".
GEMV_MAX_ROWS = 16
STREAM_MAX_ROWS = 32
_ANY_ROWS = 1 << 62

_VERBOSE = os.environ.get("ATLAS_VERBOSE", "0") not in ("", "0")


class KernelLayout(NamedTuple):
    """Device-resident kernel image of one quantized [N, K] weight (written by atlas_repack)."""

    source: object                 # the QuantizedTensor it was built from (identity-checked)
    tiles: torch.Tensor            # uint8, tile-major dense codes + 128
    scales_tiled: torch.Tensor     # fp16, [N/128][K/block][128]
    row_ptr: torch.Tensor          # int32 [N + 1], CSR over the canonical outlier streams
    chunk_ptr: torch.Tensor        # int32 [N_padded/16][K/64 + 1]
    entries: torch.Tensor          # int32 (row%16 << 24 | col), strip-major, column-sorted
    vals_sorted: torch.Tensor      # fp16 outlier values in the order of `entries`
    n_rows: int
    n_cols: int
    block_size: int
    ready: Optional[list] = None   # non-empty while the buffers may still be written (see ``_enqueued``)

    def finished(self) -> "KernelLayout":
        """This layout with its buffers final (the host waits for them) and nothing left to wait for."""
        for ready in tuple(self.ready or ()):
            ready.finish()
            _settle(self.ready, ready)
        return self if self.ready is None else KernelLayout(*self[:-1], None)

    def __reduce__(self):
        # copies and pickles read the buffers field by field on whatever stream is current: wait before the first one
        return KernelLayout, tuple(self.finished())


# (device, stream) -> cell of the layouts that the stream was last given to write
_cells = {}
_cells_lock = threading.Lock()


def _enqueued(dev: torch.device) -> list:
    """What a layout that the current stream of ``dev`` was just given to write holds as ``ready``.

    A cell with the event behind the stream's last layout.  The layouts of a stream share a cell until the first look
    that finds the event done empties it, so that all of them are known to be final and later calls look at nothing but
    an empty list.  (First pass of a small layer after loading, one token, six modules in four launches: that look takes
    it from 81 to 86 us; with an event and a new layout per module it was 89.)"""
    with _cells_lock, torch.cuda.device(dev):
        ready = _capi.native().LayoutReady()
        stream = ready.stream
        cell = _cells.get(stream)
        if not cell:   # (an emptied one is that of layouts that are final, and stays empty)
            if len(_cells) >= 16:   # streams that come and go
                for s, old in list(_cells.items()):
                    if not old or old[0].done():
                        old.clear()
                        del _cells[s]
            cell = _cells[stream] = []
        cell[:] = [ready]
        return cell


def _settle(cell: list, ready) -> None:
    """``ready`` was found done: so are the layouts of ``cell``, unless another one has come to it since."""
    try:
        cell.remove(ready)   # (atomic: another thread may have put a later event in its place)
    except ValueError:
        pass


def _pending(layout: "KernelLayout") -> bool:
    """Whether ``layout`` may still be written by the current stream (waits for it if another stream writes it)."""
    for ready in tuple(layout.ready):
        if not ready.wait():
            return True
        _settle(layout.ready, ready)
    return False


_status_words = {}


def status_word(dev: torch.device) -> torch.Tensor:
    """The device int32 kernels set non-zero when a bounded wait ran out (one per device)."""
    t = _status_words.get(dev)   # (a CPU device is a key of its own: its word must not pass for a GPU's)
    if t is None:
        if dev.type == "cuda" and dev.index is None:
            return status_word(torch.device("cuda", torch.cuda.current_device()))
        t = torch.zeros(1, dtype=torch.int32, device=dev)
        _status_words[dev] = t
    return t


def check_status(dev: torch.device) -> None:
    """Synchronise and raise if any kernel on ``dev`` reported a timed-out wait.

    The linear kernels never stall the host: a bounded wait that runs out inside a kernel (a copy that never
    lands, a peer that never arrives) sets a per-device status word and the kernel finishes on what it has.
    ``QuantizedLinear.forward`` does not read the word (that would synchronise every call); a caller that wants
    the check calls this where a synchronisation is acceptable, e.g. once per generated token or per batch.
    The word is cleared when the error is raised."""
    if int(status_word(dev).item()) != 0:
        status_word(dev).zero_()
        raise _capi.AtlasError(_capi.ERR_TIMEOUT, "a quantized-linear kernel gave up on a bounded wait")


_stream_workspaces = {}


def stream_workspace(dev: torch.device) -> torch.Tensor:
    """Scratch of the persistent streaming kernel on ``dev``: tickets and fp32 partial tiles.

    Zero-filled once; every launch leaves it zero-filled where it must be.  One per device: launches that use it
    must be ordered with respect to each other."""
    index = dev.index if dev.index is not None else torch.cuda.current_device()
    t = _stream_workspaces.get(index)
    if t is None:
        L = _capi.load()
        t = torch.zeros(int(L.atlas_qlinear_stream_workspace_bytes(STREAM_MAX_ROWS)), dtype=torch.uint8, device=dev)
        _stream_workspaces[index] = t
    return t


def kernel_layout_supported(shape, block_size: int) -> Optional[str]:
    """``None`` if a weight of ``shape`` can use the fused kernels, else the reason."""
    if len(shape) != 2:
        return f"weight must be 2-D, got shape {tuple(shape)}"
    k = int(shape[1])
    if k % 64 != 0:
        return f"in_features {k} is not a multiple of 64"
    if block_size % 16 != 0 or k % block_size != 0:
        return f"block_size {block_size} must be a multiple of 16 that divides in_features {k}"
    return None


def build_kernel_layout(q: QuantizedTensor, wait: bool = True) -> KernelLayout:
    """Expand the compacted code stream of ``q`` (on a CUDA device) into the kernel layout."""
    return build_joined_layout([q], wait)[0]


def build_joined_layout(qs, wait: bool = True):
    """The kernel layouts of ``qs`` (one device, in_features and block size) as the rows of one layout, back to back.

    Returns ``(layout, row offsets)``.  Every member but the last is padded to whole 128-row tiles, as in
    ``concat_layouts``, but the members are expanded straight into the joined buffers by one launch.  The CSR row
    pointers of the canonical streams are only written for a single tensor.

    With ``wait`` the buffers are final on return.  Without, ``layout.ready`` stands for the work under way:
    ``quantized_linear_forward`` may be called at once (it launches plainly until the work is done), any other use
    outside the current stream waits for it."""
    for q in qs:
        reason = kernel_layout_supported(q.original_shape, int(q.block_size))
        if reason is not None:
            raise NotImplementedError("QuantizedLinear: " + reason)
    dev = qs[0].fp8_data.device
    k, bs = int(qs[0].original_shape[1]), int(qs[0].block_size)
    if any((int(q.original_shape[1]), int(q.block_size)) != (k, bs) for q in qs):
        raise ValueError("fused linears must share in_features and block size")
    rows = [int(q.original_shape[0]) for q in qs]
    native = _capi.native()
    if torch.cuda.is_current_stream_capturing():
        torch.cuda.current_stream(dev).synchronize()   # raises: a layout must not live in a graph's memory
    members = [(q.fp8_data, q.fp16_outliers, q.outlier_indices, q.scale_factors, n) for q, n in zip(qs, rows)]
    buffers = native.build_layout(members, k, bs)
    ready = None
    if wait:
        torch.cuda.current_stream(dev).synchronize()
    else:
        ready = _enqueued(dev)
    offsets, row = [], 0
    for n in rows:
        offsets.append(row)
        row += (n + 127) // 128 * 128
    source = qs[0] if len(qs) == 1 else tuple(qs)
    return KernelLayout(source, *buffers, offsets[-1] + rows[-1], k, bs, ready), offsets


def quantized_linear_forward(x: torch.Tensor, layout: KernelLayout, bias: Optional[torch.Tensor],
                             force: Optional[str] = None) -> torch.Tensor:
    """``x @ W^T + bias`` on CUDA tensors through the C ABI.

    ``force``: "gemv" (per-strip streaming kernel), "gemm" (tcgen05 kernel) or "stream" (persistent streaming
    kernel, one pass for up to 32 rows); default: "gemv" up to 16 rows of x, "gemm" above."""
    if x.dtype is not torch.float16 and x.dtype is not torch.bfloat16:
        raise RuntimeError(f"QuantizedLinear expects fp16 (or bf16) activations, got {x.dtype}")
    if force is None:
        gemv_rows = GEMV_MAX_ROWS
    elif force == "stream":
        return _stream_forward(x, layout, bias)
    elif force in ("gemv", "gemm"):
        gemv_rows = _ANY_ROWS if force == "gemv" else 0
    else:
        raise ValueError(f"force={force!r}")
    pending = bool(layout.ready) and _pending(layout)
    return _capi.native().linear(x, layout.tiles, layout.scales_tiled, layout.chunk_ptr, layout.entries, layout.vals_sorted,
                                 layout.n_rows, layout.n_cols, layout.block_size, bias, status_word(x.device), gemv_rows, pending)


def _stream_forward(x: torch.Tensor, layout: KernelLayout, bias: Optional[torch.Tensor]) -> torch.Tensor:
    """``quantized_linear_forward`` on the persistent streaming kernel."""
    L = _capi.load()
    dev = x.device
    n, k = layout.n_rows, layout.n_cols
    if x.shape[-1] != k:
        raise RuntimeError(f"QuantizedLinear: input has {x.shape[-1]} features, weight expects {k}")
    pending = bool(layout.ready) and _pending(layout)
    x2 = x.reshape(-1, k)
    if x2.stride(-1) != 1 or (x2.shape[0] > 1 and x2.stride(0) < k):
        x2 = x2.contiguous()
    m = x2.shape[0]
    ldx = x2.stride(0) if m > 1 else k
    y = torch.empty((m, n), dtype=x.dtype, device=dev)
    if m:
        b = None if bias is None else bias.to(torch.float16).contiguous()
        ws = stream_workspace(dev)
        # (a bias converted just now, like a layout still under way, is written by the kernels in front)
        was = L.atlas_qlinear_plain_launch(1) if pending or b is not bias else None
        try:
            with torch.cuda.device(dev):
                status = L.atlas_qlinear_stream(
                    x2.data_ptr(), _capi.DTYPE_F16 if x.dtype == torch.float16 else _capi.DTYPE_BF16, m, ldx,
                    layout.tiles.data_ptr(), layout.scales_tiled.data_ptr(), layout.chunk_ptr.data_ptr(),
                    _capi.ptr(layout.entries), _capi.ptr(layout.vals_sorted), n, k, layout.block_size, _capi.ptr(b),
                    y.data_ptr(), n, ws.data_ptr(), ws.numel(), status_word(dev).data_ptr(), _capi.stream_ptr(dev))
        finally:
            if was is not None:
                L.atlas_qlinear_plain_launch(was)
        _capi.check(status, "atlas_qlinear_stream")
    return y.view(*x.shape[:-1], n)


def concat_layouts(layouts) -> KernelLayout:
    """One kernel layout whose rows are those of ``layouts`` back to back (same in_features and block size).

    Every member but the last is padded to a whole number of 128-row tiles (its own layout already is), so a
    member is a contiguous run of tiles, scales and strips of the result, and one launch over the result
    computes all members.  Row ``i`` of member ``j`` is row ``offsets[j] + i`` of the result."""
    first = layouts[0]
    if any(l.n_cols != first.n_cols or l.block_size != first.block_size for l in layouts):
        raise ValueError("fused linears must share in_features and block size")
    k_tiles = first.n_cols // 64
    chunk_ptrs, base = [], 0
    for l in layouts:
        if l.ready:
            _pending(l)
        chunk_ptrs.append(l.chunk_ptr + base)          # entry indices become positions in the joined list
        base += l.entries.numel()
    padded = [(l.n_rows + 127) // 128 * 128 for l in layouts]
    n_rows = sum(padded[:-1]) + layouts[-1].n_rows
    dev = first.tiles.device
    row_ptr = torch.empty(0, dtype=torch.int32, device=dev)   # CSR view of the canonical streams: not joined
    assert all(l.chunk_ptr.numel() == (p_ // 16) * (k_tiles + 1) for l, p_ in zip(layouts, padded))
    return KernelLayout(tuple(l.source for l in layouts), torch.cat([l.tiles for l in layouts]),
                        torch.cat([l.scales_tiled for l in layouts]), row_ptr, torch.cat(chunk_ptrs),
                        torch.cat([l.entries for l in layouts]), torch.cat([l.vals_sorted for l in layouts]),
                        n_rows, first.n_cols, first.block_size)


def slice_layout(fused: KernelLayout, row_offset: int, n_rows: int, source, entry_count: Optional[int] = None) -> KernelLayout:
    """The member of a fused layout that starts at ``row_offset`` (a multiple of 128), as views of its buffers."""
    if row_offset % 128:
        raise ValueError("members of a fused layout start on 128-row boundaries")
    k, bs = fused.n_cols, fused.block_size
    k_tiles = k // 64
    n_pad = (n_rows + 127) // 128 * 128
    t0, s0, c0 = row_offset * k, row_offset * (k // bs), (row_offset // 16) * (k_tiles + 1)
    return KernelLayout(source, fused.tiles[t0:t0 + n_pad * k], fused.scales_tiled[s0:s0 + n_pad * (k // bs)],
                        fused.row_ptr, fused.chunk_ptr[c0:c0 + (n_pad // 16) * (k_tiles + 1)],
                        fused.entries, fused.vals_sorted, n_rows, k, bs, fused.ready)


class FusedLinearGroup:
    """Several ``QuantizedLinear`` layers that read the same activations, computed by one launch.

    The reference issues q/k/v (and gate/up) as separate ``F.linear`` calls on the same input
    (integration/atlas_wrappers.py:67, once per module).  Here the members' kernel layouts are joined row-wise
    (``concat_layouts``); the first member that is called with an input computes the joined product and the
    other members, called with the very same tensor, return their slice of it (for prompt-sized inputs this
    also means one bf16 -> fp16 conversion of the activations instead of one per member).  A member called
    with any other input computes the joined product anew.  A member's slice equals its stand-alone output up to the rounding of
    the fp32 partial sums (the K range of a row tile is cut between CTAs at other places when the launch
    covers more rows), not bit for bit.
    """

    def __init__(self, members):
        self.members = list(members)
        self.layout: Optional[KernelLayout] = None
        self.bias: Optional[torch.Tensor] = None
        self.offsets = []
        self._cache = None      # (x, x._version, y_all, members served)
        self.launches = 0       # joined launches issued (for tests and launch counting)
        for i, mod in enumerate(self.members):
            mod._group = self
            mod._group_index = i

    def build(self, dev: torch.device) -> None:
        for mod in self.members:
            q = mod.quantized_weights
            if q.fp8_data.device != dev:
                mod.quantized_weights = q.to(dev)
            if mod.bias is not None and mod.bias.device != dev:
                mod.bias = mod.bias.to(dev)
        sources = [mod.quantized_weights for mod in self.members]
        if any(mod._has_layout_for(q) for mod, q in zip(self.members, sources)):
            # members that are laid out already are joined as they are
            layouts = [mod._layout_for(q) for mod, q in zip(self.members, sources)]
            fused = concat_layouts(layouts)
            self.offsets, off = [], 0
            for lay in layouts:
                self.offsets.append(off)
                off += (lay.n_rows + 127) // 128 * 128
        else:
            fused, self.offsets = build_joined_layout(sources, wait=False)
        rows = [int(q.original_shape[0]) for q in sources]
        if any(mod.bias is not None for mod in self.members):
            b = torch.zeros(fused.n_rows, dtype=torch.float16, device=dev)
            for mod, n, o in zip(self.members, rows, self.offsets):
                if mod.bias is not None:
                    b[o:o + n] = mod.bias.to(torch.float16)
            self.bias = b
            if fused.ready is not None:   # the bias is part of what a use waits for
                fused = fused._replace(ready=_enqueued(dev))
        # the members now look at the joined buffers; their own copies are released
        for mod, q, n, o in zip(self.members, sources, rows, self.offsets):
            mod._kernel_layout = slice_layout(fused, o, n, q)
        self.layout = fused
        if fused.ready is None:
            torch.cuda.current_stream(dev).synchronize()

    def member_forward(self, index: int, x: torch.Tensor) -> Optional[torch.Tensor]:
        """Member ``index``'s output for ``x``, or None if the group does not apply (the member computes alone)."""
        if not x.is_cuda or (x.dtype is not torch.float16 and x.dtype is not torch.bfloat16) or x.numel() == 0:
            return None
        if self.layout is None or self.layout.tiles.device != x.device:
            self.build(x.device)
        c = self._cache
        if c is None or c[0] is not x or c[1] != x._version or index in c[3]:
            y_all = quantized_linear_forward(x, self.layout, self.bias)
            self.launches += 1
            c = (x, x._version, y_all, set())
            self._cache = c
        c[3].add(index)
        off = self.offsets[index]
        n = self.members[index].original_shape[0]
        out = c[2].narrow(-1, off, n)
        if len(c[3]) == len(self.members):
            self._cache = None   # everyone has been served: do not keep x and y alive
        return out


def fuse_linears(members) -> FusedLinearGroup:
    """Join ``QuantizedLinear`` layers that share their input (e.g. q/k/v, gate/up) into one launch."""
    members = list(members)
    shapes = {(tuple(m.original_shape)[1], int(m.quantized_weights.block_size)) for m in members}
    if len(shapes) != 1:
        raise ValueError(f"fused linears must share in_features and block size, got {sorted(shapes)}")
    return FusedLinearGroup(members)


class QuantizedLinear(nn.Module):
    """A linear layer whose weight is a ``QuantizedTensor`` (reference :21-83)."""

    def __init__(self, quantized_weights: "QuantizedTensor", bias: Optional[torch.Tensor]):
        super().__init__()
        self.quantized_weights = quantized_weights
        self.bias = bias
        self.original_shape = getattr(quantized_weights, "original_shape", None)
        self._kernel_layout: Optional[KernelLayout] = None
        self._group: Optional[FusedLinearGroup] = None   # set by fuse_linears
        self._group_index = 0
        self._bias_f16 = None   # (bias it was made from, its fp16 contiguous image)

    def _bias_for(self, bias: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
        """The bias as the kernels want it (fp16, contiguous), converted once per bias tensor and made
        final before any kernel that reads it is launched."""
        if bias is None or (bias.dtype == torch.float16 and bias.is_contiguous()):
            return bias
        cached = self._bias_f16
        if cached is None or cached[0] is not bias:
            image = bias.to(torch.float16).contiguous()
            if image.device.type == "cuda":
                torch.cuda.current_stream(image.device).synchronize()
            cached = (bias, image)
            self._bias_f16 = cached
        return cached[1]

    def _has_layout_for(self, q: QuantizedTensor) -> bool:
        lay = self._kernel_layout
        return lay is not None and lay.source is q and lay.tiles.device == q.fp8_data.device

    def _layout_for(self, q: QuantizedTensor) -> KernelLayout:
        if not self._has_layout_for(q):
            self._kernel_layout = build_kernel_layout(q, wait=False)
        return self._kernel_layout

    def offload_canonical(self, device="cpu") -> None:
        """Keep only the kernel layout on the GPU: the canonical streams move to ``device`` (host by default).

        The module then holds ~1.03 bytes per weight of GPU memory instead of ~2.07 (canonical streams +
        kernel layout).  ``quantized_weights`` stays a complete ``QuantizedTensor`` (for saving, dequantizing,
        ``memory_footprint``); the forward keeps using the layout that was built from it."""
        q = self.quantized_weights
        dev = q.fp8_data.device
        if dev.type != "cuda":
            return
        lay = self._layout_for(q)
        moved = q.to(torch.device(device))
        self.quantized_weights = moved
        if self._group is not None and self._group.layout is not None:
            srcs = tuple(moved if s_ is q else s_ for s_ in self._group.layout.source)
            self._group.layout = self._group.layout._replace(source=srcs)
        self._kernel_layout = lay._replace(source=moved)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        q_tensor = self.quantized_weights
        if not hasattr(q_tensor, "fp8_data"):
            raise TypeError(
                f"Weight in QuantizedLinear ({id(self)}) is not a valid QuantizedTensor: {type(q_tensor)}")
        if self._group is not None:
            y = self._group.member_forward(self._group_index, x)
            if y is not None:
                return y
        lay = self._kernel_layout
        bias = self.bias
        if lay is not None and lay.source is q_tensor and x.is_cuda and lay.tiles.device == x.device and (
                bias is None or bias.device == x.device):
            return quantized_linear_forward(x, lay, self._bias_for(bias))
        # the kernels need a GPU; CPU activations are staged through it and the result returned
        compute_device = x.device if x.device.type == "cuda" else _capi.require_cuda()
        if lay is not None and lay.source is q_tensor and lay.tiles.device == compute_device:
            # the kernel image of these very streams is already on the device (the streams themselves may have
            # been moved off it by offload_canonical)
            bias = self.bias
            if bias is not None and bias.device != compute_device:
                self.bias = bias.to(compute_device)
                bias = self.bias
            xin = x if x.device == compute_device else x.to(compute_device)
            y = quantized_linear_forward(xin, lay, self._bias_for(bias))
            return y if x.device == compute_device else y.to(x.device)
        if q_tensor.fp8_data.device != compute_device:
            if _VERBOSE:
                print(f"QuantizedLinear {id(self)}: weights {q_tensor.fp8_data.device} -> {compute_device}")
            self.quantized_weights = q_tensor.to(compute_device)
            q_tensor = self.quantized_weights
        bias = self.bias
        if bias is not None and bias.device != compute_device:
            self.bias = bias.to(compute_device)
            bias = self.bias
        layout = self._layout_for(q_tensor)
        xin = x if x.device == compute_device else x.to(compute_device)
        y = quantized_linear_forward(xin, layout, self._bias_for(bias))
        return y if x.device == compute_device else y.to(x.device)

    def extra_repr(self) -> str:
        q_shape, q_device = None, "N/A"
        if getattr(self, "quantized_weights", None):
            q_shape = self.original_shape
            try:
                q_device = self.quantized_weights.fp8_data.device
            except AttributeError:
                pass
        return f"quantized_shape={q_shape}, bias={self.bias is not None}, device={q_device}"
