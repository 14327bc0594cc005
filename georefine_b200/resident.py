"""The resident image of a weight (layout: csrc/bxr_format.h) and the fused entry points over it.

``ResidentWeight`` follows the descriptor protocol of the reference's serving engines
(``glc_serve/fastdec.py:172-188`` ``Lin``, ``glc_serve/tbe_desc.py:127-157`` ``TBELin``,
``glc_serve/bigemm.py:468-507`` ``BILin``): attributes ``kind``, ``N``, ``K``, ``bytes``, ``coded_bytes`` and
``__call__(x[M,K], y[M,N])`` writing into a preallocated ``y`` with no allocation (but the scratch that batches above
128 rows borrow, see ``gemm``) and no host synchronisation, so a call can be captured in a CUDA graph.
"""
from __future__ import annotations

import ctypes
import hashlib

import numpy as np

from . import _native

GEMV_MAX_M = 8
LAYOUTS = {"rans": 0, "raw": 1, "window": 2, "window4": 3}   # bxr_format.h: BXR_MODE_CODED / _RAW / _WINDOW / _WINDOW4
DEFAULT_LAYOUT = "window4"                       # the fastest layout (12 bits/weight); "window" 11.3, "rans" 11.1 bits/weight


_BF16 = None


def _bfloat16():
    global _BF16
    if _BF16 is None:
        import torch

        _BF16 = torch.bfloat16
    return _BF16


def _current_device() -> int:
    import torch

    return torch._C._cuda_getDevice()


def sm_count(device) -> int:
    import torch

    return torch.cuda.get_device_properties(device).multi_processor_count


def _of_a_graph(block) -> bool:
    """Did the allocator take the block from the private pool of a capture?"""
    import torch

    at = block.data_ptr()
    return any(s["address"] <= at < s["address"] + s["total_size"] and tuple(s["segment_pool_id"]) != (0, 0) for s in torch.cuda.memory_snapshot())


def default_workers(rows: int, cols: int, sms: int) -> int:
    """How many persistent CTAs an image is built for when the caller does not say: one per SM, except for small
    weights with fewer 128-row blocks than SMs, where a multiple of the row-block count is better when it costs few
    extra chunks per CTA: every row block is then cut into the same few whole CTAs (no CTA holds the tail of one row
    block and the head of the next), which shortens the partial-tile exchange at the end of a launch (measured on a
    B200: 5120 x 5120 with 120 instead of 148 CTAs 15.1 vs 16.7 us at M = 64, 17.9 vs 19.9 us at M = 128, level at M = 1;
    5120 x 17408 with 120 CTAs is slower, 30.3 vs 28.0 us: there the streaming dominates)."""
    row_blocks, chunks = -(-rows // 128), -(-cols // 128)
    if row_blocks >= sms or row_blocks == 0:
        return sms
    per_cta = row_blocks * chunks / sms
    aligned = row_blocks * (sms // row_blocks)
    if per_cta <= 16 and row_blocks * chunks / aligned - per_cta <= 5:
        return aligned
    return sms


def build_image(words, workers: int, *, threads: int = 0, layout: str = DEFAULT_LAYOUT, force_raw: bool = False,
                source_sha256: bytes | None = None):
    """Host: BF16 words [rows, cols] -> (image bytes as uint8 array, header).

    layout: "window4" (fixed 4-bit exponent codes in a 16-binade row window: 12 bits/weight, the fastest to decode,
    operand through tensor memory), "window" (fixed 3-bit codes in an 8-binade window with per-chunk exception lists:
    11.3 bits/weight), "rans" (entropy-coded exponent streams: 11.1 bits/weight) or "raw" (plain tiles).  The builder
    demotes window4 / window -> rans -> raw when a chunk does not fit its slot; the header's ``mode`` says what was
    built."""
    mode = LAYOUTS["raw"] if force_raw else LAYOUTS[layout]
    a = np.ascontiguousarray(words, dtype=np.uint16)
    if a.ndim != 2 or not all(a.shape):
        raise ValueError("expected a non-empty 2-D uint16 array")
    if source_sha256 is None:
        source_sha256 = hashlib.sha256(a.astype("<u2").tobytes()).digest()
    digest = (ctypes.c_uint8 * 32).from_buffer_copy(source_sha256)
    ptr, size = _native.U8P(), ctypes.c_uint64()
    lib = _native.lib()
    status = lib.bxr_build(a.ctypes.data_as(_native.U16P), a.shape[0], a.shape[1], int(workers), int(threads),
                           mode, digest, ctypes.byref(ptr), ctypes.byref(size))
    if status:
        raise RuntimeError(f"bxr_build failed ({status})")
    try:
        image = np.ctypeslib.as_array(ptr, shape=(size.value,)).copy()
    finally:
        lib.bxr_free(ptr)
    return image, header_of(image)


def header_of(image) -> _native.BxrHeader:
    return _native.BxrHeader.from_buffer_copy(image[:ctypes.sizeof(_native.BxrHeader)].tobytes())


def validate_image(image) -> None:
    """Structural check of an image (layout version, offsets, work partition, blob index) before anything follows an
    offset inside it; raises ValueError.  Cheap: the blobs themselves are not read."""
    a = np.ascontiguousarray(image, dtype=np.uint8)
    if _native.lib().bxr_validate(a.ctypes.data_as(_native.U8P), a.size):
        raise ValueError("resident image is malformed or was built by another version of the layout")


def decode_image_host(image) -> np.ndarray:
    """Host twin of the GPU decoder; used to bind an image to its source digest before upload."""
    h = header_of(image)
    out = np.empty((h.rows, h.cols), dtype=np.uint16)
    status = _native.lib().bxr_decode_host(image.ctypes.data_as(_native.U8P), image.size, out.ctypes.data_as(_native.U16P))
    if status:
        raise ValueError(f"resident image is malformed ({status})")
    return out


def largest_block(sizes, device):
    """Device memory of the first of the (falling) sizes that there is room for; None if there is none for any."""
    import torch

    for size in sizes:
        try:
            return torch.empty(size, device=device, dtype=torch.uint8)
        except torch.cuda.OutOfMemoryError:
            pass
    return None


class ResidentWeight:
    kind = "bctx"

    def __init__(self, image: np.ndarray, device, *, max_m: int = 128, verify: bool = True):
        import torch

        validate_image(image)   # always: the kernels follow the image's offsets without further checks
        self.header = header_of(image)
        h = self.header
        if verify:
            words = decode_image_host(image)
            if hashlib.sha256(words.astype("<u2").tobytes()).digest() != bytes(h.source_sha256):
                raise ValueError("resident image does not reproduce its source digest")
        self.device = torch.device(device)
        if self.device.index is None:
            self.device = torch.device(self.device.type, torch.cuda.current_device())
        self.N, self.K = int(h.rows), int(h.cols)
        self.mode = int(h.mode)
        self.image = torch.from_numpy(image).to(self.device)
        self.status = torch.zeros(1, device=self.device, dtype=torch.int32)
        self.max_m = 0
        self.workspace, self._outgrown = None, []
        sizes = [int(_native.lib().grb_bxr_workspace_bytes(ctypes.byref(h), m)) for m in (128, 129)]
        self._counter_bytes = counters = (int(h.row_blocks) * 4 + 255) & ~255
        # partial tiles of the widest passes of a batch above 128 rows, where they are larger than those of 128 rows
        self.wide_scratch_bytes = sizes[1] - counters if sizes[1] > sizes[0] else 0
        # the block sizes that make a difference: the partial tiles of passes of 384, 256 and 192 rows, as far as the image has them
        row = int(h.partial_slots) * 512
        self.wide_scratch_sizes = [rows * row for rows in (384, 256, 192) if 0 < rows * row <= self.wide_scratch_bytes]
        self.next_weight = None     # see then()
        self.reserve(max_m)

    @classmethod
    def from_words(cls, words, device, *, source_sha256=None, max_m=128, workers=None, layout=None, force_raw=False,
                   verify=True, tune=None):
        """Builds the image on the host and uploads it.  ``layout`` / ``workers`` left to None come from ``tune`` (a
        mapping {(N, K): (layout, workers)} as ``georefine_b200.tune.load_tune`` returns it) when it knows the shape,
        else from the defaults: the 4-bit window layout and ``default_workers``."""
        rows, cols = int(words.shape[0]), int(words.shape[1])
        if tune and (rows, cols) in tune:
            tuned_layout, tuned_workers = tune[(rows, cols)]
            layout = tuned_layout if layout is None else layout
            workers = tuned_workers if workers is None else workers
        layout = DEFAULT_LAYOUT if layout is None else layout
        workers = default_workers(rows, cols, sm_count(device)) if workers is None else workers
        image, _ = build_image(words, workers, layout=layout, force_raw=force_raw, source_sha256=source_sha256)
        return cls(image, device, max_m=max_m, verify=verify)

    def clone(self):
        """A second copy of the image in device memory (benchmarks rotate over copies to defeat the L2)."""
        import copy

        other = copy.copy(self)
        other.image = self.image.clone()
        other.status = self.status.clone()
        other.workspace, other._outgrown = self.workspace.clone(), []
        other.next_weight = None
        return other

    # -- bookkeeping (the numerators of the roofline) ----------------------------------------------------
    @property
    def bytes(self) -> int:
        return int(self.header.total_bytes)

    @property
    def coded_bytes(self) -> int:
        """Bytes one pass of a fused kernel streams from HBM: chunk blobs, restart states, blob index."""
        return int(self.header.coded_bytes)

    @property
    def resident_bytes(self) -> int:
        return self.bytes + sum(ws.numel() for ws in (self.workspace, *self._outgrown)) + 4

    def backend_identity(self):
        h = self.header
        return {"format": "BXR1", "mode": self.mode, "workers": int(h.workers), "items": int(h.items),
                "partial_slots": int(h.partial_slots), "library": str(_native.library_path().name)}

    def _scratch_bytes(self, m: int) -> int:
        size = _native.lib().grb_bxr_workspace_bytes
        return max(256, *(int(size(ctypes.byref(self.header), rows)) for rows in (min(m, 128), GEMV_MAX_M)))

    def reserve(self, max_m: int) -> None:
        """Scratch for batches up to max_m rows (FP32 partial tiles + counters); zero-filled once.  Batches above 128 rows need
        no more of it.  Scratch that it replaces lives as long as the weight: a captured graph may have its address."""
        import torch

        max_m = max(int(max_m), GEMV_MAX_M)
        if max_m <= self.max_m:
            return
        need = self._scratch_bytes(max_m)
        if self.workspace is None or need > self.workspace.numel():
            if self.workspace is not None:
                self._outgrown.append(self.workspace)
            self.workspace = torch.zeros(need, device=self.device, dtype=torch.uint8)
        self.max_m = max_m

    def _capturing(self) -> bool:
        import torch

        with torch.cuda.device(self.device):
            return torch.cuda.is_current_stream_capturing()

    def _lent_scratch(self, capturing: bool):
        """Partial tiles for one batch above 128 rows, from the stream's allocator and back to it after the call: all weights of
        a stack share one block, and one graph's share a block of the graph's own pool.  Where the widest passes' do not fit
        the memory, those of narrower ones are asked for.  None - the batch then runs in passes of 128 rows - when none do, or
        a capture that the allocator does not know of is under way, whose graph could not keep the block."""
        block = largest_block(self.wide_scratch_sizes, self.device)
        return block if block is None or not capturing or _of_a_graph(block) else None

    # -- device entry points -------------------------------------------------------------------------
    def _stream(self):
        import torch

        return torch.cuda.current_stream(self.device).cuda_stream

    def decode(self, *, check=True):
        """Dense BF16 [N, K] decoded from the image by the decode twin of the fused kernels.  What it reports joins what the
        status word already holds (an earlier product's timeout among it); ``check`` looks at this call's own report."""
        import torch

        out = torch.empty((self.N, self.K), device=self.device, dtype=torch.bfloat16)
        status = torch.zeros_like(self.status) if check else self.status
        with torch.cuda.device(self.device):
            st = _native.lib().grb_bxr_decode(self.image.data_ptr(), ctypes.byref(self.header), out.data_ptr(),
                                              status.data_ptr(), self._stream())
        _native.check(st, "grb_bxr_decode")
        if check and status.item() != 0:
            self.status |= status
            raise ValueError(f"resident decode reported status {status.item()}")
        return out

    def _checked(self, x, y):
        """The batch size of a call, its shapes and types checked."""
        m, k = x.shape
        rows, n = y.shape
        if x.dtype is not _bfloat16() or y.dtype is not _BF16:
            raise ValueError("x and y must be 2-D BF16 tensors")
        if k != self.K or rows != m or n != self.N or x.stride(1) != 1 or y.stride(1) != 1:
            raise ValueError("shape mismatch: x [M, K], y [M, N], unit inner stride")
        return m

    def _within_reserve(self, m):
        if min(m, 128) > min(self.max_m, 128):
            raise ValueError(f"batch of {m} rows exceeds the reserved scratch ({self.max_m}); call reserve() first")

    def then(self, next_weight):
        """Tells this weight which one the stream multiplies by next (None: nobody).  A hint for the kernel: while a
        launch over this weight winds down, the L2 is asked for the first blobs of the next one.  Returns
        ``next_weight`` so that a layer can be chained in one line: ``qkv.then(o).then(gate_up).then(down)``."""
        self.next_weight = next_weight
        return next_weight

    def gemm(self, x, y, bias=None, *, scratch=None):
        """tcgen05 path, any M; rows of y are bitwise independent of M.

        A batch above 128 rows may take 192 or 384 rows per pass over the weights.  For their partial tiles it borrows ``scratch``
        (uint8, ``wide_scratch_bytes`` of it, not used by anything else until the call's work is done), or asks the allocator."""
        if x.dim() != 2 or y.dim() != 2:
            raise ValueError("x and y must be 2-D BF16 tensors")
        m = self._checked(x, y)
        if not m:
            return
        if m > self.max_m:
            self._within_reserve(m)
        self._multiply(x, y, bias, m, self.workspace, scratch)

    def _multiply(self, x, y, bias, m, workspace, scratch):
        if m > 128 and scratch is None:
            capturing = self._capturing()
            if not capturing:
                self.max_m = max(self.max_m, m)
            scratch = self._lent_scratch(capturing)
        nxt, index = self.next_weight, self.device.index
        call, entry = _native.gemm_partials()
        args = (entry, self.image.data_ptr(), ctypes.addressof(self.header), x.data_ptr(), x.stride(0), m, y.data_ptr(), y.stride(0),
                0 if bias is None else bias.data_ptr(), workspace.data_ptr(), workspace.numel(), 0 if scratch is None else scratch.data_ptr(),
                0 if scratch is None else scratch.numel(), self.status.data_ptr(), _native.raw_stream(index),
                0 if nxt is None else nxt.image.data_ptr(), 0 if nxt is None else ctypes.addressof(nxt.header))
        if _current_device() == index:   # the usual case: skip the device switch
            st = call(*args)
        else:
            import torch

            with torch.cuda.device(self.device):
                st = call(*args)
        if st:
            _native.check(st, "grb_bxr_gemm")

    def gemv(self, x, y, bias=None):
        """CUDA-core path, M <= 8; rows of y are bitwise independent of M within 1..8."""
        import torch

        if x.dim() != 2 or y.dim() != 2:
            raise ValueError("x and y must be 2-D BF16 tensors")
        m = self._checked(x, y)
        if not m:
            return
        self._within_reserve(m)
        with torch.cuda.device(self.device):
            st = _native.lib().grb_bxr_gemv(self.image.data_ptr(), ctypes.byref(self.header), x.data_ptr(), x.stride(0), m, y.data_ptr(), y.stride(0),
                                            None if bias is None else bias.data_ptr(), self.workspace.data_ptr(), self.workspace.numel(),
                                            self.status.data_ptr(), self._stream())
        if st:
            _native.check(st, "grb_bxr_gemv")

    def __call__(self, x, y):
        self.gemm(x, y)

    def linear(self, x, out=None, bias=None):
        import torch

        lead = x.shape[:-1]
        x2 = x if len(lead) == 1 else x.reshape(-1, x.shape[-1])
        if x2.stride(-1) != 1 or x2.stride(0) % 8 or x2.data_ptr() % 16:
            if self.K % 8:  # the kernels want a row stride that is a multiple of 16 bytes
                padded = torch.zeros((x2.shape[0], (self.K + 7) // 8 * 8), device=self.device, dtype=torch.bfloat16)
                padded[:, :self.K] = x2
                x2 = padded[:, :self.K]
            else:
                x2 = x2.contiguous()
        m = x2.shape[0]
        if out is not None:
            y = out.reshape(-1, self.N)
        elif x.dtype is _bfloat16() and x.device == self.device:
            y = x.new_empty((m, self.N))
        else:
            y = torch.empty((m, self.N), device=self.device, dtype=torch.bfloat16)
        if m > self.max_m and min(m, 128) > min(self.max_m, 128):
            if self._capturing():
                # Scratch of the graph's own pool, for this call only: its zero fill is the graph's, and nothing outside the
                # graph may count on it.
                if self._checked(x2, y):
                    self._multiply(x2, y, bias, m, torch.zeros(self._scratch_bytes(m), device=self.device, dtype=torch.uint8), None)
                return y if len(lead) == 1 and out is None else y.reshape(*lead, self.N)
            self.reserve(min(m, 128))
        self.gemm(x2, y, bias)
        return y if len(lead) == 1 and out is None else y.reshape(*lead, self.N)

    def check_status(self) -> int:
        """Host read of the device status word (synchronises); 0 means every call since the last reset was clean."""
        return int(self.status.item())

    def reset(self) -> None:
        """After a nonzero ``check_status()``: waits for the device, then clears the counters of the scratch - a launch that gave
        up may have counted parts that nobody added, and the next one would add tiles of it - and the status word."""
        import torch

        torch.cuda.synchronize(self.device)
        for scratch in (self.workspace, *self._outgrown):
            scratch[:self._counter_bytes].zero_()
        self.status.zero_()
        torch.cuda.synchronize(self.device)
