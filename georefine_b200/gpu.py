"""Indexed CUDA decoding of BCTX frames and the fused linear over their resident image.

Mirrors ``context-runtime/georefine_context_runtime/bitexact_context_gpu.py``: ``checkpoints`` (:51-63),
``index_frame`` (:66-106) and ``CudaContextTensor`` (:109-168) keep their names, arguments, attributes and
errors.  The tensor gains ``linear(x, out=None)`` / ``__call__(x, y)``: the seam the reference reserves for "a
backend with a fused GEMM" (bitexact_context_serving.py:3-5).  Everything that touches the GPU goes through
the C ABI of libgeorefine_b200.so; there is no other path.
"""
from __future__ import annotations

import ctypes
import hashlib
import math

import numpy as np

from . import _native
from . import codec as base
from .resident import ResidentWeight, sm_count


def _p(a, t):
    return a.ctypes.data_as(ctypes.POINTER(t))


def _walk_stream(stream, table, row_class, col_class, shape, nr, nc, stride, conditioning):
    """One serial pass of the host coder over a stream (``bcx_checkpoint``): the symbols, and the decoder's state and
    byte offset in front of every ``stride``-th symbol.  ``conditioning`` = the main symbols when the stream is the
    conditional residual stream, else None."""
    rows, cols = shape
    count = rows * cols
    blocks = -(-count // stride)
    states, offsets = np.empty(blocks, dtype=np.uint32), np.empty(blocks, dtype=np.uint32)
    symbols = np.empty(count, dtype=np.uint16)
    data = np.frombuffer(bytes(stream), dtype=np.uint8).copy() if len(stream) else np.zeros(1, dtype=np.uint8)
    table = np.ascontiguousarray(table, dtype="<u4")
    row_class = np.ascontiguousarray(row_class, dtype=np.uint8)
    col_class = np.ascontiguousarray(col_class, dtype=np.uint8)
    kind = 0 if conditioning is None else 1
    context = _native.U16P() if conditioning is None else _p(np.ascontiguousarray(conditioning, dtype=np.uint16), ctypes.c_uint16)
    status = _native.lib().bcx_checkpoint(_p(data, ctypes.c_uint8), len(stream), count, rows, cols, _p(row_class, ctypes.c_uint8),
                                          _p(col_class, ctypes.c_uint8), nr, nc, kind, context, _p(table, ctypes.c_uint32), stride,
                                          _p(states, ctypes.c_uint32), _p(offsets, ctypes.c_uint32), _p(symbols, ctypes.c_uint16))
    if status:
        raise base.CodecError(f"checkpoint validation failed ({status})")
    return states, offsets, symbols


def checkpoints(stream, freq, rows, columns, shape, nr, nc, stride, main=None):
    """(states, offsets, symbols) of one stream, under the name and argument order of the reference's helper
    (bitexact_context_gpu.py:51-63)."""
    return _walk_stream(stream, freq, rows, columns, tuple(shape), nr, nc, stride, main)


def index_frame(frame: bytes, stride: int = 1024, *, keep_words: bool = False):
    """Host index of a frame: labels, tables, streams and their restart points; the walk is bound to the
    frame's source digest.  ``keep_words`` also returns the decoded words (key ``words``)."""
    if not isinstance(stride, int) or not 1 <= stride <= 65536:
        raise base.CodecError("invalid checkpoint stride")
    if len(frame) < base.HEADER.size + 32:
        raise base.CodecError("invalid frame checksum/length")
    frame = bytes(frame)
    seal = hashlib.sha256(memoryview(frame)[:-32])
    if seal.digest() != frame[-32:]:
        raise base.CodecError("invalid frame checksum/length")
    f = base.parse_sealed(frame)
    seal.update(frame[-32:])
    r, c = f["shape"]
    n = r * c
    out = {"shape": (r, c), "mode": f["mode"], "nr": f["nr"], "nc": f["nc"], "stride": stride,
           "source_sha256": f["digest"].hex(), "frame_sha256": seal.hexdigest(), "frame_bytes": len(frame)}
    if f["mode"] == 1:
        out["raw"] = f["raw"]
        if keep_words:
            out["words"] = f["raw"].reshape(r, c)
        return out
    nr, nc = f["nr"], f["nc"]
    sf = np.frombuffer(f["main_table"], dtype="<u4").copy().reshape(nr * nc, 1024)
    rf = np.frombuffer(f["residual_table"], dtype="<u4").copy().reshape(1024, 64) if f["mode"] == 128 else None
    try:
        quick = base.frame_words(f, stride)
    except base.CodecError as exc:
        raise base.CodecError("indexed source checksum mismatch") from exc
    if quick is not None:
        words, marks = quick
    else:   # something is wrong with a stream or its tables, or they are unusual: one stream after the other
        marks = {}
        marks["main_states"], marks["main_offsets"], main = checkpoints(f["main_stream"], sf, f["rows"], f["columns"], (r, c), nr, nc, stride)
        if rf is not None:
            marks["residual_states"], marks["residual_offsets"], residual = checkpoints(f["residual_stream"], rf, f["rows"], f["columns"], (r, c),
                                                                                       nr, nc, stride, main)
        else:
            residual = base._unpack6(_native.lib(), f["residual_stream"], n)
        words = base.join_words(main, residual)
        if hashlib.sha256(words.tobytes()).digest() != f["digest"]:
            raise base.CodecError("indexed source checksum mismatch")
    out.update(rows=f["rows"], columns=f["columns"], main_freq=sf, main_stream=np.frombuffer(f["main_stream"], dtype=np.uint8).copy(),
               residual_stream=np.frombuffer(f["residual_stream"], dtype=np.uint8).copy(), **marks)
    if rf is not None:
        out["residual_freq"] = rf
    if keep_words:
        out["words"] = words.reshape(r, c)
    return out


WALK_STRIDE = 128     # words per lane of the device walk when the caller's stride allows it (see CudaContextTensor)


def _lookup_tables(freq):
    """Prefix sums and the inverse index of every context, the index thinned out so that all contexts' tables together
    stay around 128 KB (they are read once per symbol on the decoder's serial chain: they have to live in L1).
    Returns (cum, bucket, log2 of the slots per bucket)."""
    nctx, vocab = freq.shape
    cum = np.empty((nctx, vocab + 1), dtype=np.uint32)
    bucket = np.empty((nctx, 4096), dtype=np.uint16)
    f = np.ascontiguousarray(freq, dtype="<u4")
    status = _native.lib().grb_bctx_build_lookup(_p(f, ctypes.c_uint32), nctx, vocab, _p(cum, ctypes.c_uint32),
                                                 _p(bucket, ctypes.c_uint16))
    if status:
        raise base.CodecError(f"invalid frequency tables ({status})")
    shift = 4
    while shift < 8 and nctx * (65536 >> shift) * 2 > 128 * 1024:
        shift += 1
    return cum, np.ascontiguousarray(bucket[:, ::1 << (shift - 4)]), shift


def _class_shares(row_class, per_row, ctas):
    """Rows sorted by class and the share of the tensor each CTA decodes (``grb_bctx_packed.part_of``): every class gets CTAs in
    proportion to its rows, and its blocks are split evenly over them, in whole warps."""
    rows_by_class = np.argsort(row_class, kind="stable").astype(np.uint32)
    counts = np.bincount(row_class)
    used = np.flatnonzero(counts)
    blocks = counts[used].astype(np.int64) * per_row
    given = np.ones(len(used), dtype=np.int64)
    most = max(1, int(-(-blocks.sum() // 128)))        # a CTA brings its tables in first: four warps of lanes at least
    for _ in range(min(ctas, most) - len(used)):
        given[np.argmax(blocks / given)] += 1
    parts, first_row = [], np.concatenate([[0], np.cumsum(counts)])
    for cls, n, g in zip(used, blocks, given):
        share = (-(-int(n) // int(g)) + 31) // 32 * 32
        parts += [(cls, first_row[cls], lo, min(int(n), lo + share)) for lo in range(0, int(n), share)]
    return rows_by_class, np.array(parts, dtype=np.uint32)


def _packed_tables(indexed, stride):
    """A frame's models packed for the shared memory of one SM: (descriptor, image, whether CTAs keep one row class's tables),
    or None when the frame is one the packed kernel does not take (see ``grb_bctx_decode_packed``)."""
    cols, nc = indexed["shape"][1], indexed["nc"]
    if stride % 16 or not 16 <= cols <= 24576:
        return None
    main = np.ascontiguousarray(indexed["main_freq"], dtype="<u4")
    residual, coded = _native.U32P(), "residual_freq" in indexed
    if coded:
        residual_freq = np.ascontiguousarray(indexed["residual_freq"], dtype="<u4")
        residual = _p(residual_freq, ctypes.c_uint32)
    packed, pack = _native.BctxPacked(), _native.lib().grb_bctx_pack_tables
    by_class = cols % stride == 0
    # What shared memory leaves beside the column classes and the stream rings: those of 928 lanes (a 4096 x 4096 frame on all
    # SMs in one round), else, for tables that take more, of half of them.
    for lanes in (928, 464):
        limit = 232448 - 128 - lanes * (128 if coded else 64) - (cols + cols // 8 + 64)
        args = (_p(main, ctypes.c_uint32), main.shape[0], residual, nc if by_class else main.shape[0], limit, ctypes.byref(packed.shape))
        status = pack(*args, None)
        if status != 4:
            break
    if status == 4:
        return None
    if not status:
        image = np.empty(packed.shape[4], dtype=np.uint8)
        status = pack(*args, _p(image, ctypes.c_uint8))
    if status:
        raise base.CodecError(f"invalid frequency tables ({status})")
    return packed, image, by_class


class _Outcome:
    """Where the kernel writes how a checked decode went: two words of pinned host memory, {status bits, an index was out of
    range}.  One call has it to itself from the launch until it has read it.  The places of all tensors come from one
    block (a pinned allocation costs milliseconds): as many as calls are under way at a time, 512 per block."""

    free = []

    def __init__(self, block, at):
        self._block, self.at = block, at
        self.words = (ctypes.c_uint32 * 2).from_address(at)

    @classmethod
    def take(cls):
        try:
            return cls.free.pop()
        except IndexError:
            import torch

            block = torch.zeros(512, 2, dtype=torch.int32).pin_memory()
            first, *others = (cls(block, block.data_ptr() + 8 * i) for i in range(512))
            cls.free.extend(others)
            return first


class CudaContextTensor:
    """A BCTX frame resident on one GPU: the unchanged streams with their restart index (for ``decode`` and
    ``gather_rows``) and, for rank-2 weights, the resident image the fused linear streams.

    ``resident_bytes`` counts every device allocation made here, the image and its scratch included.
    ``stride`` is the restart stride the caller asks for, as in the reference; the index that is actually built and
    walked on the device may be finer (``walk_stride``, by default 128 words when that divides ``stride``): a lane's walk
    is a serial chain, so the decode time is proportional to the words per lane, and eight times more lanes cost 8 bytes
    per stream and 128 words of extra index (a 4096 x 4096 frame decodes in 0.09 ms instead of 0.19 ms).  Results do not
    depend on it.  ``fused=False`` skips the image (embedding tables that are only gathered); ``layout`` picks the image's layout
    ("window4": fixed 4-bit exponent codes, the default and the fastest; "window": 3-bit codes; "rans": entropy-coded
    exponent streams, the smallest).
    """

    def __init__(self, frame: bytes, *, stride: int = 1024, device="cuda:0", fused: bool = True, max_m: int = 128,
                 layout: str | None = None, walk_stride: int | None = None):
        import torch

        if not torch.cuda.is_available():
            raise RuntimeError("CUDA is required")
        self.device = torch.device(device)
        if self.device.index is None:
            self.device = torch.device(self.device.type, torch.cuda.current_device())
        self.stride = stride
        if not isinstance(stride, int) or not 1 <= stride <= 65536:
            raise base.CodecError("invalid checkpoint stride")
        if walk_stride is None:
            walk_stride = WALK_STRIDE if stride > WALK_STRIDE and stride % WALK_STRIDE == 0 else stride
        elif not isinstance(walk_stride, int) or walk_stride <= 0 or stride % walk_stride:
            raise ValueError("walk_stride must divide stride")
        self.walk_stride = walk_stride
        indexed = index_frame(frame, walk_stride, keep_words=fused)
        words = indexed.pop("words", None)
        # identity and geometry, as the loader checks them (bitexact_context_serving.py:560-569)
        for name in ("shape", "mode", "nr", "nc", "source_sha256", "frame_sha256", "frame_bytes"):
            setattr(self, name, indexed[name])
        self.n = math.prod(self.shape)
        # every array of the index goes to the device under its own name; coded streams get their lookup tables
        self.buffers = {name: torch.from_numpy(array).to(self.device) for name, array in indexed.items() if isinstance(array, np.ndarray)}
        self._bucket_shift = {}
        self._packed = None
        if self.mode != 1 and (packed := _packed_tables(indexed, walk_stride)) is not None:
            self._packed, image, by_class = packed
            self.buffers["packed"] = torch.from_numpy(image).to(self.device)
            self._packed.tables = self.buffers["packed"].data_ptr()
            if by_class:
                rows_by_class, parts = _class_shares(indexed["rows"], self.shape[1] // walk_stride, sm_count(self.device))
                self.buffers["rows_by_class"] = torch.from_numpy(rows_by_class.view(np.int32)).to(self.device)
                self.buffers["part_of"] = torch.from_numpy(parts.view(np.int32)).to(self.device)
                self._packed.parts, self._packed.share = len(parts), int((parts[:, 3] - parts[:, 2]).max())
                self._packed.rows_by_class, self._packed.part_of = self.buffers["rows_by_class"].data_ptr(), self.buffers["part_of"].data_ptr()
        if self._packed is not None:
            self._gather_limit = self._packed_gather_limit(by_class)
        # bctx_decode_kernel's tables: for frames without packed ones, and for gathers that it does better and that are not yet
        # a whole decode
        looked_up = self._packed is None or (by_class and self._gather_limit < self.shape[0])
        for kind in ("main", "residual"):
            table = indexed.get(kind + "_freq")
            if table is not None and looked_up:
                cum, bucket, shift = _lookup_tables(table)
                self.buffers[kind + "_cum"] = torch.from_numpy(cum).to(self.device)
                self.buffers[kind + "_bucket"] = torch.from_numpy(bucket).to(self.device)
                self._bucket_shift[kind] = shift
        self.error = torch.zeros((), device=self.device, dtype=torch.int32)
        self._error_clear, self._captured = True, False     # is the word known to be zero; may a graph's replay write it
        _Outcome.free.append(_Outcome.take())      # (the first block is allocated here and not by the first call)
        self.resident = None
        if fused and words is not None:
            self.resident = ResidentWeight.from_words(words, device=self.device, source_sha256=bytes.fromhex(self.source_sha256),
                                                      max_m=max_m, **({} if layout is None else {"layout": layout}))
        self.resident_bytes = sum(t.numel() * t.element_size() for t in self.buffers.values()) + self.error.element_size()
        if self.resident is not None:
            self.resident_bytes += self.resident.resident_bytes
        self._descriptor = None if self.mode == 1 else self._make_descriptor()
        if self._packed is not None:
            self._packed_args = ctypes.byref(self._descriptor), ctypes.byref(self._packed)

    def _packed_gather_limit(self, by_class) -> int:
        """How many rows ``gather_rows`` takes through the packed kernel at most.

        By class a CTA brings in its class's tables for every single row, 23 to 35 us per wave of CTAs, while
        ``bctx_decode_kernel`` takes any number of rows at once in 200 to 400 us; they meet between 10 waves (9504 x 5120 words
        with coded residuals, 2048 rows: 485 against 390 us) and 30 (2048 x 5120, raw residuals).  As many rows as the tensor
        has are one decode and an index (32768 rows of a 9504 x 5120 table: 430 us; by class 7100 us).  With the tables of all classes in
        every CTA a row costs what its words cost, and the tensor is decoded and indexed when that saves more words than
        the extra pass and the check of the row numbers cost (60 us, 24 M words; 32768 rows of 2048 x 5000: 499 -> 234 us)."""
        rows, cols = self.shape
        if not by_class:
            return rows + (24 << 20) // cols
        coded, shape, per_row = self.mode == 128, self._packed.shape, cols // self.walk_stride
        lanes = min(1024, -(-per_row // 32) * 32)
        memory = 128 + self.nc * shape[1] + shape[4] - shape[3] + cols + cols // 8 + 32 + lanes * (128 if coded else 64)
        per_sm = max(1, min((228 << 10) // (memory + 1024), 1024 // lanes))      # (64 registers a thread)
        return 10 * per_sm * sm_count(self.device)

    def _make_descriptor(self):
        b = self.buffers
        t = _native.BctxTensor()
        t.n, t.rows, t.cols = self.n, self.shape[0], self.shape[1]
        t.nr, t.nc, t.mode, t.stride = self.nr, self.nc, self.mode, self.walk_stride
        t.row_class, t.col_class = b["rows"].data_ptr(), b["columns"].data_ptr()
        t.main_stream, t.main_bytes = b["main_stream"].data_ptr(), b["main_stream"].numel()
        t.main_states, t.main_offsets = b["main_states"].data_ptr(), b["main_offsets"].data_ptr()
        if "main_cum" in b:
            t.main_cum, t.main_bucket = b["main_cum"].data_ptr(), b["main_bucket"].data_ptr()
            t.main_bucket_shift = self._bucket_shift["main"]
        t.residual_stream, t.residual_bytes = b["residual_stream"].data_ptr(), b["residual_stream"].numel()
        if self.mode == 128:
            t.residual_states, t.residual_offsets = b["residual_states"].data_ptr(), b["residual_offsets"].data_ptr()
            if "residual_cum" in b:
                t.residual_cum, t.residual_bucket = b["residual_cum"].data_ptr(), b["residual_bucket"].data_ptr()
                t.residual_bucket_shift = self._bucket_shift["residual"]
        return t

    def _decode_packed(self, ids=None, *, check):
        """All blocks, or the rows ``ids``, through the packed tables.  The host waits when ``check`` asks for the outcome or
        ``ids`` have to be known to be rows of the tensor."""
        import torch

        if ids is None:
            count = -(-self.n // self.walk_stride)
            result = torch.empty(count * self.walk_stride, device=self.device, dtype=torch.bfloat16)
        else:
            count = ids.numel()
            result = torch.empty((*ids.shape, self.shape[1]), device=self.device, dtype=torch.bfloat16)
        wait = check or ids is not None
        # A call that waits for its launch leaves the word as it found it, at zero, and need not clear it for the next one
        # that waits.  All others clear it on the stream, where a captured graph does so on every replay.
        if not (wait and self._error_clear):
            self.error.zero_()
        if not wait and torch.cuda.is_current_stream_capturing():
            self._captured = True
        self._error_clear = wait and not self._captured
        outcome = None
        if wait:
            outcome = _Outcome.take()
            outcome.words[0] = outcome.words[1] = 0
        stream = torch.cuda.current_stream(self.device)
        args = (*self._packed_args, None if ids is None else ids.data_ptr(), count, result.data_ptr(), self.error.data_ptr(),
                outcome.at if wait else None, stream.cuda_stream)
        if torch.cuda.current_device() == self.device.index:
            status = _native.lib().grb_bctx_decode_packed(*args)
        else:
            with torch.cuda.device(self.device):
                status = _native.lib().grb_bctx_decode_packed(*args)
        if status:
            _native.check(status, "grb_bctx_decode_packed")
        if wait:
            stream.synchronize()
            failed, outside = outcome.words[0], outcome.words[1]
            _Outcome.free.append(outcome)
            if failed or outside:
                self._error_clear = False
                if outside:
                    raise IndexError("embedding row outside tensor")
                if check:
                    raise base.CodecError("CUDA decoder checkpoint mismatch")
        return result

    def _decode_blocks(self, blocks=None, *, check=True):
        import torch

        walk = self.walk_stride                      # blocks are counted in the stride the index was built with
        if blocks is None:
            count, ids = (self.n + walk - 1) // walk, None
        else:
            blocks = blocks.to(device=self.device, dtype=torch.int64).contiguous().reshape(-1)
            count, ids = blocks.numel(), blocks.data_ptr()
        result = torch.empty(count * walk, device=self.device, dtype=torch.uint16)
        self.error.zero_()
        self._error_clear = False
        with torch.cuda.device(self.device):
            stream = torch.cuda.current_stream().cuda_stream
            status = _native.lib().grb_bctx_decode_words(ctypes.byref(self._descriptor), ids, count, result.data_ptr(),
                                                         self.error.data_ptr(), stream)
        _native.check(status, "grb_bctx_decode_words")
        if check and self.error.item() != 0:
            raise base.CodecError("CUDA decoder checkpoint mismatch")
        return result.view(torch.bfloat16)

    def decode(self, *, check=True):
        """Dense BF16 [rows, cols], decoded from the unchanged streams (transient: the caller owns it)."""
        import torch

        if self.mode == 1:
            return self.buffers["raw"].view(torch.bfloat16).reshape(self.shape)
        if self._packed is not None:
            return self._decode_packed(check=check)[:self.n].reshape(self.shape)
        return self._decode_blocks(check=check)[:self.n].reshape(self.shape)

    def gather_rows(self, ids, *, check=True):
        """Rows ``ids`` (any shape) as BF16 [..., cols].  Only the blocks of the requested rows are decoded when the frame has
        packed tables or a row is a whole number of restart blocks; otherwise (raw frames, strides that do not divide the
        row), and when more rows are asked for than that is worth, the tensor is decoded once and indexed."""
        import torch

        rows, cols = self.shape
        ids = ids.to(device=self.device, dtype=torch.int64)
        if ids.numel() == 0:
            return torch.empty((*ids.shape, cols), device=self.device, dtype=torch.bfloat16)
        if self._packed is not None and ids.numel() <= self._gather_limit:
            return self._decode_packed(ids.contiguous(), check=check)
        lowest, highest = torch.aminmax(ids)
        if int(lowest) < 0 or int(highest) >= rows:
            raise IndexError("embedding row outside tensor")
        blocks_per_row, ragged = divmod(cols, self.walk_stride)
        if self.mode == 1 or ragged or (self._packed is not None and ids.numel() >= rows):
            return self.decode(check=check)[ids]
        first_block = ids.reshape(-1, 1) * blocks_per_row
        wanted = (first_block + torch.arange(blocks_per_row, device=self.device)).reshape(-1)
        return self._decode_blocks(wanted, check=check).reshape(*ids.shape, cols)

    # -- fused linear --------------------------------------------------------------------------------
    def linear(self, x, out=None, bias=None):
        """y = x @ W.T (+ bias) with W decoded inside the kernel; x [..., cols] BF16 -> y [..., rows] BF16."""
        if self.resident is None:
            raise RuntimeError("this tensor was indexed without a resident image (fused=False)")
        return self.resident.linear(x, out=out, bias=bias)

    def __call__(self, x, y):
        self.resident(x, y)
