"""Device-resident copy table: built once per registered batch, launched once per transfer.

`CopyTable.add*` collect strided-box copies (optionally converting, fanning out to several
destinations or collapsing several Partial sources); `finalize()` packs them with the native packer,
splits them by the kernel that runs them and uploads them in one copy; `launch()` issues one kernel per group on
the given stream in one native call and, when asked, publishes an epoch to the consumers' flags after the
last tile.  Nothing here allocates or touches the host during `launch()`.

The reference does this work per chunk and per transfer in Python (`Chunk.prepare`/`Bucket.prepare`/
`finalize`, src/etha/comm/ir.py:101-141,229-310).
"""

from __future__ import annotations

import ctypes as C
from dataclasses import dataclass
from typing import Sequence

import numpy as np
import torch

from . import lib as L

_DT_CODE = {torch.float32: L.DT_F32, torch.bfloat16: L.DT_BF16, torch.float16: L.DT_F16}

DEFAULT_TILE_BYTES = 64 * 1024

# kernels launched by CopyTable.launch in this process (benchmarks report it)
LAUNCH_COUNT = [0]
# copy-engine copies enqueued by CopyTable.launch in this process (not kernels; reported separately)
DMA_COPY_COUNT = [0]


def raw_stream(stream: torch.cuda.Stream | None, device: torch.device) -> int:
    """Handle of `stream`, or of the device's current stream (read without building a Stream object)."""
    if stream is not None:
        return stream.cuda_stream
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if device.index is None else device.index)


def device_index(device: torch.device) -> int:
    """What the launching entries of the library take: -1 stands for whatever device is current."""
    return -1 if device.index is None else device.index


def dtype_code(dt: torch.dtype) -> int:
    return _DT_CODE.get(dt, L.DT_RAW)


@dataclass
class SliceRef:
    """A strided box in some GPU's memory: address of element [0,...,0], element strides, allocation bounds."""

    ptr: int
    strides: tuple[int, ...]
    dtype: torch.dtype
    lo: int = 0  # allocation [lo, hi) the box must stay inside (0, 0 = unchecked)
    hi: int = 0

    @staticmethod
    def of(view: torch.Tensor) -> "SliceRef":
        st = view.untyped_storage()
        base = st.data_ptr()
        return SliceRef(view.data_ptr(), tuple(view.stride()), view.dtype, base, base + st.nbytes())


def make_spec(shape, srcs, dsts, reduce_sizes, reduce_ops, flags: int, tile_bytes: int) -> L.OpSpec:
    """Native description of one op; the slices of either side share strides and dtype."""
    spec = L.OpSpec()
    src0, dst0 = srcs[0], dsts[0]
    n = spec.ndim = len(shape)
    spec.shape[:n], spec.src_stride[:n], spec.dst_stride[:n] = shape, src0.strides[:n], dst0.strides[:n]
    spec.src_itemsize, spec.dst_itemsize = src0.dtype.itemsize, dst0.dtype.itemsize
    spec.src_dtype, spec.dst_dtype = dtype_code(src0.dtype), dtype_code(dst0.dtype)
    if spec.src_dtype == L.DT_RAW and spec.dst_dtype == L.DT_RAW and src0.dtype != dst0.dtype:
        raise ValueError(f"no conversion from {src0.dtype} to {dst0.dtype}")
    spec.nsrc, spec.ndst = len(srcs), len(dsts)
    for i, s in enumerate(srcs):
        spec.src[i], spec.src_lo[i], spec.src_hi[i] = s.ptr, s.lo, s.hi
    for i, d in enumerate(dsts):
        spec.dst[i], spec.dst_lo[i], spec.dst_hi[i] = d.ptr, d.lo, d.hi
    sizes = list(reduce_sizes) or [len(srcs)]
    ops = list(reduce_ops) or ["sum"]
    spec.red_size[0], spec.red_size[1] = sizes[0], (sizes[1] if len(sizes) > 1 else 1)
    spec.red_op[0] = L.RED_CODES[ops[0]]
    spec.red_op[1] = L.RED_CODES[ops[1]] if len(ops) > 1 else 0
    spec.flags, spec.tile_bytes = flags, tile_bytes
    return spec


class _KernelSet:
    """Launches that run one set of ops, without and with the TMA kernel.  Until the table is uploaded their addresses are
    offsets into its buffer."""

    def __init__(self):
        self.n_ops, self.n_tiles = [0, 0], [0, 0]  # [fast class, general class]
        self.n_typed_ops = self.n_typed_tiles = 0
        self.n_bulk_ops = self.n_bulk_tiles = 0
        self.ldst: list[L.Launch] = []
        self.bulk: list[L.Launch] = []

    def at(self, base: int) -> None:
        """Make the launch lists what the native runner takes: (array of launches, its address, its length)."""
        for name in ("ldst", "bulk"):
            launches = (L.Launch * len(getattr(self, name)))(*getattr(self, name))
            for one in launches:
                one.ops += base
                one.tiles += base
            setattr(self, name, (launches, C.addressof(launches), len(launches)))


class _Blob:
    """Host image of everything a table keeps on the device, uploaded in one copy."""

    def __init__(self):
        self.parts: list[tuple[int, np.ndarray]] = []
        self.size = 0

    def add(self, array: np.ndarray) -> int:
        offset = (self.size + 15) // 16 * 16
        self.parts.append((offset, array))
        self.size = offset + array.nbytes
        return offset

    def upload(self, device) -> torch.Tensor:
        image = np.zeros(self.size, dtype=np.uint8)
        for offset, array in self.parts:
            image[offset : offset + array.nbytes] = array.view(np.uint8)
        return torch.from_numpy(image).to(device)


class CopyTable:
    """`tile_bytes`: upper bound of a tile (destination bytes); the TMA kernel uses it as it is, the others cut finer.

    `dma_min_bytes`: when set, a bit copy of at least that many bytes whose box is one run or the rows of a matrix,
    and which the caller marks `dma_ok` (its destination is on another GPU), is a candidate for the DMA engines: at
    `finalize()` the largest candidates, up to `dma_fraction` of the bytes the table delivers, become memcpy nodes
    of a CUDA graph (`dma_mode="graph"`) or asynchronous copies on `dma_streams` side streams
    (`dma_mode="streams"`); everything else is packed for the kernels.  At launch the copies run next to the
    kernels: the DMA engines write larger NVLink packets than SM stores can, and the kernels fill the gaps
    between consecutive DMA copies."""

    def __init__(self, device: torch.device | int | str, tile_bytes: int = DEFAULT_TILE_BYTES,
                 dma_min_bytes: int | None = None, dma_mode: str = "graph", dma_streams: int = 8,
                 dma_fraction: float = 1.0):
        self.device = torch.device(device) if not isinstance(device, torch.device) else device
        self.tile_bytes = int(tile_bytes)
        self.dma_min_bytes = dma_min_bytes
        self.dma_mode, self.dma_streams, self.dma_fraction = dma_mode, dma_streams, dma_fraction
        self._dma: list[L.DmaCopy] = []
        self._dma_candidates: list[tuple[int, int, list, tuple]] = []  # (bytes, position, copies, packed entry)
        self._dma_plan = None
        self.dma_bytes = 0
        self._lib = L.cuda_lib()
        self._run = self._lib.etha_run
        self._op_size = self._lib.etha_sizeof_op()
        self._packed: list[tuple[int, int, bytes, bool, int]] = []  # (class, tiles, op bytes, TMA-capable, instance key)
        # conversions / collapses over simple boxes use the streaming kernel instances, rows of any alignment the ragged ones
        self.stream_typed = True
        self.payload_bytes = 0  # bytes delivered (destination side, all replicas)
        self.read_bytes = 0
        self._final = False
        self._keepalive: list = []
        self.n_ops = [0, 0]
        self.n_tiles = [0, 0]
        # fast-class ops are kept in two groups: those the TMA kernel can run (uploaded first) and the rest
        self.n_bulk_ops = 0
        self.n_bulk_tiles = 0

    # ---- building ---------------------------------------------------------------------------
    def add(
        self,
        shape: Sequence[int],
        srcs: Sequence[SliceRef],
        dsts: Sequence[SliceRef],
        reduce_sizes: Sequence[int] = (),
        reduce_ops: Sequence[str] = (),
        multimem: bool = False,
        dma_ok: bool = False,
    ) -> None:
        """One op: `srcs` (1, or a Partial family in family order) -> every slice of `dsts`."""
        if self._final:
            raise RuntimeError("table already finalized")
        if len(shape) > 8:
            raise ValueError("at most 8 dims")
        if len(srcs) > L.MAX_SRC:
            raise ValueError(f"at most {L.MAX_SRC} Partial contributors per cell are supported on the device")
        if len(reduce_sizes) > 2:
            raise ValueError("at most two Partial mesh dims are supported on the device")
        src0 = srcs[0]
        for s in srcs[1:]:
            if s.strides != src0.strides or s.dtype != src0.dtype:
                raise ValueError("Partial contributors must share strides and dtype")
        # group destinations by (strides, dtype): one op per group of at most MAX_DST
        groups: dict[tuple, list[SliceRef]] = {}
        for d in dsts:
            groups.setdefault((d.strides, d.dtype), []).append(d)
        numel = int(np.prod(shape)) if len(shape) else 1
        for (dstrides, ddtype), members in groups.items():
            for k in range(0, len(members), L.MAX_DST):
                part = members[k : k + L.MAX_DST]
                spec = make_spec(shape, srcs, part, reduce_sizes, reduce_ops, L.FLAG_MULTIMEM if multimem else 0, self.tile_bytes)
                buf = C.create_string_buffer(self._op_size)
                err = C.create_string_buffer(512)
                rc = self._lib.etha_pack_op(C.byref(spec), buf, err, 512)
                if rc != 0:
                    raise ValueError(f"cannot pack op ({rc}): {err.value.decode(errors='replace')}")
                tiles = self._lib.etha_op_tiles(buf)
                if tiles:
                    cls = self._lib.etha_op_class(buf)
                    tma = cls == 0 and bool(self._lib.etha_op_bulk_ok(buf))
                    skey = 0  # key of the kernel instance, 0: general kernel
                    if cls == 1 and self.stream_typed:
                        skey = self._lib.etha_op_kernel_key(buf)
                        skey = 0 if skey == L.KEY_GENERAL else skey
                    entry = (cls, tiles, buf.raw, tma, skey)
                    self._packed.append(entry)
                    if dma_ok and self.dma_min_bytes is not None and numel * ddtype.itemsize >= self.dma_min_bytes:
                        out = (L.DmaCopy * L.MAX_DST)()
                        n = self._lib.etha_op_dma_copies(buf, out)
                        if n > 0:
                            copies = []
                            for j in range(n):
                                c = L.DmaCopy()
                                C.memmove(C.byref(c), C.byref(out[j]), C.sizeof(L.DmaCopy))
                                copies.append(c)
                            self._dma_candidates.append((numel * ddtype.itemsize * n, len(self._packed) - 1, copies, entry))
                self.payload_bytes += numel * ddtype.itemsize * len(part)
        self.read_bytes += numel * src0.dtype.itemsize * len(srcs)

    def add_copy(self, src: torch.Tensor, dst: torch.Tensor) -> None:
        """Local convenience: copy (and convert) `src` view into `dst` view of the same shape."""
        if tuple(src.shape) != tuple(dst.shape):
            raise ValueError(f"shape mismatch {tuple(src.shape)} vs {tuple(dst.shape)}")
        self._keepalive += [src, dst]
        self.add(tuple(src.shape), [SliceRef.of(src)], [SliceRef.of(dst)])

    def add_reduce(self, srcs: Sequence[torch.Tensor], dst: torch.Tensor, sizes: Sequence[int], ops: Sequence[str]) -> None:
        self._keepalive += list(srcs) + [dst]
        self.add(tuple(dst.shape), [SliceRef.of(s) for s in srcs], [SliceRef.of(dst)], sizes, ops)

    # ---- upload -----------------------------------------------------------------------------
    def _lay_out(self, packed, blob: _Blob) -> "_KernelSet":
        """Put one set of packed ops into `blob`, split into the launches of the kernel classes."""
        ks = _KernelSet()
        device = device_index(self.device)

        def launch(key, members):
            """One launch: tile sizes chosen for its kernel."""
            ops_host = np.frombuffer(b"".join(members), dtype=np.uint8).copy()
            starts = np.zeros(len(members) + 1, dtype=np.uint32)
            tiles = self._lib.etha_layout_tiles(ops_host.ctypes.data, len(members), self._lib.etha_key_tile_class(key),
                                                starts.ctypes.data)
            if tiles < 0:
                raise ValueError("too many tiles in one table")
            return L.Launch(key, len(members), tiles, device, blob.add(ops_host), blob.add(starts))

        rest = []  # launches of the typed and general classes
        for key in dict.fromkeys(k for c, _, _, _, k in packed if c == 1 and k):
            one = launch(key, [raw for c, _, raw, _, k in packed if c == 1 and k == key])
            rest.append(one)
            if key < L.KEY_RAGGED:
                ks.n_typed_ops += one.n_ops
                ks.n_typed_tiles += one.n_tiles
            else:
                ks.n_ops[1] += one.n_ops
                ks.n_tiles[1] += one.n_tiles
        general = [raw for c, _, raw, _, k in packed if c == 1 and not k]
        if general:
            rest.append(launch(L.KEY_GENERAL, general))
            ks.n_ops[1] += rest[-1].n_ops
            ks.n_tiles[1] += rest[-1].n_tiles
        fast = [(t, raw, tma) for c, t, raw, tma, _ in packed if c == 0]
        if fast:
            # stable split: TMA-capable ops first, relative order kept inside both groups
            tma, other = [m for m in fast if m[2]], [m for m in fast if not m[2]]
            ks.ldst.append(launch(L.KEY_FAST, [raw for _, raw, _ in tma + other]))
            ks.n_ops[0], ks.n_tiles[0] = ks.ldst[0].n_ops, ks.ldst[0].n_tiles
            if tma:
                # the TMA kernel cuts its tiles into ring stages and keeps the table's tile size
                starts = np.zeros(len(tma) + 1, dtype=np.uint64)
                np.cumsum([t for t, _, _ in tma], out=starts[1:])
                if starts[-1] >= 2**31:
                    raise ValueError("too many tiles in one table")
                ks.n_bulk_ops, ks.n_bulk_tiles = len(tma), int(starts[-1])
                ops_at = blob.add(np.frombuffer(b"".join(raw for _, raw, _ in tma), dtype=np.uint8))
                ks.bulk.append(L.Launch(L.KEY_BULK, len(tma), ks.n_bulk_tiles, device, ops_at, blob.add(starts.astype(np.uint32))))
                if other:
                    ks.bulk.append(launch(L.KEY_FAST, [raw for _, raw, _ in other]))
            else:
                ks.bulk = list(ks.ldst)
        ks.ldst += rest
        ks.bulk += rest
        return ks

    def _select_dma(self) -> set[int]:
        """Positions (in `_packed`) of the ops handed to the DMA engines: the largest candidates first, as long as the
        byte budget `dma_fraction x delivered bytes` is not exceeded (a candidate that does not fit is skipped, smaller
        ones may still fit).  Their copies are queued in table order, so the producers' rotation is kept."""
        budget = self.dma_fraction * self.payload_bytes
        taken: set[int] = set()
        for nbytes, pos, _copies, _ in sorted(self._dma_candidates, key=lambda c: (-c[0], c[1])):
            if self.dma_bytes + nbytes > budget:
                continue
            taken.add(pos)
            self.dma_bytes += nbytes
        for _nbytes, pos, copies, _ in self._dma_candidates:
            if pos in taken:
                self._dma += copies
        return taken

    def finalize(self, sm_count: int | None = None) -> "CopyTable":
        """Lay the table out and upload it.  `sm_count` is kept as an attribute; grids do not depend on it."""
        if self._final:
            return self
        if self.device.type == "cuda" and self.device.index is None:  # the table lives on one device from here on
            self.device = torch.device("cuda", torch.cuda.current_device())
        if sm_count is None:
            sm_count = torch.cuda.get_device_properties(self.device).multi_processor_count
        self.sm_count = sm_count
        taken = self._select_dma()
        blob = _Blob()
        blob.add(np.zeros(4, dtype=np.uint32))  # finished tiles and error word of the launches
        # two kernel sets share this table: every op (kernels only), and what is left next to the DMA copies
        self._all = self._lay_out(self._packed, blob)
        self._rest = self._lay_out([e for i, e in enumerate(self._packed) if i not in taken], blob) if taken else self._all
        self._buffer = blob.upload(self.device)
        self._sync = self._buffer[:16].view(torch.int32)
        self._sync_ptr = self._buffer.data_ptr()
        for ks in {id(k): k for k in (self._all, self._rest)}.values():
            ks.at(self._buffer.data_ptr())
        # [fast class, typed + general]: the streaming instances count with the general class they were taken from
        self.n_ops = [self._all.n_ops[0], self._all.n_ops[1] + self._all.n_typed_ops]
        self.n_tiles = [self._all.n_tiles[0], self._all.n_tiles[1] + self._all.n_typed_tiles]
        self.n_typed_ops = self._all.n_typed_ops
        self.n_bulk_ops, self.n_bulk_tiles = self._all.n_bulk_ops, self._all.n_bulk_tiles
        self._dma_candidates = []
        self._packed = []
        if self._dma:
            arr = (L.DmaCopy * len(self._dma))(*self._dma)
            plan = C.c_void_p()
            with torch.cuda.device(self.device):
                L.check(self._lib.etha_dma_plan_create(arr, len(self._dma), 1 if self.dma_mode == "graph" else 0,
                                                       self.dma_streams, C.byref(plan)), "dma plan")
            self._dma_plan = plan
        self._final = True
        return self

    def __del__(self):
        plan, self._dma_plan = getattr(self, "_dma_plan", None), None
        if plan:
            try:
                self._lib.etha_dma_plan_destroy(plan)
            except Exception:
                pass

    @property
    def n_dma_copies(self) -> int:
        return len(self._dma)

    @property
    def empty(self) -> bool:
        return self.n_tiles[0] + self.n_tiles[1] == 0

    def device_buffers(self) -> list[torch.Tensor]:
        """The device memory a launch reads (callers that drop the table right after a launch tie it to the stream)."""
        return [self._buffer]

    # ---- launch -----------------------------------------------------------------------------
    def launch(
        self,
        stream: torch.cuda.Stream | None = None,
        signals: torch.Tensor | None = None,
        epoch: int = 0,
        ctas_per_sm: int = 2,
        bulk: bool = False,
        dma: bool | None = None,
    ) -> None:
        """Enqueue the table on `stream`. `signals`: int64 device tensor of flag addresses to publish `epoch` to.
        Launches without signals may overlap on several streams; those with signals share the table's count of
        finished tiles and must follow one another.
        `ctas_per_sm`: 1 leaves half of every SM to other work while the 16-byte copy kernel runs; any other number
        lets it fill the SMs, and the other kernels always do.
        `bulk`: TMA ring kernel instead of the LD/ST kernel for the 16-byte bit copies; `dma=False`: every copy by
        the kernels even if the table holds a DMA plan."""
        if not self._final:
            self.finalize()
        s = raw_stream(stream, self.device)
        sig_ptr, n_sig = (0, 0) if signals is None else (signals.data_ptr(), signals.numel())
        dma = self._dma_plan is not None and dma is not False
        ks = self._rest if dma else self._all
        _, launches, n = ks.bulk if bulk else ks.ldst
        epoch &= 0xFFFFFFFF
        if n and not dma:
            rc = self._run(launches, n, self._sync_ptr, sig_ptr, n_sig, epoch, ctas_per_sm, s)
            if rc:
                L.check(rc, "m2n launch")
            LAUNCH_COUNT[0] += n
            return
        # with DMA copies in the transfer: the copies start on side streams, the kernels run next to them on
        # the caller's stream without a signal, the stream then waits for the copies and the flags go last
        if dma:
            with torch.cuda.device(self.device):
                L.check(self._lib.etha_dma_plan_launch(self._dma_plan, s), "dma launch")
            DMA_COPY_COUNT[0] += len(self._dma)
        if n:
            L.check(self._run(launches, n, self._sync_ptr, 0, 0, epoch, ctas_per_sm, s), "m2n launch")
            LAUNCH_COUNT[0] += n
        if dma:
            with torch.cuda.device(self.device):
                L.check(self._lib.etha_dma_plan_join(self._dma_plan, s), "dma join")
        if n_sig:
            L.check(self._lib.etha_set_flags(sig_ptr, n_sig, epoch, device_index(self.device), s), "set_flags")
            LAUNCH_COUNT[0] += 1

    def error_word(self) -> int:
        """Device-side error word (synchronizes): 0, or the status bits of every failure since `finalize()`.  A table
        whose word is set publishes no epoch any more; it has to be built again."""
        return int(self._sync[1].item()) if (self.n_tiles[0] + self.n_tiles[1]) else 0
