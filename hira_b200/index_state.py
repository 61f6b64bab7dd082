"""Device-resident index arrays and thin typed wrappers over the C ABI.

`IndexState` owns the torch tensors behind one `hira_index_t` (torch only supplies
memory and the stream); the functions below forward to libhira_b200.so.  Names of
the arrays follow the reference's CUDAIndexer attributes (indexer/cuda.py:40-54).
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass
from functools import lru_cache
from typing import Optional

import torch

from . import _lib as L


def aligned(t: torch.Tensor) -> torch.Tensor:
    """`t`, or a copy of it where it does not start on a 16-byte boundary: the kernels load rows in 16-byte pieces."""
    return t if t.data_ptr() % 16 == 0 else t.clone()


class IndexState:
    def __init__(self, *, n_heads: int, dim: int, vdim: int, bf: int, depth: int, cap_parents: int,
                 dtype: torch.dtype, vdtype: Optional[torch.dtype], device, with_values: bool = True,
                 int8_copy: Optional[bool] = None, cleared: bool = True):
        """`cleared=False`: for a state that `build` fills with at least one key next -- the build writes
        every array (keys, or zeros and -1 where there are none), so nothing is cleared here first."""
        if depth not in (2, 3):
            raise ValueError(f"Unsupported depth {depth}")
        self.n_heads, self.dim, self.vdim, self.bf, self.depth = n_heads, dim, vdim if with_values else 0, bf, depth
        self.dtype, self.vdtype = dtype, (vdtype if with_values else dtype)
        self.device = torch.device(device)
        if depth == 3:
            self.cap_gp = max(1, -(-cap_parents // bf))
            self.cap_parents = self.cap_gp * bf
        else:
            self.cap_gp = 0
            self.cap_parents = max(1, cap_parents)
        capC = self.cap_parents * bf
        dev = self.device
        z = torch.zeros if cleared else torch.empty
        self.children = z((n_heads, capC, dim), dtype=dtype, device=dev)
        self.values = z((n_heads, capC, self.vdim), dtype=self.vdtype, device=dev) if with_values else None
        self.slot2token = z((n_heads, capC), dtype=torch.int32, device=dev)
        if cleared:
            self.slot2token.fill_(-1)
        self.parents = z((n_heads, self.cap_parents, dim), dtype=dtype, device=dev)
        self.parent_radii = z((n_heads, self.cap_parents), dtype=torch.float32, device=dev)
        self.parent_sqnorm = z((n_heads, self.cap_parents), dtype=torch.float32, device=dev)
        self.child_counts = z((n_heads, self.cap_parents), dtype=torch.int32, device=dev)
        if depth == 3:
            self.grand_parents = z((n_heads, self.cap_gp, dim), dtype=dtype, device=dev)
            self.gp_radii = z((n_heads, self.cap_gp), dtype=torch.float32, device=dev)
            self.gp_sqnorm = z((n_heads, self.cap_gp), dtype=torch.float32, device=dev)
            self.gp_counts = z((n_heads, self.cap_gp), dtype=torch.int32, device=dev)
        else:
            self.grand_parents = self.gp_radii = self.gp_sqnorm = self.gp_counts = None
        self.used = z((n_heads, 4), dtype=torch.int32, device=dev)
        # int8 side copy of the children for the tensor-core pre-filter of the search (D = 128):
        # +52 % on the bf16 keys' memory (128 B + 4 B per slot), about half the search's traffic
        if int8_copy is None:
            int8_copy = dim == 128 and self.device.type == "cuda"
        if int8_copy and dim != 128:
            raise ValueError("the int8 side copy needs dim == 128")
        self.int8_copy = bool(int8_copy)
        if self.int8_copy:
            self.children_q8 = z((n_heads, capC, 128), dtype=torch.int8, device=dev)
            self.children_q8_meta = z((n_heads, capC), dtype=torch.int32, device=dev)   # (step, error bound) as two fp16
            self.q8_chan_scale = z((n_heads, L.Q8_CHAN), dtype=torch.float32, device=dev)
            if cleared:
                self.q8_chan_scale.fill_(1.0)
            self.q8_query_scratch = z((n_heads, L.Q8_QUERY_BYTES), dtype=torch.uint8, device=dev)
        else:
            self.children_q8 = self.children_q8_meta = self.q8_chan_scale = self.q8_query_scratch = None
        self.status = z((1,), dtype=torch.int32, device=dev)
        self.arrays_device = self.status.device     # with its index, which `device` may lack
        self._struct = None
        self._append_bytes = {}
        self._append_ws = None, 0      # scratch of the appends, and the stream it was allocated on
        # streams the arrays are kept alive for: the one they are allocated on, and those of `used_on`
        self._streams = {L.current_stream(dev)} if dev.type == "cuda" else set()
        self._active_parents = 0
        self.refresh_struct()

    ARRAYS = ("children", "values", "slot2token", "parents", "parent_radii", "parent_sqnorm", "child_counts",
              "grand_parents", "gp_radii", "gp_sqnorm", "gp_counts", "used")
    # derived from `children` (and scratch): not part of a checkpoint
    Q8_ARRAYS = ("children_q8", "children_q8_meta", "q8_chan_scale", "q8_query_scratch")

    @property
    def cap_children(self) -> int:
        return self.cap_parents * self.bf

    def refresh_struct(self):
        s = L.HiraIndexStruct()
        s.dtype = L.dtype_code(self.dtype)
        s.vdtype = L.dtype_code(self.vdtype)
        s.depth, s.bf, s.dim, s.vdim = self.depth, self.bf, self.dim, self.vdim
        s.n_heads, s.cap_parents, s.cap_gp = self.n_heads, self.cap_parents, self.cap_gp
        s.active_parents = self._active_parents
        for name in self.ARRAYS + self.Q8_ARRAYS:
            setattr(s, name, L.ptr(getattr(self, name)))
        self._struct = s
        self._byref = C.byref(s)
        return s

    @property
    def active_parents(self) -> int:
        """Host's upper bound on the parent slots in use; 0 = unknown (all of cap_parents).
        Search, sparse attention and kth_score skip the tiles beyond it."""
        return self._active_parents

    @active_parents.setter
    def active_parents(self, n: int):
        n = int(n)
        if n < 0 or n >= self.cap_parents:
            n = 0
        if n == self._active_parents:
            return
        self._active_parents = n
        self._struct.active_parents = n

    def used_on(self, stream):
        """Keeps the memory of the arrays from being handed out again before the work enqueued on `stream` when
        they are dropped is done."""
        if stream.cuda_stream in self._streams:
            return
        self._streams.add(stream.cuda_stream)
        for name in self.ARRAYS + self.Q8_ARRAYS + ("status",):
            t = getattr(self, name)
            if t is not None:
                t.record_stream(stream)

    @property
    def struct(self):
        return self._byref

    def state_dict(self) -> dict:
        d = {name: getattr(self, name) for name in self.ARRAYS if getattr(self, name) is not None}
        d["meta"] = dict(n_heads=self.n_heads, dim=self.dim, vdim=self.vdim, bf=self.bf, depth=self.depth,
                         cap_parents=self.cap_parents, dtype=str(self.dtype), vdtype=str(self.vdtype))
        return d

    def load_arrays(self, arrays: dict):
        """Copies host/device arrays with matching shapes into the index (checkpoint import,
        moving an index between the oracle and the device)."""
        for name in self.ARRAYS:
            dst = getattr(self, name)
            if dst is None or name not in arrays or arrays[name] is None:
                continue
            src = arrays[name]
            if not torch.is_tensor(src):
                src = torch.as_tensor(src)
            if src.dtype == torch.uint16 or (dst.dtype == torch.bfloat16 and src.dtype == torch.int16):
                src = src.view(torch.bfloat16)
            dst.copy_(src.reshape(dst.shape).to(dst.dtype))
        self.used[:, 3] = 0      # the appends count in it: zero between calls
        self.refresh_int8_copy()

    def enable_int8_copy(self, on: bool = True):
        """Switches the search between the int8 pre-filter (when the index carries the side copy)
        and the plain streaming kernel; results are identical either way."""
        for name in self.Q8_ARRAYS:
            setattr(self._struct, name, L.ptr(getattr(self, name)) if (on and self.int8_copy) else None)

    def refresh_int8_copy(self):
        """Recomputes the int8 side copy from the children as stored now."""
        if self.int8_copy and self.device.type == "cuda":
            L.check(L.load().hira_q8_refresh(self.struct, L.current_stream(self.device)), "hira_q8_refresh")

    def grown(self, new_cap_parents: int) -> "IndexState":
        """A copy with more parent slots (and grandparent slots); existing slots keep their positions."""
        new = IndexState(n_heads=self.n_heads, dim=self.dim, vdim=self.vdim, bf=self.bf, depth=self.depth,
                         cap_parents=new_cap_parents, dtype=self.dtype, vdtype=self.vdtype, device=self.device,
                         with_values=self.values is not None, int8_copy=self.int8_copy, cleared=self.device.type != "cuda")
        new.status.copy_(self.status)
        if self.device.type == "cuda":
            self.used_on(torch.cuda.current_stream(self.device))     # the caller drops the old arrays right away
            old = L.HiraIndexStruct.from_buffer_copy(self._struct)
            for name in self.Q8_ARRAYS:     # also when enable_int8_copy has left them out of the view
                setattr(old, name, L.ptr(getattr(self, name)))
            L.check(L.load().hira_grow(C.byref(old), new.struct, L.current_stream(self.device)), "hira_grow")
            return new
        for name in self.ARRAYS + self.Q8_ARRAYS:
            src = getattr(self, name)
            if src is None or name == "used":
                continue
            if name in ("q8_chan_scale", "q8_query_scratch"):
                getattr(new, name).copy_(src)
                continue
            getattr(new, name)[:, : src.shape[1]].copy_(src)
        new.used.copy_(self.used)
        return new


@dataclass
class CompactResult:
    """Compacted search output (see hira_search in include/hira_b200.h)."""
    idx: torch.Tensor      # (H_q, cap_children) int32, slot ids, valid in the first count entries of each tile segment
    score: torch.Tensor    # (H_q, cap_children) float32
    count: torch.Tensor    # (H_q, n_tiles) int32
    tile_parents: int
    tile_rows: int
    n_tiles_active: Optional[int] = None   # tiles the last search wrote (None: all)

    def __post_init__(self):
        """What a search has to be like for these buffers to take its output (compact_fits), None if nothing can."""
        hq, slots = self.idx.shape
        bf = self.tile_rows // self.tile_parents
        whole = (self.score.shape == self.idx.shape and bf * self.tile_parents == self.tile_rows
                 and self.count.shape == (hq, -(-(slots // bf) // self.tile_parents)))
        self.made_for = (hq, slots, bf, self.tile_parents, self.idx.device) if whole else None

    def to_lists(self):
        """Per query head: (slots, scores) as 1-D CPU tensors, ascending slot order."""
        idx, score, count = self.idx.cpu(), self.score.cpu(), self.count.cpu()
        out = []
        for qh in range(idx.shape[0]):
            sl, sc = [], []
            for t in range(count.shape[1] if self.n_tiles_active is None else self.n_tiles_active):
                c = int(count[qh, t])
                if c:
                    b = t * self.tile_rows
                    sl.append(idx[qh, b:b + c])
                    sc.append(score[qh, b:b + c])
            out.append((torch.cat(sl) if sl else torch.empty(0, dtype=torch.int32),
                        torch.cat(sc) if sc else torch.empty(0)))
        return out


def tile_parents(st: IndexState) -> int:
    tp = getattr(st, "_tile_parents", None)
    if tp is None:   # depends on bf, depth, capacity, heads and whether the int8 copy is in use now; kept from then on
        tp = st._tile_parents = int(L.load().hira_search_tile_parents(st.struct))
    return tp


def n_tiles(st: IndexState, tp: Optional[int] = None) -> int:
    tp = tp or tile_parents(st)
    return -(-st.cap_parents // tp)


def _f32(t: Optional[torch.Tensor], dev) -> Optional[torch.Tensor]:
    if t is None:
        return None
    return t.to(device=dev, dtype=torch.float32).contiguous()


def search(st: IndexState, q: torch.Tensor, tau: torch.Tensor, *, scaling=None, qnorm=None, q2kv=None,
           max_group: int = 0, flags: int = 0, out_dense=None, compact: Optional[CompactResult] = None,
           want_compact: bool = False, stats=None, tp: Optional[int] = None, scan_key=None, scan_out=None):
    """q (H_q, D) fp32, tau (H_q,) fp32 on the index device.  Returns (out_dense, CompactResult|None).
    With `scan_key` (n_heads, D) in the index dtype and `scan_out` (new_scan_slots), the parents are
    also scored against that key for the `append_scanned` that follows."""
    lib = L.load()
    hq = q.shape[0]
    tp = tp or (tile_parents(st) if compact is None else compact.tile_parents)
    if compact is not None:
        _check_compact(st, hq, compact, tp)
    elif want_compact:
        compact = alloc_compact(st, hq, tp)
    if scan_out is not None:
        if q2kv is not None:
            raise ValueError("the fused parent scan needs the default head grouping")
        assert scan_key.dtype == st.dtype and scan_key.shape[0] == st.n_heads and scan_key.stride(-1) == 1
        rc = lib.hira_search_scan(st.struct, L.ptr(q), L.ptr(tau), L.ptr(scaling), L.ptr(qnorm), hq, flags, tp,
                                  L.ptr(out_dense), L.ptr(compact.idx) if compact else None,
                                  L.ptr(compact.score) if compact else None, L.ptr(compact.count) if compact else None,
                                  L.ptr(stats), L.ptr(scan_key), scan_key.stride(0), L.ptr(scan_out),
                                  L.current_stream(st.device))
        L.check(rc, "hira_search_scan")
        if compact is not None:
            compact.n_tiles_active = None if (st.active_parents == 0 or out_dense is not None) \
                else -(-st.active_parents // tp)
        return out_dense, compact
    rc = lib.hira_search(st.struct, L.ptr(q), L.ptr(tau), L.ptr(scaling), L.ptr(qnorm), L.ptr(q2kv), hq,
                         max_group, flags, tp, L.ptr(out_dense),
                         L.ptr(compact.idx) if compact else None, L.ptr(compact.score) if compact else None,
                         L.ptr(compact.count) if compact else None, L.ptr(stats), L.current_stream(st.device))
    L.check(rc, "hira_search")
    if compact is not None:
        compact.n_tiles_active = None if (st.active_parents == 0 or out_dense is not None) \
            else -(-st.active_parents // tp)
    return out_dense, compact


def q8_fallback_count(device=None) -> int:
    """CTAs of the int8 pre-filter search on `device` (default: current) that took their exact fallback
    because a bounded wait ran out, since the library was loaded (hira_q8_fallback_count; synchronises)."""
    import ctypes as C
    v = C.c_uint32(0)
    with torch.cuda.device(device if device is not None else torch.cuda.current_device()):
        L.check(L.load().hira_q8_fallback_count(C.byref(v)), "hira_q8_fallback_count")
    return int(v.value)


def new_stats(hq: int, device) -> torch.Tensor:
    """Zeroed traffic counters for `search(..., stats=)`: (H_q, HIRA_SEARCH_STATS) int32."""
    return torch.zeros((hq, L.SEARCH_STATS), dtype=torch.int32, device=device)


def alloc_compact(st: IndexState, hq: int, tp: Optional[int] = None) -> CompactResult:
    tp = tp or tile_parents(st)
    dev = st.device
    return CompactResult(
        idx=torch.empty((hq, st.cap_children), dtype=torch.int32, device=dev),
        score=torch.empty((hq, st.cap_children), dtype=torch.float32, device=dev),
        count=torch.zeros((hq, n_tiles(st, tp)), dtype=torch.int32, device=dev),
        tile_parents=tp, tile_rows=tp * st.bf)


def compact_fits(st: IndexState, hq: int, c: CompactResult, tp: int) -> bool:
    """Whether `c` can take what a search of `st` by `hq` heads in tiles of `tp` parents writes.  The tile size
    is part of that: two indexes of equal capacity need not have the same."""
    return c.made_for == (hq, st.cap_children, st.bf, tp, st.arrays_device)


def _check_compact(st: IndexState, hq: int, c: CompactResult, tp: int):
    if not compact_fits(st, hq, c, tp):
        raise ValueError(f"compact buffers of {tuple(c.idx.shape)} slots and {tuple(c.count.shape)} tiles of {c.tile_parents} "
                         f"parents do not fit a search of this index by {hq} heads in tiles of {tp}")


def compact_for(st: IndexState, hq: int, have: Optional[CompactResult]) -> CompactResult:
    """`have` where a search of `st` by `hq` heads can reuse it, else new buffers."""
    return have if have is not None and compact_fits(st, hq, have, tile_parents(st)) else alloc_compact(st, hq)


@lru_cache(maxsize=256)
def _default_splits(hq: int, tiles: int) -> int:   # a pure function of the two numbers
    return int(L.load().hira_attn_default_splits(hq, tiles))


def attn_splits(st: IndexState, hq: int, tp: Optional[int] = None) -> int:
    tp = tp or tile_parents(st)
    tiles = n_tiles(st, tp) if st.active_parents == 0 else -(-st.active_parents // tp)
    return _default_splits(hq, tiles)


def queue_stride(t: torch.Tensor) -> Optional[int]:
    """Elements between the heads of a (B, H, n, D) or (H, n, D) queue whose rows lie one behind another from
    a 16-byte boundary -- a whole tensor or the filled part of a queue buffer --, None for any other layout.
    A stride along a dimension of one says nothing and is not looked at."""
    shape, strides = t.shape, t.stride()
    h, n, d, hs = shape[-3], shape[-2], shape[-1], strides[-3]
    if t.ndim == 4 and shape[0] > 1:
        if h == 1:                   # the heads to step over are the batch
            h, hs = shape[0], strides[0]
        elif strides[0] != h * hs:
            return None
    if h == 1:
        hs = n * d
    if strides[-1] != 1 or (n > 1 and strides[-2] != d) or hs < n * d or t.data_ptr() % 16 or hs * t.element_size() % 16:
        return None
    return hs


def dense_rows(t: torch.Tensor, dtype: torch.dtype, device) -> torch.Tensor:
    """A (..., n, D) queue as (H, n, D) rows that `queue_stride` accepts, copied where it does not as it is."""
    return aligned(t.reshape(-1, t.shape[-2], t.shape[-1]).to(device=device, dtype=dtype).contiguous())


def _queue_layout(st: IndexState, queued_k: torch.Tensor, queued_v: torch.Tensor):
    """(queued keys per head, elements between the heads): one stride serves both arrays."""
    assert queued_k.dtype == st.dtype and queued_v.dtype == st.vdtype
    if st.vdim != st.dim:
        raise ValueError("queued keys/values with vdim != dim are not supported")
    stride = queue_stride(queued_k)
    if stride is None or stride != queue_stride(queued_v):
        raise ValueError("queued keys and values must be rows one behind another from a 16-byte boundary, with one head stride")
    return queued_k.shape[-2], stride


def sparse_attn(st: IndexState, q, scaling, compact: CompactResult, *, q2kv=None, queued_k=None, queued_v=None,
                n_splits: Optional[int] = None, workspace=None, out=None, out_ml=None):
    """`out` / `out_ml` may be strided views (rows of a packed (H_q, 2 + V) message): only the
    last dimension has to be contiguous."""
    lib = L.load()
    hq = q.shape[0]
    _check_compact(st, hq, compact, compact.tile_parents)
    n_splits = n_splits or attn_splits(st, hq, compact.tile_parents)
    dev = st.device
    if workspace is None:
        workspace = torch.empty((hq * n_splits * (st.vdim + 2),), dtype=torch.float32, device=dev)
    if out is None:
        out = torch.empty((hq, st.vdim), dtype=torch.float32, device=dev)
    n_queued, qstride = 0, 0
    if queued_k is not None and queued_k.shape[-2] > 0:
        n_queued, qstride = _queue_layout(st, queued_k, queued_v)
    rc = lib.hira_sparse_attn(st.struct, L.ptr(q), L.ptr(scaling), L.ptr(q2kv), hq, compact.tile_parents,
                              L.ptr(compact.idx), L.ptr(compact.score), L.ptr(compact.count),
                              L.ptr(queued_k) if n_queued else None, L.ptr(queued_v) if n_queued else None,
                              n_queued, qstride, n_splits, L.ptr(workspace), L.ptr(out), L.ptr(out_ml),
                              out.stride(0), out_ml.stride(0) if out_ml is not None else 0, L.current_stream(dev))
    L.check(rc, "hira_sparse_attn")
    return out


def merge_partials(part_o, part_ml, out=None, out_ml=None):
    """part_o (n_parts, H_q, V), part_ml (n_parts, H_q, 2): any strides with a contiguous last
    dimension (e.g. two views of one gathered (n_parts, H_q, 2 + V) buffer)."""
    lib = L.load()
    n_parts, hq, vdim = part_o.shape
    assert part_o.stride(2) == 1 and part_ml.stride(2) == 1
    if out is None:
        out = torch.empty((hq, vdim), dtype=torch.float32, device=part_o.device)
    rc = lib.hira_merge_partials(L.ptr(part_o), L.ptr(part_ml), n_parts, hq, vdim, part_o.stride(0), part_o.stride(1),
                                 part_ml.stride(0), part_ml.stride(1), L.ptr(out), L.ptr(out_ml),
                                 L.current_stream(part_o.device))
    L.check(rc, "hira_merge_partials")
    return out


def _check_rows(t: torch.Tensor, h: int, m: int, width: int, dtype: torch.dtype):
    if t.numel() != h * m * width:
        raise ValueError(f"expected ({h}, {m}, {width}) rows, got {tuple(t.shape)}")
    assert t.is_contiguous() and t.dtype == dtype


def append(st: IndexState, new_k: torch.Tensor, new_v: Optional[torch.Tensor], token_base: int = -1,
           use_workspace: bool = True):
    """new_k (n_heads, M, D), new_v (n_heads, M, V) contiguous, index dtypes, on 16-byte boundaries."""
    lib = L.load()
    m = new_k.shape[1]
    _check_rows(new_k, st.n_heads, m, st.dim, st.dtype)
    if new_v is not None:
        _check_rows(new_v, st.n_heads, m, st.vdim, st.vdtype)
    ws, nbytes, stream = None, 0, L.current_stream(st.device)
    if use_workspace:
        sizes = st._append_bytes     # depends on the heads, the capacity and m only
        nbytes = sizes.get(m)
        if nbytes is None:
            nbytes = sizes[m] = int(lib.hira_append_workspace_bytes(st.struct, m))
        if nbytes:
            ws, home = st._append_ws
            if ws is None or ws.numel() < nbytes or home != stream:    # scratch of the stream it is used on
                ws = torch.empty((nbytes,), dtype=torch.uint8, device=st.device)
                st._append_ws = ws, stream
    rc = lib.hira_append(st.struct, L.ptr(new_k), L.ptr(new_v), m, m * st.dim,
                         m * st.vdim if new_v is not None else 0, token_base, L.ptr(st.status),
                         L.ptr(ws), nbytes, stream)
    L.check(rc, "hira_append")


def new_scan_slots(st: IndexState) -> torch.Tensor:
    """The (n_heads,) buffer `search(..., scan_out=)` fills and `append_scanned` consumes."""
    return torch.full((st.n_heads,), -1, dtype=torch.int64, device=st.device)


def append_scanned(st: IndexState, new_k: torch.Tensor, new_v: Optional[torch.Tensor], scan: torch.Tensor,
                   token_base: int = -1):
    """One key per head, new_k (n_heads, 1, D) / new_v (n_heads, 1, V) in the index dtypes, whose
    nearest parent the preceding `search(..., scan_key=new_k[:, 0], scan_out=scan)` found."""
    lib = L.load()
    assert new_k.dtype == st.dtype and new_k.shape == (st.n_heads, 1, st.dim) and new_k.stride(-1) == 1
    if new_v is not None:
        assert new_v.dtype == st.vdtype and new_v.shape == (st.n_heads, 1, st.vdim) and new_v.stride(-1) == 1
    rc = lib.hira_append_scanned(st.struct, L.ptr(new_k), L.ptr(new_v), new_k.stride(0),
                                 new_v.stride(0) if new_v is not None else 0, token_base, L.ptr(st.status),
                                 L.ptr(scan), L.current_stream(st.device))
    L.check(rc, "hira_append_scanned")


def threshold(samples: torch.Tensor, q: torch.Tensor, method: int, k: int = 1, q2kv=None, out=None):
    """samples (H_kv, S, D) contiguous fp32/bf16, q (H_q, D) fp32 -> tau (H_q,)."""
    lib = L.load()
    hkv, s, d = samples.shape
    hq = q.shape[0]
    if out is None:
        out = torch.empty((hq,), dtype=torch.float32, device=q.device)
    rc = lib.hira_threshold(L.ptr(samples), L.dtype_code(samples.dtype), hkv, s, d, s * d, L.ptr(q), L.ptr(q2kv),
                            hq, method, k, L.ptr(out), L.current_stream(q.device))
    L.check(rc, "hira_threshold")
    return out


def prepare_query(q: torch.Tensor, sm_scale: float, q_hat=None, logit_scale=None):
    """q (H_q, D) fp32/bf16 contiguous -> (q_hat (H_q, D) fp32, logit_scale (H_q,) fp32)."""
    lib = L.load()
    hq, d = q.shape
    if q_hat is None:
        q_hat = torch.empty((hq, d), dtype=torch.float32, device=q.device)
    if logit_scale is None:
        logit_scale = torch.empty((hq,), dtype=torch.float32, device=q.device)
    rc = lib.hira_prepare_query(L.ptr(q), L.dtype_code(q.dtype), hq, d, float(sm_scale), L.ptr(q_hat),
                                L.ptr(logit_scale), L.current_stream(q.device))
    L.check(rc, "hira_prepare_query")
    return q_hat, logit_scale


def decode_attention(st: IndexState, q: torch.Tensor, sm_scale: float, tau: torch.Tensor, compact: CompactResult,
                     q_hat: torch.Tensor, logit_scale: torch.Tensor, *, q2kv=None, max_group: int = 0, flags: int = 0,
                     queued_k=None, queued_v=None, n_splits: int, workspace: torch.Tensor, out: torch.Tensor,
                     out_ml=None, scan_key=None, scan_out=None, searched_event=None, tau_samples=None,
                     tau_method: int = 0, tau_k: int = 1):
    """prepare_query + search (compact) + sparse_attn in one library call.  q (H_q, D) fp32/bf16
    contiguous; everything else preallocated by the caller.  With `tau_samples` (H_kv, S, D) in the index
    dtype the threshold is found on the way, into `tau`."""
    lib = L.load()
    hq = q.shape[0]
    _check_compact(st, hq, compact, compact.tile_parents)
    n_queued, qstride = 0, 0
    if queued_k is not None and queued_k.shape[-2] > 0:
        n_queued, qstride = _queue_layout(st, queued_k, queued_v)
    rest = (L.ptr(q2kv), hq, max_group, flags, compact.tile_parents, L.ptr(q_hat), L.ptr(logit_scale),
            L.ptr(compact.idx), L.ptr(compact.score), L.ptr(compact.count),
            L.ptr(queued_k) if n_queued else None, L.ptr(queued_v) if n_queued else None,
            n_queued, qstride, n_splits, L.ptr(workspace), L.ptr(out), L.ptr(out_ml),
            out.stride(0), out_ml.stride(0) if out_ml is not None else 0,
            L.ptr(scan_key) if scan_out is not None else None,
            scan_key.stride(0) if scan_out is not None else 0, L.ptr(scan_out),
            searched_event, L.current_stream(st.device))
    if tau_samples is None:
        rc = lib.hira_decode_attention(st.struct, L.ptr(q), L.dtype_code(q.dtype), float(sm_scale), L.ptr(tau), *rest)
    else:
        assert tau_samples.dtype == st.dtype and tau_samples.is_contiguous() and tau_samples.shape[0] == st.n_heads
        rc = lib.hira_decode_attention_sampled(st.struct, L.ptr(q), L.dtype_code(q.dtype), float(sm_scale),
                                               L.ptr(tau_samples), tau_samples.shape[1], tau_samples.stride(0),
                                               tau_method, tau_k, L.ptr(tau), *rest)
    L.check(rc, "hira_decode_attention")
    compact.n_tiles_active = None if st.active_parents == 0 else -(-st.active_parents // compact.tile_parents)
    return out


def kth_score(st: IndexState, compact: CompactResult, k: torch.Tensor, out=None):
    lib = L.load()
    hq = compact.idx.shape[0]
    _check_compact(st, hq, compact, compact.tile_parents)
    if out is None:
        out = torch.empty((hq,), dtype=torch.float32, device=st.device)
    rc = lib.hira_kth_score(st.struct, hq, compact.tile_parents, L.ptr(compact.score), L.ptr(compact.count),
                            L.ptr(k), L.ptr(out), L.current_stream(st.device))
    L.check(rc, "hira_kth_score")
    return out


def build(st: IndexState, keys: torch.Tensor, values: Optional[torch.Tensor], *, cent_idx1=None, cent_idx2=None,
          n_iters: int = 1, balance_rounds: int = 0, use_tensor_cores: bool = True, token_base: int = 0):
    """keys (n_heads, n, D), values (n_heads, n, V) contiguous, index dtypes."""
    lib = L.load()
    assert keys.is_contiguous() and keys.dtype == st.dtype
    n = keys.shape[1]
    if values is not None:
        assert values.is_contiguous() and values.dtype == st.vdtype
    st.status.zero_()
    nbytes = int(lib.hira_build_workspace_bytes(st.struct, n))
    ws = torch.empty((max(nbytes, 1),), dtype=torch.uint8, device=st.device)
    rc = lib.hira_build(st.struct, L.ptr(keys), L.ptr(values), n, n * st.dim,
                        n * st.vdim if values is not None else 0, token_base, L.ptr(cent_idx1), L.ptr(cent_idx2),
                        n_iters, int(balance_rounds), 1 if use_tensor_cores else 0, L.ptr(st.status), L.ptr(ws), nbytes,
                        L.current_stream(st.device))
    L.check(rc, "hira_build")


def stratified(u: torch.Tensor, n: int) -> torch.Tensor:
    """u (H, k) in [0, 1) -> (H, k) int32: the point u draws out of each of k equal strides of n points."""
    h, k = u.shape
    out = torch.empty((h, k), dtype=torch.int32, device=u.device)
    L.check(L.load().hira_stratified(L.ptr(u), h, n, k, L.ptr(out), L.current_stream(u.device)), "hira_stratified")
    return out


def recompute_radii(st: IndexState):
    L.check(L.load().hira_recompute_radii(st.struct, L.current_stream(st.device)), "hira_recompute_radii")


def export(st: IndexState, n_out: int, token_base: int = 0):
    lib = L.load()
    out_k = torch.zeros((st.n_heads, n_out, st.dim), dtype=st.dtype, device=st.device)
    out_v = torch.zeros((st.n_heads, n_out, st.vdim), dtype=st.vdtype, device=st.device) if st.values is not None else None
    rc = lib.hira_export(st.struct, token_base, n_out, L.ptr(out_k), L.ptr(out_v), L.current_stream(st.device))
    L.check(rc, "hira_export")
    return out_k, out_v


def assign(points: torch.Tensor, cents: torch.Tensor, use_tensor_cores: bool = False):
    """points (H, n, D), cents (H, k, D) -> (idx (H, n) int32, dist2 (H, n) fp32)."""
    lib = L.load()
    h, n, d = points.shape
    k = cents.shape[1]
    dev = points.device
    idx = torch.empty((h, n), dtype=torch.int32, device=dev)
    d2 = torch.empty((h, n), dtype=torch.float32, device=dev)
    csq = torch.empty((h, k), dtype=torch.float32, device=dev)
    rc = lib.hira_assign(L.ptr(points.contiguous()), L.ptr(cents.contiguous()), L.dtype_code(points.dtype), h, n, k, d,
                         1 if use_tensor_cores else 0, L.ptr(csq), L.ptr(idx), L.ptr(d2), L.current_stream(dev))
    L.check(rc, "hira_assign")
    return idx, d2


class DecodeStep:
    """Device scratch and events of `hira_decode_step` for one index: the whole decode step of a
    layer (query copy, threshold, search, sparse attention, output copy and, beside them on a
    second stream, the 1-key append) behind one library call with host buffers in and out."""

    def __init__(self, st: IndexState, n_qheads: int, q_dtype: torch.dtype = torch.float32, *, flags: int,
                 fused_scan: bool = False, tau_samples: Optional[torch.Tensor] = None,
                 tau_method: int = L.HIRA_TAU_SAMPLE_MEAN_TOPK, tau_k: int = 16):
        lib = L.load()
        dev = st.device
        self.st, self.n_qheads, self.q_dtype = st, n_qheads, q_dtype
        tp = tile_parents(st)
        self.compact = alloc_compact(st, n_qheads, tp)
        # splits sized for the whole capacity: the bound on the slots in use moves from step to step
        self.n_splits = int(lib.hira_attn_default_splits(n_qheads, n_tiles(st, tp)))
        f32 = dict(dtype=torch.float32, device=dev)
        self.q_dev = torch.empty((n_qheads, st.dim), dtype=q_dtype, device=dev)
        self.k_dev = torch.empty((st.n_heads, st.dim), dtype=st.dtype, device=dev)
        self.v_dev = torch.empty((st.n_heads, max(st.vdim, 1)), dtype=st.vdtype, device=dev)
        self.q_hat = torch.empty((n_qheads, st.dim), **f32)
        self.logit_scale = torch.empty((n_qheads,), **f32)
        self.tau = torch.empty((n_qheads,), **f32)
        self.workspace = torch.empty((n_qheads * self.n_splits * (st.vdim + 2),), **f32)
        self.out_dev = torch.empty((n_qheads, st.vdim), **f32)
        self.scan = new_scan_slots(st) if fused_scan else None
        nbytes = int(lib.hira_append_workspace_bytes(st.struct, 1))
        self.append_ws = torch.empty((max(nbytes, 1),), dtype=torch.uint8, device=dev) if nbytes else None
        self.tau_samples = tau_samples
        s = L.HiraStepStruct()
        for name in ("q_dev", "k_dev", "v_dev", "q_hat", "logit_scale", "tau", "workspace", "out_dev", "scan",
                     "append_ws", "tau_samples"):
            setattr(s, name, L.ptr(getattr(self, name)))
        s.idx, s.score, s.count = L.ptr(self.compact.idx), L.ptr(self.compact.score), L.ptr(self.compact.count)
        s.status = L.ptr(st.status)
        s.append_ws_bytes = nbytes
        if tau_samples is not None:
            assert tau_samples.dtype == st.dtype and tau_samples.is_contiguous() and tau_samples.shape[0] == st.n_heads
            s.n_samples, s.samples_head_stride = tau_samples.shape[1], tau_samples.stride(0)
        s.tau_method, s.tau_k = tau_method, tau_k
        s.n_splits, s.tile_parents, s.flags = self.n_splits, tp, flags
        self._struct = s
        L.check(lib.hira_step_events_create(C.byref(s)), "hira_step_events_create")

    def __del__(self):
        try:
            L.load().hira_step_events_destroy(C.byref(self._struct))
        except Exception:
            pass

    def run(self, q_host: torch.Tensor, out_host: torch.Tensor, *, sm_scale: float, tau: Optional[torch.Tensor] = None,
            k_host: Optional[torch.Tensor] = None, v_host: Optional[torch.Tensor] = None, side_stream=None):
        """q_host (H_q, D), k_host (H_kv, D), v_host (H_kv, V), out_host (H_q, V) fp32: contiguous
        (pinned) host tensors.  `tau` (H_q,) on the device, or None to find it from the samples."""
        st = self.st
        assert q_host.dtype == self.q_dtype and q_host.is_contiguous() and out_host.is_contiguous()
        rc = L.load().hira_decode_step(st.struct, C.byref(self._struct), q_host.data_ptr(), L.dtype_code(self.q_dtype),
                                       float(sm_scale), self.n_qheads, L.ptr(tau),
                                       None if k_host is None else k_host.data_ptr(),
                                       None if v_host is None else v_host.data_ptr(), out_host.data_ptr(),
                                       L.current_stream(st.device),
                                       None if side_stream is None else side_stream.cuda_stream)
        L.check(rc, "hira_decode_step")
