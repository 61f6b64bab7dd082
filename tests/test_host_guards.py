"""Host-side guards between the Python classes and the kernels, on the CPU: a call whose buffers do not fit what a
kernel would write or read is refused, or given buffers that do, before anything is launched."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from hira_b200 import CUDAIndexer, CUDASearcher, DeviceMode, HiraCacheLayer, hira_decode_attention
from hira_b200 import _lib as L
from hira_b200 import index_state as S


def _state(dim, n_heads=8, bf=32, depth=3, cap_parents=288, dtype=torch.bfloat16, **kw):
    return S.IndexState(n_heads=n_heads, dim=dim, vdim=dim, bf=bf, depth=depth, cap_parents=cap_parents, dtype=dtype,
                        vdtype=dtype, device="cpu", **kw)


def _two_tilings():
    """Two indexes of the same heads, branching and capacity whose searches use tiles of different sizes."""
    a, b = _state(128, int8_copy=True), _state(64)
    assert a.cap_children == b.cap_children and S.tile_parents(a) != S.tile_parents(b)
    return a, b


def test_search_refuses_compact_buffers_of_another_tiling():
    a, b = _two_tilings()
    q, tau = torch.zeros(16, 64), torch.zeros(16)
    assert S.compact_fits(b, 16, S.alloc_compact(a, 16), S.tile_parents(a))    # any tile size, as long as the buffers are its
    for have in (S.alloc_compact(_state(64, bf=16, cap_parents=576), 16), S.alloc_compact(b, 15)):
        with pytest.raises(ValueError, match="do not fit"):
            S.search(b, q, tau, compact=have)
        with pytest.raises(ValueError, match="do not fit"):
            S.sparse_attn(b, q, tau, have)
    with pytest.raises(ValueError, match="do not fit"):      # a tile size the buffers were not made for
        S.search(b, q, tau, compact=S.alloc_compact(b, 16), tp=S.tile_parents(a))


def test_one_searcher_serves_indexes_of_different_tilings(monkeypatch):
    a, b = _two_tilings()
    searcher, seen = CUDASearcher(), []
    monkeypatch.setattr(S, "search", lambda st, q, tau, **kw: seen.append((st, q.shape[0], kw["compact"])))
    monkeypatch.setattr(S, "decode_attention", lambda st, q, sc, tau, compact, *r, **kw: seen.append((st, q.shape[0], compact)))
    for st in (a, b, b, a):
        ix = SimpleNamespace(state=st)
        searcher.search_compact(torch.zeros(16, st.dim), torch.zeros(16), ix)
        out = SimpleNamespace(indexer=ix, searcher=searcher, queued_keys=None, queued_values=None)
        hira_decode_attention(torch.zeros(1, 16, 1, st.dim), out, threshold=torch.zeros(16))
    for st, hq, c in seen:
        tp = S.tile_parents(st)
        assert (c.tile_parents, c.tile_rows) == (tp, tp * st.bf) and c.count.shape == (hq, S.n_tiles(st, tp))
    assert seen[2][2] is seen[4][2] and seen[3][2] is seen[5][2]     # kept while the index stays the same


def _indexer(h=4, dim=64, vdim=64, dtype=torch.bfloat16):
    """An indexer on host memory: its appends are recorded by `_record_appends`."""
    ix = CUDAIndexer(3, 1, 8, max_context=4096)
    ix.state = S.IndexState(n_heads=h, dim=dim, vdim=vdim, bf=8, depth=3, cap_parents=512, dtype=dtype, vdtype=dtype, device="cpu")
    ix.num_heads, ix.dim = h, dim
    return ix


def _record_appends(monkeypatch):
    seen = []

    def append(st, k, v, *a, **kw):
        S._check_rows(k, st.n_heads, k.shape[1], st.dim, st.dtype)
        S._check_rows(v, st.n_heads, k.shape[1], st.vdim, st.vdtype)
        assert k.data_ptr() % 16 == 0 and v.data_ptr() % 16 == 0
        seen.append((k, v))
    monkeypatch.setattr(S, "append", append)
    return seen


def _layer(ix, update_every=1):
    layer = HiraCacheLayer(DeviceMode.CUDA_ONLY, update_every, {}, {})
    layer.indexer_cls, layer.searcher_cls = lambda **kw: ix, lambda **kw: None
    ix.build = lambda k, v: ix
    st = ix.state
    layer.update(torch.zeros(1, st.n_heads, 3, st.dim, dtype=st.dtype), torch.zeros(1, st.n_heads, 3, st.vdim, dtype=st.dtype))
    return layer


def _off_by(shape, elements, dtype=torch.bfloat16):
    """A contiguous tensor that starts `elements` behind a 16-byte boundary, as a view into a fused projection does."""
    n = torch.Size(shape).numel()
    t = torch.arange(n + elements).to(dtype)[elements:].view(shape)
    assert t.is_contiguous() and t.data_ptr() % 16 == elements * t.element_size() % 16
    return t


@pytest.mark.parametrize("width", [32, 72, 128])
def test_values_of_another_width_are_refused(monkeypatch, width):
    seen = _record_appends(monkeypatch)
    ix = _indexer()
    layer = _layer(ix)
    with pytest.raises(RuntimeError):            # as the queue refuses them
        layer.update(torch.zeros(1, 4, 1, 64, dtype=torch.bfloat16), torch.zeros(1, 4, 1, width, dtype=torch.bfloat16))
    with pytest.raises(ValueError, match="wide"):
        ix.update(torch.zeros(1, 4, 1, 64, dtype=torch.bfloat16), torch.zeros(1, 4, 1, width, dtype=torch.bfloat16))
    assert not seen


def test_what_the_queue_broadcasts_is_still_broadcast(monkeypatch):
    seen = _record_appends(monkeypatch)
    layer = _layer(_indexer())
    k, v = torch.randn(1, 4, 3, 64).bfloat16(), torch.randn(1, 4, 1, 1).bfloat16()
    layer.update(k, v)
    assert torch.equal(seen[0][0], k[0]) and torch.equal(seen[0][1], v[0].expand(4, 3, 64)) and layer.get_seq_length() == 6


@pytest.mark.parametrize("elements", [0, 1, 4, 7])
@pytest.mark.parametrize("batch", [1, 2])
def test_unaligned_keys_and_values_are_copied_to_a_boundary(monkeypatch, elements, batch):
    seen = _record_appends(monkeypatch)
    ix = _indexer()
    k, v = _off_by((batch, 4 // batch, 2, 64), elements), _off_by((batch, 4 // batch, 2, 64), 2 * elements)
    ix.update(k, v)
    if batch == 1:
        _layer(ix, 2).update(k, v)
    for a, b in seen:
        assert torch.equal(a, k.view(4, 2, 64)) and torch.equal(b, v.view(4, 2, 64))
        assert elements or a.data_ptr() == k.data_ptr()      # nothing is copied without need
    assert len(seen) == 3 - batch
    assert ix.begin_scanned_update(k[:, :, :1])[0].data_ptr() % 16 == 0


def test_append_refuses_unaligned_rows_before_any_launch():
    lib, st = L.load(), _indexer().state
    status = torch.zeros(1, dtype=torch.int32)
    base = torch.zeros(4 * 2 * 64 + 8, dtype=torch.bfloat16).data_ptr()
    assert base % 16 == 0
    for k, v, ks, vs in ((base + 2, base, 64, 64), (base, base + 8, 64, 64), (base, base, 68, 64), (base, base, 64, 65)):
        for rc in (lib.hira_append(st.struct, k, v, 1, ks, vs, -1, status.data_ptr(), None, 0, None),
                   lib.hira_append_scanned(st.struct, k, v, ks, vs, -1, status.data_ptr(), status.data_ptr(), None)):
            assert rc == L.HIRA_ERR_ARG and b"16-byte" in lib.hira_last_error()
    with pytest.raises(ValueError, match="rows"):
        S.append(st, torch.zeros(4, 1, 64, dtype=torch.bfloat16), torch.zeros(4, 1, 32, dtype=torch.bfloat16))


class _FakeStream:
    cuda_stream = 0

    def __init__(self, name, log):
        self.name, self.log = name, log

    def wait_stream(self, other):
        self.log.append((self.name, "waits for", other.name))

    def wait_event(self, event):
        self.log.append((self.name, "waits for", "event"))


def _fake_streams(monkeypatch, log):
    main, side = _FakeStream("main", log), _FakeStream("side", log)
    active = [main]

    class _On:
        def __init__(self, s):
            self.s = s

        def __enter__(self):
            active.append(self.s)

        def __exit__(self, *a):
            active.pop()
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: active[-1])
    monkeypatch.setattr(torch.cuda, "stream", _On)
    monkeypatch.setattr(torch.cuda, "Event", lambda: SimpleNamespace(record=lambda s: log.append((s.name, "record"))))
    return side, active


def test_growth_of_a_side_stream_update_runs_where_the_index_lives(monkeypatch):
    """The old arrays are read, and the new ones allocated, on the stream whose memory they are."""
    log = []
    side, active = _fake_streams(monkeypatch, log)
    grown = S.IndexState.grown
    monkeypatch.setattr(S.IndexState, "grown", lambda st, n: log.append((active[-1].name, "grows")) or grown(st, n))
    monkeypatch.setattr(S.IndexState, "used_on", lambda st, s: log.append((s.name, "uses", st.cap_parents)), raising=False)
    monkeypatch.setattr(S, "append", lambda st, k, v: log.append((active[-1].name, "appends")))
    ix = _indexer()
    ix._parents_bound, ix._gp_bound = ix.state.cap_parents, ix.state.cap_gp
    ix.state.used[:, 0], ix.state.used[:, 1] = ix._parents_bound, ix._gp_bound
    row = torch.zeros(1, 4, 1, 64, dtype=torch.bfloat16)
    ix.update(row, row, stream=side)
    assert log == [("side", "waits for", "main"), ("main", "waits for", "side"), ("main", "grows"), ("side", "waits for", "main"),
                   ("side", "uses", 768), ("side", "appends"), ("side", "record")]
    log.clear()
    ix.update(row, row)
    assert log == [("main", "waits for", "event"), ("main", "appends")]


def _odd_queues():
    """Queues that are dense, or become so by a copy, in layouts a caller can come by; (keys, values) of 4 heads."""
    def whole(n, b=1):
        return torch.randn(b, 4 // b, n, 64).bfloat16()
    yield "whole", whole(3), whole(3)
    yield "batch", whole(3, 2), whole(3, 2)
    yield "filled part", whole(8, 2)[:, :, :3], whole(8, 2)[:, :, :3]
    yield "another head stride", whole(8)[:, :, :3], whole(5)[:, :, :3]
    yield "unaligned", _off_by((1, 4, 3, 64), 1), _off_by((1, 4, 3, 64), 3)
    yield "unaligned values", whole(3), _off_by((1, 4, 3, 64), 4)
    yield "one row, transposed", torch.randn(1, 1, 4, 64).bfloat16().transpose(1, 2), torch.randn(1, 1, 4, 64).bfloat16().transpose(1, 2)
    yield "one head a batch item", whole(3, 4), torch.randn(3, 4, 1, 64).bfloat16().permute(1, 2, 0, 3)
    yield "strides of ones", whole(1).as_strided((1, 4, 1, 64), (7, 64, 9, 1)), whole(1).as_strided((1, 4, 1, 64), (1, 64, 1, 1))
    yield "broadcast", whole(1).expand(1, 4, 3, 64), whole(3)
    yield "floats", whole(3).float(), whole(3).float()


@pytest.mark.parametrize("what,qk,qv", [pytest.param(*c, id=c[0]) for c in _odd_queues()])
def test_queues_of_any_layout_reach_the_attention(monkeypatch, what, qk, qv):
    seen = []
    monkeypatch.setattr(S, "decode_attention", lambda *a, queued_k, queued_v, **kw: seen.append((queued_k, queued_v)))
    ix = _indexer()
    out = SimpleNamespace(indexer=SimpleNamespace(state=ix.state), searcher=CUDASearcher(), queued_keys=qk, queued_values=qv)
    hira_decode_attention(torch.zeros(1, 8, 1, 64), out, threshold=torch.zeros(8))
    n, stride = S._queue_layout(ix.state, *seen[0])
    assert n == qk.shape[-2]
    for got, want in zip(seen[0], (qk, qv)):
        assert got.data_ptr() % 16 == 0
        assert torch.equal(torch.as_strided(got, (4, n, 64), (stride, 64, 1)), want.reshape(4, n, 64).bfloat16())
    if what in ("whole", "batch", "filled part", "one row, transposed"):
        assert seen[0][0] is qk and seen[0][1] is qv       # read in place


def test_dense_three_dimensional_queues_are_taken():
    st = _indexer().state
    row = torch.randn(1, 4, 64).bfloat16().transpose(0, 1)      # (H, 1, D), contiguous whatever its row stride
    assert row.is_contiguous() and S._queue_layout(st, row, row) == (1, 64)
    with pytest.raises(ValueError, match="16-byte"):
        S._queue_layout(st, _off_by((4, 3, 64), 1), _off_by((4, 3, 64), 1))


@pytest.mark.parametrize("batch", [1, 2])
def test_an_update_without_keys_changes_nothing(monkeypatch, batch):
    seen = _record_appends(monkeypatch)
    ix = _indexer()
    none = torch.zeros(batch, 4 // batch, 0, 64, dtype=torch.bfloat16)
    assert ix.update(none, none) is ix and not seen and ix._appended == 0


@pytest.mark.parametrize("sample_size,want", [(-3, 1), (0, 1), (1, 1), (40, 40), (64, 64), (1000, 64)])
def test_threshold_samples_are_at_least_one_and_at_most_the_keys(sample_size, want):
    from hira_b200.attention.hira_attention import _samples_for
    for built in (0, 64):                       # loaded from arrays (the keys are counted), or built from 64 of them
        ix = SimpleNamespace(state=_state(64, n_heads=4, bf=8, cap_parents=16, dtype=torch.float32), _built_keys=built)
        ix.state.slot2token[:, :64] = torch.arange(64)
        ix.state.children[:, :64] = 1.0
        rows = _samples_for(ix, sample_size)
        assert rows.shape == (4, want, 64) and bool((rows == 1.0).all())
        assert _samples_for(ix, sample_size).shape == rows.shape


@pytest.mark.parametrize("dim,dtype,cap,rows", [(64, torch.float32, 1024, 512), (64, torch.bfloat16, 1024, 512), (64, torch.float32, 512, 256),
                                                (200, torch.float32, 1024, 1024), (200, torch.float32, 896, 512), (200, torch.float32, 512, 512),
                                                (128, torch.float32, 1024, 1024), (256, torch.bfloat16, 992, 512), (256, torch.bfloat16, 480, 256),
                                                (64, torch.float32, 32, 256), (256, torch.bfloat16, 32, 256)])
def test_tile_size_follows_the_bytes_of_a_row(dim, dtype, cap, rows):
    """8 heads of branching 32: tiles are halved while they are too few to keep the memory busy, of long rows fewer."""
    assert S.tile_parents(_state(dim, cap_parents=cap, dtype=dtype)) * 32 == rows


@pytest.mark.parametrize("heads,cap,depth,parts", [(1, 4096, 3, 32), (1, 32768, 2, 64), (8, 4096, 3, 32), (8, 32768, 3, 36), (32, 1024, 3, 8), (32, 1024, 2, 8),
                                                   (32, 2048, 2, 9), (64, 1024, 3, 3), (128, 1024, 3, 2), (128, 512, 3, 1), (128, 4096, 3, 2), (128, 512, 2, 2),
                                                   (80, 4096, 3, 6), (80, 1024, 3, 2), (400, 512, 3, 1), (400, 4096, 3, 2), (8, 128, 3, 1)])
def test_append_slices_fit_the_gpu_at_once(heads, cap, depth, parts):
    """The workspace holds one result of 8 bytes a slice and one of the grandparents, per key and head."""
    st = _state(8, n_heads=heads, bf=8, depth=depth, cap_parents=cap)
    for m in (1, 32):
        assert L.load().hira_append_workspace_bytes(st.struct, m) == heads * m * (parts + 1) * 8
    assert L.load().hira_append_workspace_bytes(st.struct, 33) == 0


def test_a_refused_side_stream_update_does_not_hide_the_one_before(monkeypatch):
    log = []
    side, active = _fake_streams(monkeypatch, log)
    monkeypatch.setattr(S.IndexState, "used_on", lambda st, s: None)
    monkeypatch.setattr(S, "append", lambda st, k, v: None)
    ix = _indexer()
    row = torch.zeros(1, 4, 1, 64, dtype=torch.bfloat16)
    ix.update(row, row, stream=side)
    with pytest.raises(ValueError):
        ix.update(row[..., :32], row, stream=side)
    log.clear()
    ix.wait_pending_update()
    assert log == [("main", "waits for", "event")]
