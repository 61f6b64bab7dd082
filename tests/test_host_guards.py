"""Host-side guards between the Python classes and the kernels, on the CPU: a call whose buffers do not fit what a
kernel would write or read is refused, or given buffers that do, before anything is launched."""
from types import SimpleNamespace

import pytest
import torch

from hira_b200 import CUDASearcher, hira_decode_attention
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
