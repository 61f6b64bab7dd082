"""Kernels at the sizes where they can go wrong: edges of tiles, remainders, the smallest and largest of a range."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from hira_b200 import _lib as L
from hira_b200 import index_state as S
from oracle import oracle as O

from util import assert_index_equal, build_both, make_keys, make_queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("d", [8, 64, 128, 200])
@pytest.mark.parametrize("s,k", [(1, 1), (31, 31), (32, 32), (33, 32), (33, 33), (1000, 32), (1000, 33), (1025, 7), (4096, 32), (4096, 4096)])
def test_threshold_lists_and_full_sort(dtype, d, s, k):
    """Up to 32 wanted scores come from merged lists, more from a sort of all: both sides of that line."""
    h, group = 2, 2
    samples = make_keys(h, s, d, 3, dtype)
    q = make_queries(h * group, d, seed=4)
    for method in (L.HIRA_TAU_SAMPLE_MAX, L.HIRA_TAU_SAMPLE_MEAN_TOPK, L.HIRA_TAU_SAMPLE_KTH):
        got = S.threshold(samples, q, method, k).cpu().numpy()
        want = O.threshold(samples, q, method, k)
        assert np.array_equal(got.view(np.uint32), np.asarray(want, np.float32).view(np.uint32))


def test_threshold_sorts_nan_scores_last():
    samples = make_keys(1, 100, 64, 5)
    samples[0, 17, 3] = float("nan")
    q = make_queries(1, 64, seed=6)
    keep = torch.cat([samples[:, :17], samples[:, 18:]], dim=1).contiguous()
    for k in (5, 40):
        assert torch.equal(S.threshold(samples, q, L.HIRA_TAU_SAMPLE_MEAN_TOPK, k), S.threshold(keep, q, L.HIRA_TAU_SAMPLE_MEAN_TOPK, k))
