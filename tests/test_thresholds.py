"""Thresholds of a screen from rows of group values at the sizes where the kernel that ranks them changes. Every row is an
anchor, so the k-th largest group value lets through little more than k rows: a threshold that is too high loses answers, one that
is too low keeps many rows."""

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,metric", [("float32", "l2"), ("int8", "ip")])
@pytest.mark.parametrize("groups", [4, 32, 508, 512, 516, 1020, 1024, 1028, 4096, 4100])
@pytest.mark.parametrize("k", [1, 2, 100, 1000])
def test_thresholds_at_the_edges(k, groups, dtype, metric):
    if 2 * k > groups:
        pytest.skip("fewer groups than a threshold needs")
    rng = np.random.default_rng(groups + k)
    n, d, nq = groups * 64, 24, 13
    x = rng.integers(-127, 128, (n, d)).astype(dtype)
    q = rng.integers(-127, 128, (nq, d)).astype(dtype)
    index = certex.Index(d, metric=metric, anchor_stride=1)
    index.add(torch.from_numpy(x).cuda())
    with certex.search_stats() as st:
        _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=k, return_scores=True)
    assert st.screen_passes == 1 and st.dense_queries == 0 and st.rescreened == 0
    assert st.survivors <= nq * (3 * k + 64)
    want_ids, want_scores = oracle.knn(x, q, k, metric)
    assert np.array_equal(ids.cpu().numpy(), want_ids) and np.array_equal(scores.cpu().numpy(), want_scores)
