"""The selection of searches that score every row: rows of scores around the sizes where its blocks change, more equal scores
than its pool holds, scores over many orders of magnitude, fewer rows that may be returned than k, rows cut into chunks."""

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from oracle import oracle

pytestmark = pytest.mark.gpu


def _case(kind, n, d, rng):
    if kind == "equal":
        return np.tile(rng.integers(-5, 5, (1, d)), (n, 1)).astype(np.float32)
    if kind == "few":  # a handful of distinct rows: thousands of equal scores at every rank
        return rng.integers(-5, 5, (7, d)).astype(np.float32)[rng.integers(0, 7, n)]
    if kind == "wide":
        return (rng.standard_normal((n, d)) * 10.0 ** rng.uniform(-12, 3, (n, 1))).astype(np.float32)
    return rng.standard_normal((n, d)).astype(np.float32)


@pytest.mark.parametrize("kind", ["normal", "equal", "few", "wide"])
@pytest.mark.parametrize("n,k", [(1, 1), (5, 5), (300, 17), (2048, 2048), (8192, 100), (8193, 2047), (40_000, 2048), (270_000, 100)])
@pytest.mark.parametrize("metric", ["l2", "ip"])
def test_dense_selection(n, k, kind, metric):
    rng = np.random.default_rng(n + k)
    d, nq = 8, 5
    x, q = _case(kind, n, d, rng), _case(kind, nq, d, rng)
    index = certex.Index(d, metric=metric)
    index.add(torch.from_numpy(x).cuda())
    index._test_mode(1)
    masks = [None] if n > 100_000 else [None, rng.random((nq, n)) < min(1.0, 1.2 * k / n)]
    for mask in masks:
        with certex.search_stats() as st:
            _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=k, return_scores=True,
                                          filter=None if mask is None else torch.from_numpy(mask).cuda())
        assert st.dense_queries == nq
        want_ids, want_scores = oracle.knn(x, q, k, metric, keep_pair=mask)
        assert np.array_equal(ids.cpu().numpy(), want_ids)
        assert np.array_equal(scores.cpu().numpy(), want_scores)
