"""Long lists whose scores crowd: ties, and spreads of many orders of magnitude, where places are not found by comparing the
entries of a score interval; lists just below and above that rule, in blocks of 256 and of 1024 threads."""

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from oracle import oracle

pytestmark = pytest.mark.gpu


def _rows(kind, n, d, rng):
    if kind == "equal":
        return np.tile(rng.integers(-9, 10, (1, d)), (n, 1)).astype(np.float32)
    if kind == "halves":  # half of the rows alike, the others apart
        x = rng.standard_normal((n, d)).astype(np.float32)
        x[rng.random(n) < 0.5] = 1.0
        return x
    if kind == "cluster":  # a few near rows, the others in one far cluster
        x = (100 + 1e-3 * rng.standard_normal((n, d))).astype(np.float32)
        x[rng.permutation(n)[:5]] = rng.standard_normal((5, d))
        return x
    return (rng.standard_normal((n, d)) * 10.0 ** rng.uniform(-12, 3, (n, 1))).astype(np.float32)


@pytest.mark.parametrize("kind", ["equal", "halves", "cluster", "wide"])
@pytest.mark.parametrize("n,k", [(900, 700), (1100, 1030), (5000, 2048), (9000, 2048), (40_000, 1500), (300_000, 700)])
def test_every_row_scored(n, k, kind):
    rng = np.random.default_rng(n + k)
    x, q = _rows(kind, n, 16, rng), rng.standard_normal((3, 16)).astype(np.float32)
    index = certex.Index(16)
    index.add(torch.from_numpy(x).cuda())
    index._test_mode(1)
    _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=k, return_scores=True)
    want_ids, want_scores = oracle.knn(x, q, k, "l2")
    assert np.array_equal(scores.cpu().numpy(), want_scores) and np.array_equal(ids.cpu().numpy(), want_ids)


@pytest.mark.parametrize("dtype", ["uint8", "float32"])
@pytest.mark.parametrize("k,copies", [(300, 3), (300, 290), (1000, 990), (2048, 40), (2048, 2040)])
def test_after_a_screen(k, copies, dtype):
    rng = np.random.default_rng(k + copies)
    n, d, nq = 140 * k, 32, 4
    x = rng.integers(0, 200, (n, d)).astype(dtype)
    for i in range(nq):  # every query has that many neighbours at one distance
        x[i * copies : (i + 1) * copies] = x[i * copies]
    q = x[np.arange(nq) * copies] + (1 if dtype == "uint8" else 0.5)
    order = rng.permutation(n)
    x, q = np.ascontiguousarray(x[order]), q.astype(dtype)
    index = certex.Index(d)
    index.add(torch.from_numpy(x).cuda())
    with certex.search_stats() as st:
        _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=k, return_scores=True)
    assert st.dense_queries == 0
    want_ids, want_scores = oracle.knn(x, q, k, "l2")
    assert np.array_equal(scores.cpu().numpy(), want_scores) and np.array_equal(ids.cpu().numpy(), want_ids)
