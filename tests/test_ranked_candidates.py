"""The candidates of a screen are ranked by the products it leaves before any is scored exactly. Cases where the ranking is
tight or worthless: many equal rows around the k-th place, chains of 16 rows that are kept whole, rows removed or filtered out
inside kept chains, and lists on both sides of the size that one warp ranks."""

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from oracle import oracle

pytestmark = pytest.mark.gpu


def _rows(kind, n, d, rng):
    if kind == "distinct":
        x = rng.integers(-60, 60, (n, d))
    elif kind == "repeated":  # every row 40 times: ties at every rank, whole chains of equal rows
        x = np.repeat(rng.integers(-60, 60, (n // 40 + 1, d)), 40, axis=0)[:n]
        x = x[rng.permutation(n)]
    else:  # one cluster far from the rest: the products hardly differ within it
        x = rng.integers(-3, 4, (n, d)) + np.where(rng.random((n, 1)) < 0.1, 90, -90)
    return x


@pytest.mark.parametrize("dtype", ["int8", "float32"])
@pytest.mark.parametrize("metric", ["l2", "ip"])
@pytest.mark.parametrize("kind", ["distinct", "repeated", "cluster"])
@pytest.mark.parametrize("k", [1, 31, 100, 257, 1000])
def test_ranked_candidates_are_the_exact_ones(k, kind, metric, dtype):
    rng = np.random.default_rng(k)
    n, d, nq = max(20_000, 140 * k), 40, 37
    x = _rows(kind, n, d, rng).astype(dtype)
    q = _rows(kind, nq, d, rng).astype(dtype)
    index = certex.Index(d, metric=metric)
    index.add(torch.from_numpy(x).cuda())
    gone = rng.permutation(n)[: n // 100]
    index.remove(torch.from_numpy(gone).cuda())
    keep = rng.random(n) < 0.5
    for mask in (None, keep):
        alive = np.ones(n, dtype=bool)
        alive[gone] = False
        if mask is not None:
            alive &= mask
        _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=k, return_scores=True,
                                      filter=None if mask is None else torch.from_numpy(mask).cuda())
        left = np.nonzero(alive)[0]
        want_ids, want_scores = oracle.knn(x[left], q, k, metric)
        assert np.array_equal(scores.cpu().numpy(), want_scores)
        assert np.array_equal(ids.cpu().numpy(), left[want_ids])
