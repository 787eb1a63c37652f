"""The fp16 encoding of float rows at the edges of its launch: rows that fill no 16-byte piece, rows split over 8 lanes and
over a whole warp, and more rows than the blocks that are resident take in one turn. The rounding allowance of every
search comes from the largest norms of that pass, so the rows that decide them sit in the last turn."""

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float16"])
@pytest.mark.parametrize("n,d", [(3000, 1), (3001, 7), (40_001, 24), (3000, 127), (3000, 129), (12_000, 257), (2500, 2048)])
@pytest.mark.parametrize("metric", ["l2", "ip", "cosine"])
def test_rows_at_the_edges_of_the_encoding(n, d, dtype, metric):
    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d)).astype(dtype)
    x[-1] *= dtype == "float32" and 3.3 or np.float16(3)  # the largest norm belongs to the last row
    q = rng.standard_normal((21, d)).astype(dtype)
    index = certex.Index(d, metric=metric)
    index.add(torch.from_numpy(x).cuda())
    with certex.search_stats() as st:
        _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=5, return_scores=True)
    assert st.screen_passes == 1  # the screen and its thresholds ran
    want_ids, want_scores = oracle.knn(x, q, 5, metric)
    assert np.array_equal(ids.cpu().numpy(), want_ids) and np.array_equal(scores.cpu().numpy(), want_scores)
