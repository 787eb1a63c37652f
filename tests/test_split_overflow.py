"""Candidate lists that overflow where ranking, scoring and sorting are launches of their own (k > 256, and long float rows with
k > 32): a list that holds k rows gives a tighter threshold for a second screen, one that holds fewer sends its query to the
search without a screen."""

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from oracle import oracle

pytestmark = pytest.mark.gpu


# vectors, coordinates, k, anchor_stride, a list of more than k that the second pass fits in, and one of fewer than k
@pytest.mark.parametrize("n,d,k,stride,fits,fewer", [(120_000, 40, 300, 64, 700, 200), (20_000, 512, 40, 16, 100, 30),
                                                     (400_000, 24, 1500, 256, 2600, 1000)])
@pytest.mark.parametrize("dtype,metric", [("uint8", "l2"), ("int8", "ip"), ("float32", "l2"), ("float32", "ip"), ("float16", "cosine")])
def test_lists_that_overflow(dtype, metric, n, d, k, stride, fits, fewer):
    if d == 512 and dtype in ("uint8", "int8"):
        pytest.skip("rows of 8-bit vectors are never long")
    rng = np.random.default_rng(k)
    nq = 12
    lo = 0 if dtype == "uint8" else -100
    x = rng.integers(lo, 100, (n, d)).astype(dtype)
    q = rng.integers(lo, 100, (nq, d)).astype(dtype)
    index = certex.Index(d, metric=metric, anchor_stride=stride)
    index.add(torch.from_numpy(x).cuda())
    want_ids, want_scores = oracle.knn(x, q, k, metric)
    for cap in (fits, fewer):
        index._test_mode(2, cap=cap)
        with certex.search_stats() as st:
            _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=k, return_scores=True)
        assert np.array_equal(ids.cpu().numpy(), want_ids) and np.array_equal(scores.cpu().numpy(), want_scores)
        assert st.screen_passes == 2 and st.rescreened > 0
        assert st.dense_queries < st.rescreened if cap == fits else st.dense_queries > 0
