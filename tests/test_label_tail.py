"""Searches by labels while rows are newer than the label partition: those rows are screened one by one against the queries of
their label, beside the routed passes over the partition."""

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,metric", [("uint8", "l2"), ("int8", "ip"), ("float16", "ip"), ("float32", "l2"), ("float32", "cosine")])
@pytest.mark.parametrize("d", [1, 100, 300, 700])
@pytest.mark.parametrize("n_tail", [1, 17, 1500])
def test_rows_newer_than_the_partition(n_tail, d, dtype, metric):
    rng = np.random.default_rng(d + n_tail)
    n, nq, k = 16_000, 60, 9
    lo = 0 if dtype == "uint8" else -100
    x = rng.integers(lo, 100, (n + n_tail, d)).astype(dtype)
    q = rng.integers(lo, 100, (nq, d)).astype(dtype)
    lab = rng.integers(0, 5, n + n_tail).astype(np.int32)
    lab[n:][rng.random(n_tail) < 0.2] = 7  # a label that the partition does not know
    lab[:n][lab[:n] == 4] = 3
    lab[:40] = 4                           # and one with too few rows there for a screen
    ql = rng.integers(0, 9, nq).astype(np.int32)
    index = certex.Index(d, metric=metric, partition_labels="lazy")
    index.add(torch.from_numpy(x[:n]).cuda(), labels=lab[:n])
    index.add(torch.from_numpy(x[n:]).cuda(), labels=lab[n:])
    assert index.info()["n_partitioned"] == n
    gone = np.unique(rng.integers(n - 100, n + n_tail, 50))
    index.remove(torch.from_numpy(gone).cuda())
    with certex.search_stats() as st:
        _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=k, labels=torch.from_numpy(ql).cuda(), return_scores=True)
    assert st.routed_queries > 0
    keep = np.ones(n + n_tail, dtype=bool)
    keep[gone] = False
    want_ids, want_scores = oracle.knn(x, q, k, metric, keep_row=keep, row_labels=lab, query_labels=ql)
    assert np.array_equal(ids.cpu().numpy(), want_ids) and np.array_equal(scores.cpu().numpy(), want_scores)
