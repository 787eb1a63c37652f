"""Batches that fill no query tile, with the next batch's queries behind them: what lies there must leave no trace."""

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 100, 129])
@pytest.mark.parametrize("d,metric", [(40, "ip"), (100, "l2"), (200, "cosine")])
def test_a_query_beyond_the_fp16_range_in_the_next_batch(d, metric, batch):
    """Its code is infinite, and so are its products, in the lanes behind the batch before it."""
    rng = np.random.default_rng(d + batch)
    n, k = 20_000, 5
    nq = 2 * batch + 3
    x = rng.standard_normal((n, d)).astype(np.float32)
    q = rng.standard_normal((nq, d)).astype(np.float32)
    q[batch, 0], q[batch, 1] = 1e6, -1e6
    q[2 * batch] = 1e5
    index = certex.Index(d, metric=metric)
    index.add(torch.from_numpy(x).cuda())
    with certex.search_stats() as st:
        _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=k, batch=batch, return_scores=True)
    assert st.screen_passes > 1 and st.dense_queries == nq  # screened, then answered without the screen
    want_ids, want_scores = oracle.knn(x, q, k, metric)
    assert np.array_equal(ids.cpu().numpy(), want_ids) and np.array_equal(scores.cpu().numpy(), want_scores)
    # and a batch whose followers are plain
    with certex.search_stats() as st:
        _, ids, scores = index.search(torch.from_numpy(np.ascontiguousarray(q[:batch])).cuda(), k=k, batch=batch, return_scores=True)
    assert st.dense_queries == 0
    assert np.array_equal(ids.cpu().numpy(), want_ids[:batch]) and np.array_equal(scores.cpu().numpy(), want_scores[:batch])
