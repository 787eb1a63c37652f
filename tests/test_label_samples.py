"""The tiles of a label that give its queries' thresholds: how many they are, and how many values a query then has, from the
smallest labels to the largest, and searches of labels on both sides of where the rule changes."""

import ctypes

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from libcertex_b200 import _lib
from oracle import oracle


def _sample(k_blocks, rows, k):
    out = (ctypes.c_int64 * 3)()
    _lib.check(_lib.lib().certexB200LabelSample(k_blocks, rows, k, out))
    return tuple(out)


@pytest.mark.parametrize("k_blocks", [1, 2, 3, 12, 32])
@pytest.mark.parametrize("k", [1, 10, 100, 400, 1000, 2048])
def test_a_sample_is_bounded(k_blocks, k):
    for rows in sorted({32 * k, 128 * k, 15_600, 65_536, 262_144, 263_000, 400_000, 1_000_000, 4_000_000, 100_000_000}):
        if rows < 32 * k:  # no routed pass
            continue
        group, step, tiles = _sample(k_blocks, rows, k)
        nt = -(-rows // 256)
        assert (tiles - 1) * step < nt  # inside the label
        assert tiles * (256 // group) >= min(2 * k, rows // group)  # values enough for a threshold
        # 1024 tiles, a sixteenth of the label, what k asks for; a whole number of steps may take up to twice that
        need = min(nt, max(1024, -(-nt // 16), k, -(-24 * k * nt // (10 * max(2048, 2 * k)))))
        assert tiles <= 2 * need
        # as many values a query as those have in groups of 64, or chains where these are no more than 4096 or nothing else will do
        assert tiles * (256 // group) <= 8 * need if group == 64 else rows < 128 * k or tiles * 16 <= 4096


def test_long_rows_take_a_quarter_of_a_small_label():
    assert _sample(12, 15_600, 100) == (16, 3, 21)
    assert _sample(1, 15_600, 100) == (64, 1, 61)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,metric,d", [("float16", "l2", 130), ("uint8", "ip", 300)])
def test_labels_on_both_sides_of_the_rule(d, dtype, metric):
    rng = np.random.default_rng(d)
    sizes = [9_000, 200_000, 300_000, 1_100_000]
    lab = rng.permutation(np.repeat(np.arange(len(sizes), dtype=np.int32), sizes))
    x = rng.integers(0, 20, (len(lab), d)).astype(dtype)
    q = rng.integers(0, 20, (8, d)).astype(dtype)
    ql = np.arange(8, dtype=np.int32) % len(sizes)
    index = certex.Index(d, metric=metric)
    index.add(torch.from_numpy(x).cuda(), labels=lab)
    for k in (1, 10, 60):
        with certex.search_stats() as st:
            _, ids, scores = index.search(torch.from_numpy(q).cuda(), k=k, labels=torch.from_numpy(ql).cuda(), return_scores=True)
        assert st.routed_queries >= 8 and st.dense_queries == 0
        assert st.verified <= 8 * 2048
        want_ids, want_scores = oracle.knn(x, q, k, metric, row_labels=lab, query_labels=ql)
        assert np.array_equal(ids.cpu().numpy(), want_ids) and np.array_equal(scores.cpu().numpy(), want_scores)
