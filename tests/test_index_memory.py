"""Indexes that come and go share a pool of device memory: answers stay right when the memory of a dropped index, with a search
of it still on the device, is handed to the next, on several streams and threads, and what no index uses is given back."""

import threading

import numpy as np
import pytest
import torch

import libcertex_b200 as certex
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,labels", [(300, 16, False), (30_000, 48, False), (30_000, 48, True)])
def test_indexes_made_and_dropped_on_several_threads(n, d, labels):
    failures = []

    def work(seed):
        try:
            rng = np.random.default_rng(seed)
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(6):
                    x, q = (rng.standard_normal((m, d)).astype(np.float32) for m in (n, 9))
                    lab = rng.integers(0, 2, n).astype(np.int32) if labels else None
                    ql = rng.integers(0, 2, 9).astype(np.int32) if labels else None
                    index = certex.Index(d)
                    index.add(torch.from_numpy(x).cuda(), labels=lab)
                    out = index.search(torch.from_numpy(q).cuda(), k=4, labels=ql, return_scores=True)
                    del index  # its last search may still run
                    ids, scores = oracle.knn(x, q, 4, "l2", row_labels=lab, query_labels=ql)
                    assert np.array_equal(out[1].cpu().numpy(), ids) and np.array_equal(out[2].cpu().numpy(), scores)
        except Exception as e:  # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]


def test_memory_of_a_large_index_goes_back():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    x = torch.zeros((1 << 20, 1024), dtype=torch.float32, device="cuda")  # 4 GiB of vectors, 2 GiB of codes
    before = torch.cuda.mem_get_info()[0]
    index = certex.Index(1024)
    index.add(x)
    assert before - torch.cuda.mem_get_info()[0] > 5 << 30
    del index
    torch.cuda.synchronize()
    certex.Index(8).add(torch.zeros((16, 8), device="cuda"))
    torch.cuda.synchronize()
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept < 4 << 30, f"{kept} bytes are still held"
