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


def test_memory_of_a_dropped_index_goes_back():
    keep = 1 << 30  # what the pool of the index arrays may hold on to
    # arrays of up to 4 GiB, and eight indexes whose arrays all come from the pool, more than it keeps
    for n, d in [(1 << 20, 1024), (220_000, 256)]:
        x = torch.zeros((n, d), dtype=torch.float32, device="cuda")

        def make(count):
            out = [certex.Index(d) for _ in range(count)]
            for index in out:
                index.add(x)
            return out

        count = 1 if n == 1 << 20 else 8
        held = make(count)  # what a first build takes besides (kernels, scratch memory) stays
        del held
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        held = make(count)
        arrays = count * n * d * (4 + 2)
        assert before - torch.cuda.mem_get_info()[0] > arrays - keep
        del held
        after = torch.cuda.mem_get_info()[0]  # with nothing in between
        assert before - after < keep, f"{before - after} bytes are still held"
        del x
        torch.cuda.empty_cache()


def test_a_large_index_from_several_threads():
    """Arrays above the size that comes from the pool, made and dropped beside small ones."""
    failures = []

    def work(n, d, turns):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                x = torch.arange(n, device="cuda", dtype=torch.float32)[:, None].expand(n, d).contiguous()
                for _ in range(turns):
                    index = certex.Index(d, capacity=n)
                    index.add(x[: n // 2])
                    index.add(x[n // 2 :])
                    _, ids = index.search(x[n - 3 :], k=2)
                    del index
                    assert ids[:, 0].tolist() == [n - 3, n - 2, n - 1]
        except Exception as e:  # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=work, args=a) for a in [(600_000, 128, 4), (600_000, 256, 4), (3000, 16, 60)]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]
