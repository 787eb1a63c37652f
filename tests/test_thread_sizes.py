"""Searches of different sizes from several threads at once: the kernels' shared memory depends on the number of queries, on k
and on the length of a row, and what one thread asks for must not take from another."""

import threading

import pytest
import torch

import libcertex_b200 as certex

pytestmark = pytest.mark.gpu


def _rows(n, d, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dtype == torch.uint8:
        return torch.randint(0, 256, (n, d), generator=g, device="cuda", dtype=torch.uint8)
    return torch.randn((n, d), generator=g, device="cuda").to(dtype)


# (vectors, coordinates, type, queries, k) of every thread
@pytest.mark.parametrize("calls", [
    [(60_000, 128, torch.uint8, 1, 10), (60_000, 128, torch.uint8, 300, 10), (60_000, 128, torch.uint8, 900, 10)],  # panels of 1, 3, 7 tiles
    [(3000, 32, torch.uint8, 2, 1100), (3000, 32, torch.uint8, 2, 1500), (3000, 32, torch.uint8, 2, 2048)],        # every row scored
    [(20_000, 16, torch.float32, 2, 1100), (20_000, 16, torch.float32, 2, 1700), (20_000, 16, torch.float32, 2, 2048)],  # the same, long rows
    [(30_000, 40, torch.float32, 9, 10), (30_000, 90, torch.float32, 9, 10), (30_000, 128, torch.float32, 9, 10)],  # rows scored in one launch
], ids=["panels", "selection", "wide selection", "rows"])
def test_threads_with_calls_of_different_sizes(calls):
    indexes, failures = {}, []
    for n, d, dtype, _, _ in calls:
        if (n, d) not in indexes:
            indexes[n, d] = certex.Index(d)
            indexes[n, d].add(_rows(n, d, dtype, 1))

    def work(i):
        n, d, dtype, nq, k = calls[i]
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                q = _rows(nq, d, dtype, 2 + i)
                want = indexes[n, d].search(q, k=k)
                for _ in range(400):
                    got = indexes[n, d].search(q, k=k)
                assert all(torch.equal(a, b) for a, b in zip(got, want))
        except Exception as e:  # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]
