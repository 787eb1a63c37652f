"""What search_stats says about the kernels that a search launched."""

import pytest
import torch

import libcertex_b200 as certex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,metric,k,launches", [("uint8", "l2", 256, 7), ("uint8", "l2", 257, 9), ("float32", "ip", 10, 8),
                                                     ("float32", "ip", 300, 10)])
def test_launches_of_a_search_are_counted(dtype, metric, k, launches):
    """The queries' codes (and norms), the anchors' e, two passes and the thresholds, the verification in one or three, the answers."""
    x = torch.randint(0, 100, (60_000, 64), device="cuda").to(getattr(torch, dtype))
    index = certex.Index(64, metric=metric)
    index.add(x)
    with certex.search_stats() as st:
        index.search(x[:5], k=k)
    assert st.dense_queries == 0 and st.rescreened == 0
    assert st.launches == launches
