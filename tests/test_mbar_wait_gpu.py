"""The bounded wait of the GEMM pipelines on a shared-memory barrier."""

import pytest
import torch

from pplx_kernels_b200.ops import _ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit_ms", [0.5, 3.0, 40.0, 200.0])
def test_the_limit_is_a_time(limit_ms):
    """A barrier that others arrive on but that never completes: the wait gives up after the limit,
    not before it, and later by a few sleeps of the barrier unit at most (up to a millisecond each)."""
    ok, ns = _ops.mbar_wait_probe(torch.zeros(1, device="cuda"), limit_ms)
    assert ok == 0
    # (20 ms: time slices that other work on the GPU may take.)
    assert limit_ms * 1e6 <= ns <= limit_ms * 1e6 + 20e6
    assert float(torch.ones(4, device="cuda").sum()) == 4.0  # the context is still usable
