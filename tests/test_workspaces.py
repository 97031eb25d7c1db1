"""Scratch memory of the ops: whose it is, checked without a GPU."""
import pytest
import torch

from pippy_b200.ops import _lib
from pippy_b200.ops import functional as pf

pytestmark = pytest.mark.skipif(not _lib.available(), reason="the CUDA library is not built")


def test_norm_backward_calls_share_no_partial_sums(monkeypatch):
    """Two calls of one width may be in flight on two streams, or one of them inside a graph."""
    monkeypatch.setattr(pf, "sm_count", lambda: 148)
    pf._ensure_restypes()
    a, b = (pf._norm_scratch(768, torch.device("cpu")) for _ in range(2))
    assert a.numel() == b.numel() == 148 * 2 * 2 * 768
    assert a.untyped_storage().data_ptr() != b.untyped_storage().data_ptr()
