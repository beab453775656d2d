"""Workspaces on a nearly full GPU, without one: the smaller size is asked for
where the larger cannot be had."""
import pytest
import torch

from bitwise_spgemm_gb300 import ops


def _full(limit):
    real = torch.empty

    def empty(n, **kw):
        if n > limit:
            raise torch.OutOfMemoryError("full")
        return real(n, dtype=kw["dtype"])
    return empty


@pytest.mark.parametrize("limit,n,least,want", [(100, 50, 10, 50), (20, 50, 10, 10), (20, 50, 0, None),
                                                (100, 0, 0, None), (9, 50, 10, MemoryError), (9, 50, 50, MemoryError)])
def test_scratch_takes_the_largest_that_fits(limit, n, least, want, monkeypatch):
    monkeypatch.setattr(ops.torch, "empty", _full(limit))
    if want is MemoryError:
        with pytest.raises(torch.OutOfMemoryError):
            ops._scratch("cpu", n, lambda: least)
    else:
        got = ops._scratch("cpu", n, lambda: least)
        assert (got.numel() if got is not None else None) == want
