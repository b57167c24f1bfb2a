"""What the target order is given and gives on (host side, no launch)."""
import ctypes
import importlib
import types

import numpy as np
import pytest
import torch

from sseqs_b200 import select

sw = importlib.import_module("sseqs_b200.sw")


@pytest.fixture
def given(monkeypatch):
    """The target numbers that the length sort would read, as it reads them."""
    seen = []

    def sort(delim, idx, g0, n, *rest):
        seen.append(np.ctypeslib.as_array(ctypes.cast(idx, ctypes.POINTER(ctypes.c_int32)),
                                          (n,)).tolist())
        return 0

    L = types.SimpleNamespace(sseqs_length_order_workspace_bytes=lambda: 16,
                              sseqs_length_order=sort)
    monkeypatch.setattr(select, "lib", lambda: L)
    monkeypatch.setattr(select, "stream_ptr", lambda: 0)
    return seen


def test_targets_of_any_integer_type_and_stride(given):
    delim = torch.arange(100, dtype=torch.int32)
    want = [7, 3, 90, 41, 5]
    wide = torch.tensor(want).repeat_interleave(2)
    for idx in (torch.tensor(want, dtype=torch.int32), torch.tensor(want), wide[::2],
                wide.to(torch.int32)[::2]):
        select.length_order(delim, 5, good_idx=idx)
    assert given == [want] * 4


def test_too_few_targets_are_refused(given):
    delim = torch.arange(100, dtype=torch.int32)
    with pytest.raises(ValueError):
        select.length_order(delim, 6, good_idx=torch.arange(5))
    with pytest.raises(ValueError):
        select.length_order(delim, 5, good_idx=torch.arange(5, device="meta"))
    assert given == []


@pytest.mark.parametrize("order", [torch.arange(4, dtype=torch.int32), torch.arange(4)])
def test_an_order_in_host_memory_is_refused(order):
    with pytest.raises(ValueError):
        sw._order(order, 4)
