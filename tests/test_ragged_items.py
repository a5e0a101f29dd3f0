"""The item table that RaggedBatch.run hands to the library: whatever has five
fields that int() takes, as numbers, arrays or tensors, each field's low 32
bits.  No GPU: the library call is replaced."""
import ctypes as C

import numpy as np
import pytest
import torch


class _OnDevice:
    """Like a scalar tensor in device memory: int() works, numpy's conversion does not."""

    def __init__(self, x):
        self.x = x

    def __int__(self):
        return self.x

    def __array__(self, *args, **kwargs):
        raise TypeError("can't convert a device tensor to numpy")


def _table(nwg, monkeypatch, items):
    batch = nwg.RaggedBatch.__new__(nwg.RaggedBatch)
    batch.h, batch.n, batch.num_graphs = None, np.array([4, 6], np.uint64), 2
    seen = []

    class Lib:
        @staticmethod
        def nwg_ragged_bfs(h, k, table, *rest):
            address = table if isinstance(table, int) else C.addressof(table)
            seen.append(np.ctypeslib.as_array((C.c_uint32 * (5 * k)).from_address(address)).reshape(k, 5).tolist() if k else [])
            return 0

    monkeypatch.setattr(nwg, "lib", Lib)
    batch.run(items, parents_dev=4096)
    return seen[0]


ITEM = (1, 3, 15, 18, 32)
FORMS = {
    "tuples": [ITEM, (0, 2, 15, 18, 64)],
    "lists": [list(ITEM)],
    "array": np.array([ITEM, ITEM], np.uint32),
    "numpy scalars": [(np.uint32(1), np.int64(3), np.int32(15), 18, np.uint8(32))],
    "floats": [(1, 3.9, 15.0, 18.0, 32.0)],
    "tensors": [tuple(torch.tensor(x) for x in ITEM)],
    "device tensors": [(1, _OnDevice(3), 15, 18, 32)],
    "one-element arrays": [(1, np.array([3]), 15, 18, 32)],
    "one-element tensors": [(1, torch.tensor([3]), 15, 18, 32)],
    "text": [(1, "3", "15", "18", "32")],
    "negative": [(-1, -2, -15, -18, 32)],
    "past 32 bits": [(1, (1 << 40) + 3, 15, 18, 32)],
    "past 64 bits": [(1, (1 << 70) + 3, 15, 18, 32)],
    "none": [],
}


@pytest.mark.filterwarnings("ignore:Conversion of an array")
@pytest.mark.parametrize("form", sorted(FORMS))
def test_every_form_of_item(nwg, monkeypatch, form):
    items = FORMS[form]
    want = [[int(x) & 0xFFFFFFFF for x in it] for it in items]
    assert _table(nwg, monkeypatch, items) == want


@pytest.mark.parametrize("items", [[(1, 3, 15, 18)], [(1, 3, 15, 18, 32, 0)], [(1, [3], 15, 18, 32)], [([1], [3], [15], [18], [32])],
                                   [(1, None, 15, 18, 32)], [(1, float("nan"), 15, 18, 32)], [1, 2, 3, 4, 5],
                                   [(1.0, 3, 15, 18, 32)], [("1", 3, 15, 18, 32)]])
def test_what_is_no_item(nwg, monkeypatch, items):
    with pytest.raises((TypeError, ValueError, IndexError)):
        _table(nwg, monkeypatch, items)
