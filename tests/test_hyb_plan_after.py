"""The HYB work lists where some warps have block rows to do first (hbicg__hyb_plan_after, host code): the greedy rule
from the given loads, at no items, one list, more lists than items, equal and very uneven loads."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.parametrize("ni,hnw,kind", [(0, 3, "uneven"), (7, 1, "uneven"), (5, 16, "equal"), (400, 24, "uneven"),
                                         (400, 24, "falling"), (900, 33, "none")])
def test_lists_start_from_the_given_loads(lib, ni, hnw, kind):
    rng = np.random.default_rng(ni + hnw)
    cost = rng.integers(1, 40, ni).astype(np.uint32)
    base = {"equal": np.full(hnw, 9), "uneven": rng.integers(0, 500, hnw), "falling": np.arange(hnw)[::-1] * 7,
            "none": np.zeros(hnw)}[kind].astype(np.uint32)
    f = lib.hbicg__hyb_plan_after
    f.restype = C.c_int
    f.argtypes = [C.c_size_t, C.c_void_p, C.c_void_p, C.c_uint, C.c_void_p, C.c_void_p]
    hwbeg, hitem = np.zeros(hnw + 1, dtype=np.uint32), np.zeros(max(ni, 1), dtype=np.uint32)
    assert f(ni, cost.ctypes.data, None if kind == "none" else base.ctypes.data, hnw, hwbeg.ctypes.data,
             hitem.ctypes.data) == 0
    load, lists = [int(b) for b in base], [[] for _ in range(hnw)]
    for i in sorted(range(ni), key=lambda i: (-int(cost[i]), i)):
        w = min(range(hnw), key=lambda w: (load[w], w))
        lists[w].append(i)
        load[w] += int(cost[i])
    assert [list(hitem[hwbeg[w]:hwbeg[w + 1]]) for w in range(hnw)] == lists
