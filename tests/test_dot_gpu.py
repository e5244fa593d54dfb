"""The ordered dot product (cmg_op_dot, k_box_dot) on box sizes around its chunk of 1024 cells: equal to adding every
box's products one by one, k, j, i with i fastest, and the boxes in layout order."""
import ctypes

import numpy as np
import pytest


def ordered_dot(boxes, x, y):
    total, pos = 0.0, 0
    for b in boxes:
        n = [b[d + 3] - b[d] + 1 for d in range(3)]
        g = (n[2] + 2, n[1] + 2, n[0] + 2)
        size = g[0] * g[1] * g[2]
        p = (x[pos:pos + size] * y[pos:pos + size]).reshape(g)[1:-1, 1:-1, 1:-1].ravel()
        total += np.add.accumulate(np.concatenate([[0.0], p]))[-1]
        pos += size
    return total


@pytest.mark.gpu
@pytest.mark.parametrize("n0,cuts", [(4, (2,)), (16, (8,)), (20, (10,)), (24, (8,)), (32, (8, 24)), (36, (16,)), (64, (32,))])
def test_dot_adds_in_order(cmg, n0, cuts):
    e = [0, *cuts, n0]  # the same cuts in every direction
    r = range(len(e) - 1)
    boxes = [(e[i], e[j], e[k], e[i + 1] - 1, e[j + 1] - 1, e[k + 1] - 1) for k in r for j in r for i in r]
    h = cmg.Hierarchy(n0, [boxes])
    order = h.boxes(0)
    size = sum((b[3] - b[0] + 3) * (b[4] - b[1] + 3) * (b[5] - b[2] + 3) for b in order)
    rng = np.random.default_rng(n0)
    x, y = rng.standard_normal(size), rng.standard_normal(size) * 10.0 ** rng.integers(-8, 8, size)
    out = ctypes.c_double()
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    cmg._check(cmg.lib().cmg_op_dot(h.h, 0, ptr(x), ptr(y), ctypes.byref(out)))
    assert out.value == ordered_dot(order, x, y)
    h.close()
