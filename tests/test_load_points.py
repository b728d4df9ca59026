"""Loading field points one call at a time takes time in proportion to their
number (host only: nothing is uploaded before render_cuda)."""
import ctypes as C
import time

import numpy as np


def test_single_point_loads_are_not_quadratic(api):
    L = api.lib()
    p = np.zeros(3, np.float32)
    ptr = p.ctypes.data_as(C.POINTER(C.c_float))
    api.TearDownCuda()
    took = []
    try:
        for n in (20000, 80000):
            t = time.perf_counter()
            for _ in range(n):
                L.load_field_points(ptr, 1)
            took.append(time.perf_counter() - t)
            api._check()
            api.TearDownCuda()
    finally:
        api.TearDownCuda()
    print("20,000: %.3f s, 80,000: %.3f s" % tuple(took))
    # four times as many: 4 when in proportion, about 28 when every call copies
    # all points; 0.2 s for a busy machine
    assert took[1] < 10.0 * took[0] + 0.2
