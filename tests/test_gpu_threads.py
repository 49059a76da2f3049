"""Contexts of several threads stepping at the same time, each launch of the one-launch
steps as large as such a launch gets: the bits of the same steps one context after the
other, and no wait gives up."""
import threading

import numpy as np
import pytest

import dg_b200

pytestmark = pytest.mark.gpu

XY = [1.0, 0.4, -0.3, 1.0, 2.0, 5.0, 4.5, 10.0, 9.0]


def cases():
    box = lambda n: dg_b200.periodic_box(n, (0.0, 0.0, 0.0), (10.0, 9.0, 10.0), rotate_seed=2)
    return [dg_b200.Case(box((8, 8, 9)), 3, gas_constant=1.0), dg_b200.Case(box((6, 7, 7)), 5, gas_constant=1.0),
            dg_b200.Case(box((10, 10, 11)), 1, gas_constant=1.0, precision="mixed_fp32"),
            dg_b200.Case(box((12, 12, 12)), 2, gas_constant=1.0),
            dg_b200.Case2D(dg_b200.periodic_box_2d((50, 45), (0.0, 0.0), (10.0, 9.0)), 4, flux="HLLC", gas_constant=1.0),
            dg_b200.Case2D(dg_b200.periodic_box_2d((20, 21), (0.0, 0.0), (10.0, 9.0)), 1, gas_constant=1.0)]


def test_contexts_of_several_threads():
    def work(case, out, i):
        try:
            case.project_ic("IsentropicVortexXY", XY)
            for _ in range(10):
                case.rk4(1e-4, 30)
                case.fe(1e-5, 7)
            out[i] = case.get_state()
        except Exception as e:
            out[i] = e

    alone, together = [None] * 6, [None] * 6
    for i, c in enumerate(cases()):
        work(c, alone, i)
    cs = cases()
    threads = [threading.Thread(target=work, args=(c, together, i)) for i, c in enumerate(cs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, (a, b) in enumerate(zip(alone, together)):
        assert not isinstance(a, Exception) and not isinstance(b, Exception), (i, a, b)
        assert np.array_equal(a, b), i
