"""solve_symmetric on host arrays keeps an idle factor with the analysis: calls
in a row, after a refused system and from several threads at once give the
bits of a first call on a fresh analysis."""
import threading

import numpy as np
import pytest

import aphi_b200 as ab

pytestmark = pytest.mark.gpu


def test_kept_factor_gives_a_fresh_calls_bits(cuda):
    w = ab.Workload.cylinder(6)
    perm = ab.amd_ordering(w.row_ptr, w.col_idx)
    asm = ab.Assembly(ab.workload_arrays(w))
    systems = [asm.refill_host(2 * np.pi * hz) for hz in (50.0, 400.0, 3.0e3)]
    fresh = []
    for v, b in systems:
        ok, x, _ = ab.solve_symmetric(ab.Analysis(w.row_ptr, w.col_idx, perm), v, b)
        assert ok
        fresh.append(x)
    an = ab.Analysis(w.row_ptr, w.col_idx, perm)
    for k in (0, 1, 0, 2):
        ok, x, _ = ab.solve_symmetric(an, *systems[k])
        assert ok and np.array_equal(x, fresh[k])
    ok, _, report = ab.solve_symmetric(an, np.zeros_like(systems[0][0]), systems[0][1])
    assert not ok and report["columns_done"] == 1
    ok, x, _ = ab.solve_symmetric(an, *systems[0])
    assert ok and np.array_equal(x, fresh[0])
    wrong = []

    def work(k):
        for _ in range(4):
            ok, x, _ = ab.solve_symmetric(an, *systems[k])
            if not ok or not np.array_equal(x, fresh[k]):
                wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
