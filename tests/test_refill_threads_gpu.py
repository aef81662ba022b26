"""Refills of several meshes from several threads at once, of one and of 64
frequencies: a kernel's shared-memory limit belongs to the kernel, not to the
call, so no call may lower it under another one's launch. Both instances of the
fill (one and four tets a warp), bits compared with the calls made alone."""
import threading

import numpy as np
import pytest
import torch

import aphi_b200 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(5, 6, 7, 8), (12, 13, 14, 15)], ids=["one_tet_a_warp", "four_tets_a_warp"])
def test_concurrent_refills_of_one_and_many_frequencies(cells, cuda):
    om = 2 * np.pi * np.geomspace(50.0, 1.0e6, 64)
    calls = []
    for k, nf in zip(cells, (64, 1, 1, 1)):
        asm = ab.Assembly(ab.workload_arrays(ab.Workload.cylinder(k)))
        alone = tuple(t.cpu().numpy() for t in asm.refill(om[:nf]))
        out = tuple(torch.empty_like(torch.from_numpy(t), device="cuda") for t in alone)
        calls.append((asm, om[:nf].copy(), out, alone, torch.cuda.Stream()))
    torch.cuda.synchronize()
    wrong, go = [], threading.Barrier(len(calls))

    def work(asm, omegas, out, alone, stream):
        # The C entry point itself: Python's own work between two calls would
        # keep the threads out of each other's way.
        refill = ab.lib().aphi_refill_batch
        args = (asm._h, omegas.size, ab._ptr(omegas, ab.C.c_double), ab.COND_ROW_SCALED, ab.dptr(out[0]),
                ab.dptr(out[1]), ab.stream_ptr(stream))
        go.wait()
        for _ in range(2000 if omegas.size == 1 else 500):
            if refill(*args) != 0:
                wrong.append(ab.lib().aphi_last_error().decode())
                return
        stream.synchronize()
        if not all(np.array_equal(g.cpu().numpy(), x) for g, x in zip(out, alone)):
            wrong.append("bits differ")

    threads = [threading.Thread(target=work, args=c) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
