"""Positions large enough to go through the ring of pinned chunks at the first read into fresh memory, then again into the same
memory (the driver's copy), and from two threads at once, of which one finds the ring taken."""
import threading

import numpy as np
import pytest

from test_gpu_readback import _solver

pytestmark = pytest.mark.gpu


def test_large_positions(gpu_lib):
    from mpm_snow_sim2d_b200._lib import fptr
    pairs = [_solver(2, 5500003 + k, k) for k in range(2)]
    bad = []

    def reader(s, want, fresh):
        try:
            for k in range(4):
                if fresh or k == 0:
                    out = np.empty_like(want["position"])
                if not fresh:
                    out.fill(-1.0)
                assert s._lib.mpm_get_positions(s._h, fptr(out), out.size) == 0
                assert np.array_equal(out, want["position"])
        except BaseException as e:  # noqa: BLE001 - reported by the main thread
            bad.append(e)

    reader(*pairs[0], True)
    reader(*pairs[1], False)
    threads = [threading.Thread(target=reader, args=(*p, True)) for p in pairs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, _ in pairs:
        s.close()
    assert not bad, bad
