"""Reading a solver back: whatever route a field's size takes (one pinned piece up
to 256 KiB for all fields together, the driver's copy, the ring of pinned chunks from
8 MiB per field), and with readers on several threads, the arrays are the uploaded
ones, bit for bit, in creation order although the slots are sorted by cell."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("position", "velocity", "affine_b", "elastic_f", "plastic_det")


def _solver(dim, n, seed):
    from mpm_snow_sim2d_b200 import Solver, _lib
    import ctypes as C
    p = _lib.MpmParams()
    _lib.load().mpm_params_default(C.byref(p), dim)
    p.dim, p.width, p.height, p.depth, p.border_margin = dim, 96, 80, 64 if dim == 3 else 0, 2
    rng = np.random.default_rng(seed)
    lo, hi = 8.0, np.array([88.0, 72.0, 56.0][:dim])
    pos = (lo + rng.random((n, dim)) * (hi - lo)).astype(np.float32)
    s = Solver(p, pos, np.full(n, 1e-3, np.float32))
    s.Step(1)  # sorts: slot order is no longer creation order
    want = {"position": pos,
            "velocity": rng.standard_normal((n, dim)).astype(np.float32),
            "affine_b": rng.standard_normal((n, dim, dim)).astype(np.float32),
            "elastic_f": rng.standard_normal((n, dim, dim)).astype(np.float32),
            "plastic_det": rng.random(n).astype(np.float32)}
    s.set_state(**want)
    return s, want


def _check(s, want):
    assert np.array_equal(s.GetParticlePositions(), want["position"])
    got = s.get_state()
    for f in FIELDS:
        assert np.array_equal(getattr(got, f), want[f]), f


# positions: 256 KiB and one particle more; 8 MiB and one more; several rounds of the
# ring with a ragged last chunk. Whole states: 2520 x 104 bytes (3D) just fit 256 KiB.
@pytest.mark.parametrize("dim,n", [(2, 1), (3, 2520), (3, 2521), (2, 32768), (2, 32769), (2, 1048576), (2, 1048577),
                                   (2, 2359301), (3, 1500001)])
def test_fields_come_back_whole(gpu_lib, dim, n):
    s, want = _solver(dim, n, n)
    with s:
        _check(s, want)


def test_readers_on_several_threads(gpu_lib):
    pairs = [_solver(2, n, n) for n in (700, 50021, 1200007, 2400003)]
    bad = []

    def reader(s, want):
        try:
            for _ in range(3):
                _check(s, want)
        except BaseException as e:  # noqa: BLE001 - reported by the main thread
            bad.append(e)

    threads = [threading.Thread(target=reader, args=p) for p in pairs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, _ in pairs:
        s.close()
    assert not bad, bad


@pytest.mark.parametrize("n", [1000, 1048577, 2359301])
def test_read_into_pinned_memory(gpu_lib, n):
    import ctypes as C
    import torch
    s, want = _solver(2, n, n)
    with s:
        out = torch.full((n, 2), -1.0, dtype=torch.float32, pin_memory=True)
        st = gpu_lib.mpm_get_positions(s._h, C.cast(out.data_ptr(), C.POINTER(C.c_float)), out.numel())
        assert st == 0 and np.array_equal(out.numpy(), want["position"])
