"""A batch whose grids do not fit the device's free memory together: created all the same, and every scene as it is in a batch that
has the memory, bitwise, through steps, uploads, time stamps, configuration and the trial."""
import numpy as np
import pytest

from test_gpu_batch import _equal

pytestmark = pytest.mark.gpu


def _scenes(k, n):
    """k scenes of n particles each on grids of 255 x 255 nodes and a few others."""
    from mpm_snow_sim2d_b200 import scenes
    base = scenes.batch_scene_2d(0)
    out = []
    for i in range(k):
        w = 254 - 5 * (i % 3)
        rng = np.random.default_rng(i)
        pos = (w * (0.3 + 0.4 * rng.random((n + i % 5, 2)))).astype(np.float32)
        m = pos.shape[0]
        out.append(base.with_(width=w, height=w, position=pos, velocity=(5.0 * rng.standard_normal((m, 2))).astype(np.float32),
                              volume=np.full(m, base.volume[0], np.float32), mass=np.full(m, base.mass[0], np.float32)))
    return out


def _run(b, picked, scs):
    b.set_config(sort_period=5)
    b.step(7)
    st = b.get_state(picked[1])
    b.set_state(picked[1], velocity=-st.velocity)
    b.step(3)
    cfg, ms = b.tune(2)
    assert cfg == b.config and cfg["sort_period"] == 5 and ms > 0
    b.step(4)
    t = b.step_times()
    assert t.shape == (len(scs), 5) and np.all(t > 0) and np.all(np.diff(t.astype(np.int64), axis=1) >= 0)
    return [(b.get_state(s), b.positions(s), b.status(s)) for s in picked]


def test_grids_larger_than_free_memory(gpu_lib):
    import torch
    from mpm_snow_sim2d_b200._lib import MpmError
    from mpm_snow_sim2d_b200.batch import Batch
    k, n = 700, 40
    scs = _scenes(k, n)
    picked = [0, 1, 349, 350, k - 1]
    grids = sum((s.width + 1) * (s.height + 1) for s in scs) * 48
    with Batch(scs) as b:
        want = _run(b, picked, scs)
        assert b.total_particles == sum(s.count for s in scs)
    torch.cuda.empty_cache()
    left = grids // 3
    hold = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        with Batch(scs) as b:
            assert b.total_particles == sum(s.count for s in scs)
            got = _run(b, picked, scs)
            with pytest.raises(MpmError) as e:
                b.set_config(max_cluster=1)  # the grids of all parts are checked
            assert e.value.status == 11 and b.config["max_cluster"] == 8
            with torch.cuda.stream(torch.cuda.Stream()) as _:
                b.set_stream(torch.cuda.current_stream().cuda_stream)
                b.step(1)
                b.set_stream(None)
    finally:
        del hold
        torch.cuda.empty_cache()
    for (a, x, f), (c, y, g) in zip(want, got):
        assert _equal(a, c) and np.array_equal(x, y) and f == g
