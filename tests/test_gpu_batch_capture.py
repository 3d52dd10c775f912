"""A batch's steps captured into a CUDA graph of the caller's: replayed any number of times, with uploads and plain calls in between,
every scene is bitwise what plain calls make of it."""
import numpy as np
import pytest

from test_gpu_batch import _equal, _mixed_scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,period", [(1, 16), (3, 16), (7, 7), (40, 8), (65, 16)])
def test_captured_steps(gpu_lib, steps, period):
    import torch
    from mpm_snow_sim2d_b200.batch import Batch
    scs = _mixed_scenes(k=4, steps=200)

    def reset(b):
        st = b.get_state(1)
        b.set_state(1, position=st.position, velocity=-2.0 * st.velocity)

    with Batch(scs) as b:
        b.step(2 + 2 * steps)
        b.step(3 * steps)
        reset(b)
        b.step(steps)
        b.step(steps)
        b.step(5)
        b.step(3 * steps)
        b.step(4 + 4 * steps)
        want = [b.get_state(k) for k in range(4)]
    with Batch(scs) as b:
        b.set_config(sort_period=period)
        b.step(2 + 2 * steps)  # also makes room for the time stamps of a call
        stream = torch.cuda.Stream()
        b.set_stream(stream.cuda_stream)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            g.capture_begin(capture_error_mode="relaxed")
            b.step(steps)
            g.capture_end()
            for _ in range(3):
                g.replay()
        reset(b)
        with torch.cuda.stream(stream):
            g.replay()
            g.replay()
        t = b.step_times()
        assert t.shape == (4, steps + 1) and np.all(t > 0) and np.all(np.diff(t.astype(np.int64), axis=1) >= 0)
        b.step(5)  # sorts once for some periods
        g2 = torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            g.replay()
            g2.capture_begin(capture_error_mode="relaxed")
            b.step(2 * steps)
            g2.capture_end()
            g2.replay()
        b.step(4 + 3 * steps)  # more time stamps than there was room for
        with torch.cuda.stream(stream):
            g.replay()
        stream.synchronize()
        got = [b.get_state(k) for k in range(4)]
        b.set_stream(None)
        del g, g2
    for k in range(4):
        assert _equal(got[k], want[k]), k
