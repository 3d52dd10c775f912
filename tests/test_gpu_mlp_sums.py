"""How the training kernel adds up a gradient: parts of 64 rows, each rounded alike wherever it falls in the batch,
added in FP32 within a CTA and in FP64 between CTAs. Parts come from gradients of 64 rows alone: with all counts
powers of two, the factor 1 / rows only moves the exponent, so that every rounding is the same."""
import numpy as np
import pytest

from test_gpu_mlp import synthetic_pairs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(gpu_lib):
    from mpm_snow_sim2d_b200 import mlp
    pairs = synthetic_pairs(4096, seed=9)
    m = mlp.Mlp(seed=21)
    m.set_normalization(*mlp.normalization(pairs))
    return m, pairs


@pytest.mark.parametrize("at", [0, 128, 1000])
def test_two_parts_bitwise(net, at):
    """128 rows: one tile of one CTA, its two parts added once."""
    m, pairs = net
    rows = pairs[at:at + 128]
    whole, _ = m.gradient(rows)
    a, b = (m.gradient(rows[k:k + 64])[0] * np.float32(0.5) for k in (0, 64))
    assert np.array_equal(whole, a + b)


@pytest.mark.parametrize("tiles", [2, 128, 256])
def test_sum_over_ctas(net, tiles):
    """One tile a CTA, and two (256 tiles are more than there are CTAs): at most three FP32 additions of parts in a
    CTA and one rounding of the FP64 total."""
    m, pairs = net
    rows = pairs[np.random.default_rng(tiles).integers(0, len(pairs), tiles * 128)]
    whole, loss = m.gradient(rows)
    parts = [m.gradient(rows[k:k + 64]) for k in range(0, len(rows), 64)]
    g = np.stack([p[0] for p in parts]).astype(np.float64) / len(parts)
    bound = 2.0 ** -24 * (3 * np.abs(g).sum(0) + np.abs(g.sum(0)))
    assert np.all(np.abs(whole - g.sum(0)) <= bound)
    want = np.mean([p[1] for p in parts], dtype=np.float64)
    # the loss: FP32 sums of positive terms, at most 64 + 8 + 2 of them in a row
    assert abs(loss - want) <= 2 * 74 * 2.0 ** -24 * want


def test_creating_a_network_takes_little_memory(net):
    """The parameters, their moments and a gradient, 5 x 40 KB, from pieces of 2 MB that the driver has mapped or maps; the
    training launch's partial sums (6 MB) come with the first training."""
    import torch
    from mpm_snow_sim2d_b200 import mlp

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    m, pairs = net
    before = free()
    other = mlp.Mlp(seed=3)
    assert before - free() <= 2 << 20
    other.set_normalization(*m.norm)
    for n in (128, 4096, 128):  # the room grows, and is kept
        got, _ = other.gradient(pairs[:n])
        again, _ = other.gradient(pairs[:n])
        assert np.array_equal(got, again) and np.isfinite(got).all() and got.any()
    kept = free()
    other.gradient(pairs[:4096])
    assert free() == kept


@pytest.mark.parametrize("count", [1000, 13108])  # 80 KB of pairs; 1 MB and one row
def test_first_training_allocates_nothing_behind_a_large_set(net, count):
    """A set of pairs of 1 MB or more brings the room for training's partial sums with it. Sets that follow one another
    leave a network that trains as a new one with the last set."""
    import torch
    from mpm_snow_sim2d_b200 import mlp

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    m, pairs = net
    sets = [synthetic_pairs(k, seed=k) for k in (count, 20000, 500, count)]

    def train(net_, p):
        net_.set_params(m.params())
        net_.set_normalization(*m.norm)
        net_.load_pairs(p)
        before = free()
        losses = net_.train(2, 16384, 1e-3, 1e-4, seed=5)
        return before - free(), np.concatenate([net_.params(), np.asarray(losses, np.float32)])

    used = mlp.Mlp(seed=1)
    for k, p in enumerate(sets):
        taken, got = train(used, p)
        if k == 0:
            assert (taken <= 2 << 20) == (count > 13107)
        fresh = mlp.Mlp(seed=2)
        _, want = train(fresh, p)
        assert np.array_equal(got, want) and np.isfinite(got).all()
        assert np.array_equal(used.gradient(p[:300])[0], fresh.gradient(p[:300])[0])
