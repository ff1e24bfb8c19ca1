"""Shared memory of the chunked pull gather: layouts that take all of it, and
simulations of different sizes side by side."""
import numpy as np
import pytest

import neuronephys_clean_gb300 as nn

pytestmark = pytest.mark.gpu


def _sim(ctx, n, deg, dmax, seed=55):
    rng = np.random.default_rng(seed)
    c = nn.default_config(n)
    c.seed, c.max_delay, c.delivery = seed, dmax, nn.NN_DELIVERY_PULL
    s = nn.Simulation(ctx, c)
    cnt = rng.integers(0, 2 * deg + 1, n)
    m = int(cnt.sum())
    s.set_network(np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64), rng.integers(0, n, m).astype(np.int32),
                  (rng.random(m) * 0.05).astype(np.float32), rng.integers(1, dmax + 1, m).astype(np.uint8),
                  (rng.random(n) < 0.2).astype(np.uint8))
    s.init_state(-65.0, 0.0, 12.0)
    s.set_field("V", rng.uniform(-70, -10, n).astype(np.float32))
    return s


def _state(s):
    return np.stack([s.get_field(q) for q in ("V", "M", "H", "N", "GE", "GI")])


@pytest.mark.parametrize("n,deg,dmax", [(139849, 1, 8), (80965, 49, 60), (100_000, 3, 3), (131_072, 2, 20)])
def test_layouts_near_the_limit(ctx, monkeypatch, n, deg, dmax):
    """As the gather without chunks, which sums in FP32 in another order: the
    conductances to 1e-6, everything else follows within a few steps' rounding."""
    a = _sim(ctx, n, deg, dmax)
    monkeypatch.setenv("NN_PULL_UNSLICED", "1")
    b = _sim(ctx, n, deg, dmax)
    a.step(60)
    b.step(60)
    x, y = _state(a), _state(b)
    assert np.array_equal(a.raster()[1], b.raster()[1])
    assert np.abs(x[4:] - y[4:]).max() <= 1e-6 * max(1.0, np.abs(y[4:]).max())
    assert np.abs(x[:4] - y[:4]).max() <= 1e-3


def test_a_small_simulation_beside_a_large_one(ctx):
    """Creating the second leaves the first its shared memory (the gather's sums
    are whole numbers: equal bits)."""
    alone = _sim(ctx, 60_000, 100, 20)
    alone.step(30)
    a = _sim(ctx, 60_000, 100, 20)
    a.step(7)
    b = _sim(ctx, 300, 3, 2)
    b.step(5)
    a.step(23)
    assert np.array_equal(_state(a), _state(alone))
