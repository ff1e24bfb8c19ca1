"""The one-launch Crank-Nicolson solve and the sub-tile coupling scatter at the
edges of their splits, against the oracle.

Solve tolerance: 1e-5 of the largest value the FP32 solve carries, the density
(the paracrine module's test has the same bound) or the initial guess
u + dt D lap u, which for D = 5 and a rough u is 40 times as large; the density
is set, no neuron deposits.  Coupling: whole counts, equal."""
import numpy as np
import pytest

import neuronephys_clean_gb300 as nn

pytestmark = pytest.mark.gpu
TIMEOUT = 6  # NN_ERR_TIMEOUT


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 2, 7), (5, 31, 33), (9, 64, 97), (70, 80, 90)])
@pytest.mark.parametrize("D,max_iter", [(0.05, 20), (5.0, 20), (5.0, 0)])
def test_cn_solve_matches_oracle(ctx, orc, shape, D, max_iter):
    p = nn.ParacrineModule.default_params()
    p.nz, p.ny, p.nx = shape
    p.h, p.D, p.decay, p.par_dt, p.max_iter = 1.0, D, 3e-4, 1.0, max_iter
    zero = ctx.to_device(np.zeros(1, np.float32))
    pm = nn.ParacrineModule(ctx, ctx.empty((1,), np.float32), 1, p, zero, zero, zero)
    u = np.random.default_rng(1).random(int(np.prod(shape))).astype(np.float32)
    for _ in range(2):
        pm.set_density(u)
        it, _ = pm.update_on_own_timescale()
        ref, rit, _ = orc.paracrine_cn_solve(u.astype(np.float64), shape, 1.0, p.D, p.decay, 1.0, 1e-6, max_iter, 1)
        assert it == rit
        got = pm.density().astype(np.float64)
        guess = u.max() * (1 + D * 256 / 30)  # |lap u| <= (128 + 128) / 30 max u for h = 1
        assert np.abs(got - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max(), guess)
        u = got.astype(np.float32)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 2047, 2048, 2049, 14638, 40961])
@pytest.mark.parametrize("frac", [0.0, 0.05, 1.0])
def test_coupling_scatter_edges(ctx, orc, n, frac):
    rng = np.random.default_rng(n)
    deg = rng.integers(0, 140, n)
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    idx = rng.integers(0, n, max(int(off[-1]), 1)).astype(np.int32)
    out = np.where(rng.random(n) < frac, 0.5, 0.05).astype(np.float32)
    cp = nn.AtomicCoupling(ctx, n)
    ins = ctx.to_device(np.full(n, 7.0, np.float32))
    nf = cp(nn.AdjacencyList(ctx.to_device(idx), ctx.to_device(off)), ins, ctx.to_device(out))
    rnf, rin, rfire = orc.coupling_push(idx, off, out, nn.NN_SIGNAL_COUNT)
    assert nf == rnf
    assert np.array_equal(ins.numpy(), rin)
    assert np.array_equal(cp.get_firing_neurons()[:nf], rfire)


@pytest.mark.parametrize("shape", [(61, 79, 80), (90, 100, 110), (130, 125, 128)])
def test_cn_solve_blocks_per_sm(ctx, orc, shape):
    """One, two and three blocks an SM, whose blocks read what others wrote
    through L1; bounds as above."""
    p = nn.ParacrineModule.default_params()
    p.nz, p.ny, p.nx = shape
    p.h, p.D, p.decay, p.par_dt, p.max_iter = 1.0, 5.0, 3e-4, 1.0, 20
    zero = ctx.to_device(np.zeros(1, np.float32))
    pm = nn.ParacrineModule(ctx, ctx.empty((1,), np.float32), 1, p, zero, zero, zero)
    u = np.random.default_rng(4).random(int(np.prod(shape))).astype(np.float32)
    pm.set_density(u)
    it, _ = pm.update_on_own_timescale()
    ref, rit, _ = orc.paracrine_cn_solve(u.astype(np.float64), shape, 1.0, p.D, p.decay, 1.0, 1e-6, 20, 1)
    assert it == rit
    guess = u.max() * (1 + p.D * 256 / 30)
    assert np.abs(pm.density().astype(np.float64) - ref).max() <= 1e-5 * max(1.0, np.abs(ref).max(), guess)


def test_cn_solve_reports_a_barrier_that_gave_up(ctx, monkeypatch):
    """With no polls allowed the barrier's waits run out at once: a call that
    reads the outcome reports it, one that does not leaves it to the module's
    next update, each once; the density stays, and the context is usable."""
    p = nn.ParacrineModule.default_params()
    p.nx = p.ny = p.nz = 64
    zero, g = ctx.to_device(np.zeros(1, np.float32)), ctx.empty((1,), np.float32)
    monkeypatch.setenv("NN_CN_POLLS", "0")
    pm = nn.ParacrineModule(ctx, g, 1, p, zero, zero, zero)
    monkeypatch.delenv("NN_CN_POLLS")
    u = np.random.default_rng(1).random(64 ** 3).astype(np.float32)
    pm.set_density(u)
    with pytest.raises(nn.NNError) as e:
        pm.update_on_own_timescale()
    assert e.value.status == TIMEOUT
    own, fine = nn.lib().nn_paracrine_ref_own, nn.lib().nn_paracrine_ref_fine
    cp = nn.AtomicCoupling(ctx, 1)
    for later in (lambda: own(pm.handle, None, None), lambda: fine(pm.handle, cp.handle)):
        assert own(pm.handle, None, None) == 0
        ctx.synchronize()
        assert later() == TIMEOUT
    assert fine(pm.handle, cp.handle) == 0
    assert np.array_equal(pm.density(), u)
    ok = nn.ParacrineModule(ctx, g, 1, p, zero, zero, zero)
    ok.set_density(u)
    assert ok.update_on_own_timescale()[0] > 0


@pytest.mark.parametrize("n", [778_240, 778_241, 1_000_003, 10_100_001])
@pytest.mark.parametrize("frac", [0.01, 1.0])
def test_coupling_scatter_of_many_neurons(ctx, orc, n, frac):
    """Longer stretches a block, and several of them; whole counts, equal."""
    rng = np.random.default_rng(n)
    off = np.concatenate([[0], np.cumsum(rng.integers(0, 4, n))]).astype(np.int32)
    idx = rng.integers(0, n, int(off[-1])).astype(np.int32)
    out = np.where(rng.random(n) < frac, 0.5, 0.05).astype(np.float32)
    cp = nn.AtomicCoupling(ctx, n)
    ins = ctx.to_device(np.full(n, 7.0, np.float32))
    nf = cp(nn.AdjacencyList(ctx.to_device(idx), ctx.to_device(off)), ins, ctx.to_device(out))
    rnf, rin, rfire = orc.coupling_push(idx, off, out, nn.NN_SIGNAL_COUNT)
    assert nf == rnf
    assert np.array_equal(ins.numpy(), rin)
    assert np.array_equal(cp.get_firing_neurons()[:nf], rfire)
