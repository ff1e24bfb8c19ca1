"""The CG of one kernel an iteration, on grids too large for the resident
solve: tiles cut short, rows that end inside a quad, several tiles along a row,
single planes and cells a row, odd and even iteration counts.

Tolerance of a solve: the recurrence's relative residual <= rtol.  The true
residual may exceed it by the rounding of the FP32 recurrences: 2^-24 |A| |x|
an iteration, adding up like sqrt(100) = 10 over the iterations here, with
|A| <= 1 + beta + 12 alpha max D and |x| <= the larger of guess and solution.
The error is at most the residual over the smallest eigenvalue, 1 + beta."""
import numpy as np
import pytest

import neuronephys_clean_gb300 as nn

pytestmark = pytest.mark.gpu

HETERO = [(80, 66, 260), (109, 111, 113), (400, 700, 5), (37, 37, 1030), (2, 3, 240001), (9000, 2, 80)]
CONST = [(136, 135, 137), (900, 1000, 3), (2, 1100, 1152)]


def _problem(shape, hetero, seed=3):
    rng = np.random.default_rng(seed)
    G = int(np.prod(shape))
    D = rng.lognormal(0.0, 0.7, shape).astype(np.float32) if hetero else None
    b = (0.01 * rng.random(G)).astype(np.float32)
    b[rng.integers(0, G, max(1, G // 300))] += 1.0
    return D, b, rng.random(G).astype(np.float32)


@pytest.mark.parametrize("shape,hetero", [(s, True) for s in HETERO] + [(s, False) for s in CONST])
def test_streamed_solve_matches_oracle(ctx, orc, shape, hetero):
    nz, ny, nx = shape
    D, b, x0 = _problem(shape, hetero)
    alpha, beta = 1.5, 0.2
    pc = nn.PCG(ctx, nx, ny, nz, alpha, beta, ctx.to_device(D.ravel()) if hetero else None)
    db = ctx.to_device(b)
    norm = 1 + beta + 12 * alpha * (1.0 if D is None else float(D.max()))
    for guess, rtol in ((np.zeros_like(b), 1e-5), (x0, 1e-6)):  # a second solve of the same object
        dx = ctx.to_device(guess)
        it, rel = pc.solve(db, dx, rtol=rtol, max_iter=500)
        assert 0 < it <= 100 and rel <= rtol
        x = dx.numpy()
        gap = 10 * 2.0 ** -24 * norm * max(np.linalg.norm(guess), np.linalg.norm(x))
        bound = rtol * np.linalg.norm(b) + gap
        assert np.linalg.norm(b - orc.apply7(x, shape, alpha, beta, D)) <= bound
    it, rel = pc.solve(db, dx, rtol=1e-4, max_iter=10)  # recognised without an iteration
    assert it == 0 and rel <= 1e-4 and np.array_equal(dx.numpy(), x)


@pytest.mark.parametrize("shape,hetero", [((70, 131, 153), True), ((130, 140, 136), False)])
def test_streamed_iterates_match_two_kernels(ctx, monkeypatch, shape, hetero):
    """x after n iterations, n odd and even, against the two-kernel solver's.
    Both run the same recurrence in FP32 from x = 0: the rounding of some ten
    operations an iteration, 1e-5 of the iterate with room."""
    nz, ny, nx = shape
    D, b, _ = _problem(shape, hetero)
    dD, db = ctx.to_device(D.ravel()) if hetero else None, ctx.to_device(b)
    got = []
    for env in (False, True):
        if env:
            monkeypatch.setenv("NN_PCG_TWO_KERNEL", "1")
        pc = nn.PCG(ctx, nx, ny, nz, 2.0, 0.1, dD)
        monkeypatch.delenv("NN_PCG_TWO_KERNEL", raising=False)
        xs = []
        for n in (0, 1, 2, 3, 4, 17, 18):
            dx = ctx.to_device(np.zeros_like(b))
            with pytest.raises(nn.NNError) as e:
                pc.solve(db, dx, rtol=1e-12, max_iter=n)
            assert e.value.status == nn.NN_ERR_NOT_CONVERGED
            xs.append(dx.numpy())
        got.append(xs)
    for n, (x, y) in enumerate(zip(*got)):
        assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y), n


@pytest.mark.parametrize("grid", [140, 141])
def test_streamed_solve_overlaps_as_in_line(ctx, grid):
    """Field solves of the second stream, finished a period later, give the bits
    of solves in line, whether the iterations work on the field itself (whole
    quads) or on a padded copy; the sums have a fixed order."""
    got = []
    for overlap in (0, 1):
        c = nn.default_config(2000)
        c.seed, c.grid, c.timescale, c.delivery, c.par_overlap = 7, grid, 50, nn.NN_DELIVERY_PULL, overlap
        s = nn.Simulation(ctx, c)
        s.generate_network(nn.default_net_spec(nn.NN_NET_ER))
        s.init_state(-65.0, 5.0, 15.0)
        s.set_field("V", np.random.default_rng(7).uniform(-65, -35, 2000).astype(np.float32))
        for n in (50, 100, 50):
            s.step(n)
        got.append((s.get_density(), s.get_field("V")))
    assert np.linalg.norm(got[0][0]) > 0
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("n", [12, 112])
@pytest.mark.parametrize("solver", ["cg", "two kernels", "multigrid"])
def test_infinite_diffusivity_does_not_converge(ctx, monkeypatch, n, solver):
    """A cell with infinite diffusion has the face coefficients inf / inf: no
    solver converges, on the chip, streamed or with multigrid."""
    D = np.ones((n, n, n), np.float32)
    D[5, 6, 7] = np.inf
    b = ctx.to_device(np.random.default_rng(0).random(n ** 3).astype(np.float32))
    dD = ctx.to_device(D.ravel())
    if solver == "two kernels":
        monkeypatch.setenv("NN_PCG_TWO_KERNEL", "1")
    pc = nn.PCG(ctx, n, n, n, 4.0, 0.1, dD)
    s = nn.MultigridPCG(pc) if solver == "multigrid" else pc
    with pytest.raises(nn.NNError) as e:
        s.solve(b, ctx.to_device(np.zeros(n ** 3, np.float32)), rtol=1e-6, max_iter=200)
    assert e.value.status in (nn.NN_ERR_NOT_CONVERGED, 5)  # 5: non-finite state
