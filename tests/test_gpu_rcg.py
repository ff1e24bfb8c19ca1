"""The resident CG (whole solve in one kernel) against the FP64 oracle at the
edges of its bricks: rows that end inside a quad, single planes, rows and
cells, last bricks cut short, and the largest grids it takes.

Tolerance: the recurrence's relative residual <= rtol.  The true residual may
exceed it by the rounding of the FP32 recurrences: 2^-24 |A| |x| an iteration,
adding up like sqrt(60) < 8 over the 60 or so iterations here, with
|A| <= 1 + beta + 12 alpha max D and |x| <= the larger of guess and solution.
The error is at most the residual over the smallest eigenvalue, 1 + beta."""
import threading

import numpy as np
import pytest

import neuronephys_clean_gb300 as nn

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (7, 5, 3), (1, 9, 130), (50, 1, 4), (6, 17, 2), (11, 20, 97), (5, 33, 255), (64, 64, 64),
          (37, 41, 61), (9, 10, 2048), (96, 101, 75)]


def _problem(shape, hetero, seed=3):
    rng = np.random.default_rng(seed)
    G = int(np.prod(shape))
    D = rng.lognormal(0.0, 1.0, shape).astype(np.float32) if hetero else None
    b = (0.01 * rng.random(G)).astype(np.float32)
    b[rng.integers(0, G, max(1, G // 300))] += 1.0
    return D, b, rng.random(G).astype(np.float32)


@pytest.mark.parametrize("hetero", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_resident_solve_matches_oracle(ctx, orc, shape, hetero):
    nz, ny, nx = shape
    D, b, x0 = _problem(shape, hetero)
    alpha, beta = 6.0, 0.05
    pc = nn.PCG(ctx, nx, ny, nz, alpha, beta, ctx.to_device(D.ravel()) if hetero else None)
    ref, _, _ = orc.pcg7(b, np.zeros(b.size), shape, alpha, beta, D, rtol=1e-12)
    db = ctx.to_device(b)
    for guess in (np.zeros_like(b), x0):  # a second solve of the same object, from another guess
        dx = ctx.to_device(guess)
        it, rel = pc.solve(db, dx, rtol=1e-6, max_iter=5000)
        assert rel <= 1e-6
        norm = 1 + beta + 12 * alpha * (1.0 if D is None else float(D.max()))
        gap = 8 * 2.0 ** -24 * norm * max(np.linalg.norm(guess), np.linalg.norm(ref))
        bound = 1e-6 * np.linalg.norm(b) + gap
        assert np.linalg.norm(b - orc.apply7(dx.numpy(), shape, alpha, beta, D)) <= bound
        assert np.linalg.norm(dx.numpy() - ref) <= bound / (1 + beta)
    # a solution is recognised without an iteration; zero iterations are not enough otherwise
    it, rel = pc.solve(db, dx, rtol=1e-4, max_iter=10)
    assert it == 0 and rel <= 1e-4
    zero = ctx.to_device(np.zeros_like(b))
    with pytest.raises(nn.NNError) as e:
        pc.solve(db, zero, rtol=1e-6, max_iter=0)
    assert e.value.status == nn.NN_ERR_NOT_CONVERGED


def test_resident_zero_diffusivity_as_two_kernel(ctx, monkeypatch):
    """One cell without diffusion is solved; two adjacent ones have the face
    coefficient 0 / 0 and do not converge, as in the two-kernel solver."""
    n = 12
    D = np.ones((n, n, n), np.float32)
    D[5, 5, 5] = 0.0
    b = np.random.default_rng(0).random(n ** 3).astype(np.float32)
    for two in (False, True):
        if two:
            D[5, 5, 6] = 0.0
        dD = ctx.to_device(D.ravel())
        sols = []
        for env in (False, True):
            if env:
                monkeypatch.setenv("NN_PCG_TWO_KERNEL", "1")
            pc = nn.PCG(ctx, n, n, n, 4.0, 0.1, dD)
            monkeypatch.delenv("NN_PCG_TWO_KERNEL", raising=False)
            x = ctx.to_device(np.zeros(n ** 3, np.float32))
            if two:
                with pytest.raises(nn.NNError) as e:
                    pc.solve(ctx.to_device(b), x, rtol=1e-6, max_iter=200)
                assert e.value.status == nn.NN_ERR_NOT_CONVERGED
            else:
                pc.solve(ctx.to_device(b), x, rtol=1e-6, max_iter=200)
                sols.append(x.numpy())
        if not two:
            assert np.linalg.norm(sols[0] - sols[1]) <= 1e-5 * np.linalg.norm(sols[1])


def test_resident_solves_from_two_threads(built_lib):
    """Two contexts on two host threads solve at the same time; every solve
    gives the bits of a solve alone (its sums have a fixed order)."""
    shape, res, errors = (96, 96, 96), {}, []
    D, b, _ = _problem(shape, False)

    def solve(ctx, pc, db, dx):
        dx.zero()
        pc.solve(db, dx, rtol=1e-6)
        return dx.numpy()

    def work(k):
        try:
            with nn.Context(0) as ctx:
                pc = nn.PCG(ctx, *shape[::-1], 20.0, 0.0)
                db, dx = ctx.to_device(b), ctx.empty((b.size,), np.float32)
                res[k] = [solve(ctx, pc, db, dx) for _ in range(40)]
                pc.close()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    work("alone")
    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for k in range(2):
        assert all(np.array_equal(r, res["alone"][0]) for r in res[k])


@pytest.mark.parametrize("sides", [[1], [2, 1, 3], [64, 5, 33, 17, 50, 9], [7] * 200, [40] * 20 + [21] * 40 + [100]])
def test_resident_batch_matches_oracle(ctx, orc, sides):
    """All instances of a batch in one launch: single cells, more instances
    than blocks (lists of several), groups of different widths."""
    alpha_unit, beta = 3e-3, 0.02
    bp = nn.BatchedPCG(ctx, sides, alpha_unit, beta)
    rng = np.random.default_rng(5)
    b = (0.01 * rng.random(int(bp.offsets[-1]))).astype(np.float32)
    b[rng.integers(0, b.size, max(1, b.size // 300))] += 1.0
    db, dx = ctx.to_device(b), ctx.to_device(np.zeros_like(b))
    for guess in (0.0, 0.3):  # a second solve of the same object, from another guess
        dx.copy_from(np.full_like(b, guess))
        its, bad = bp.solve(db, dx, 1e-6, 5000)
        assert bad == 0
        x = dx.numpy()
        for k in {0, len(sides) // 2, len(sides) - 1}:
            g, lo, hi = sides[k], int(bp.offsets[k]), int(bp.offsets[k + 1])
            al = alpha_unit * g * g
            ref, rit, _ = orc.pcg7(b[lo:hi], np.full(hi - lo, guess), (g, g, g), al, beta, rtol=1e-12)
            gap = 8 * 2.0 ** -24 * (1 + beta + 12 * al) * max(guess * (hi - lo) ** 0.5, np.linalg.norm(ref))
            bound = 1e-6 * np.linalg.norm(b[lo:hi]) + gap
            assert np.linalg.norm(x[lo:hi] - ref) <= bound / (1 + beta), k
    its, bad = bp.solve(db, dx, 1e-3, 10)
    assert bad == 0 and np.all(its == 0)
    dx.zero()
    its, bad = bp.solve(db, dx, 1e-6, 0)
    assert bad == len(sides)
