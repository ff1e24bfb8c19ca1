"""Range of the CG kernels' sums: the same system with its right-hand side and
guess scaled by a power of two is solved in the same iterations to the scaled
solution, for tiny and huge values, while squares of the residual over the
diagonal stay representable.

Tolerance: scaling by a power of two is exact, so the two solves differ only
through squares near the ends of the float range.  Iteration counts within 5 %
(at least three); the solutions both reach the relative residual 1e-6, so they
differ by at most 2e-6 |b| over the smallest eigenvalue 1 + beta, plus the
rounding of the FP32 recurrences: 2^-24 |A| |x| an iteration, adding up like
the root of their number, with |A| <= 1 + beta + 12 alpha max D."""
import numpy as np
import pytest

import neuronephys_clean_gb300 as nn

pytestmark = pytest.mark.gpu
BETA = 0.05

# shape (nz, ny, nx), cell field, alpha, exponents
CASES = [((40, 44, 48), False, 6.0, (-40, 50)), ((40, 44, 48), True, 6.0, (-40, 50)),
         ((5, 4, 7), False, 1.5, (-40, 50)), ((5, 4, 7), True, 1.5, (-40, 50)),
         ((21, 33, 35), True, 6.0, (-40, 50)), ((48, 48, 48), False, 2000.0, (-46, 45)),
         ((134, 130, 136), False, 6.0, (-40, 50)), ((134, 130, 136), False, 2000.0, (-46, 45)),
         ((110, 109, 112), True, 6.0, (-40, 50))]


def _bound(b, x, norm, it):
    return (2e-6 * np.linalg.norm(b) + 2 * it ** 0.5 * 2.0 ** -24 * norm * np.linalg.norm(x)) / (1 + BETA)


@pytest.mark.parametrize("shape,hetero,alpha,exps", CASES)
def test_scaled_system_solves_alike(ctx, shape, hetero, alpha, exps):
    rng = np.random.default_rng(2)
    nz, ny, nx = shape
    G = nx * ny * nz
    D = rng.lognormal(0.0, 0.7, G).astype(np.float32) if hetero else None
    b = rng.random(G).astype(np.float32)
    pc = nn.PCG(ctx, nx, ny, nz, alpha, BETA, ctx.to_device(D) if hetero else None)
    x, its = {}, {}
    for e in (0,) + exps:
        dx = ctx.to_device(np.zeros(G, np.float32))
        its[e], rel = pc.solve(ctx.to_device(np.ldexp(b, e)), dx, rtol=1e-6, max_iter=20000)
        assert rel <= 1e-6
        x[e] = np.ldexp(dx.numpy().astype(np.float64), -e)
    norm = 1 + BETA + 12 * alpha * (1.0 if D is None else float(D.max()))
    for e in exps:
        assert abs(its[e] - its[0]) <= max(3, 0.05 * its[0]), e
        assert np.linalg.norm(x[e] - x[0]) <= _bound(b, x[0], norm, its[0]), e


def test_scaled_batch_solves_alike(ctx):
    """Instances of one batch at different scales."""
    sides, exps = [32, 32, 32, 20, 20, 5, 5], [0, -40, 50, 0, -40, 0, -40]
    unit = 6.0 / 32 ** 2
    bp = nn.BatchedPCG(ctx, sides, unit, BETA)
    rng = np.random.default_rng(2)
    one = {g: rng.random(g ** 3).astype(np.float32) for g in set(sides)}
    db = ctx.to_device(np.concatenate([np.ldexp(one[g], e) for g, e in zip(sides, exps)]))
    dx = ctx.to_device(np.zeros(sum(g ** 3 for g in sides), np.float32))
    its, bad = bp.solve(db, dx, 1e-6, 5000)
    assert bad == 0
    x = [np.ldexp(dx.numpy()[lo:hi].astype(np.float64), -e)
         for lo, hi, e in zip(bp.offsets, bp.offsets[1:], exps)]
    for k, ref in ((1, 0), (2, 0), (4, 3), (6, 5)):
        g = sides[k]
        assert abs(int(its[k]) - int(its[ref])) <= 3, k
        assert np.linalg.norm(x[k] - x[ref]) <= _bound(one[g], x[ref], 1 + BETA + 12 * unit * g * g, its[ref]), k
