"""Grids too large for the resident solve that are thin or narrow: single
planes, a few planes, rows of one cell, planes of one small tile.

Tolerance: as of the streamed solve's tests, a relative residual of 1e-6 plus
the rounding of the FP32 recurrences, 2^-24 |A| |x| an iteration, adding up like
sqrt(100) over at most 100 of them."""
import numpy as np
import pytest

import neuronephys_clean_gb300 as nn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hetero", [False, True])
@pytest.mark.parametrize("shape", [(1, 1500, 1600), (1700, 1500, 1), (2, 1030, 1041), (4, 600, 1300), (8, 400, 900),
                                   (3000, 6, 7), (5000, 20, 20), (40001, 1, 3), (2600, 32, 33), (1, 1, 300001)])
def test_thin_grids_match_oracle(ctx, orc, shape, hetero):
    nz, ny, nx = shape
    G, alpha, beta = nx * ny * nz, 1.5, 0.2
    rng = np.random.default_rng(3)
    D = rng.lognormal(0.0, 0.7, shape).astype(np.float32) if hetero else None
    b = (0.01 * rng.random(G)).astype(np.float32)
    b[rng.integers(0, G, max(1, G // 300))] += 1.0
    pc = nn.PCG(ctx, nx, ny, nz, alpha, beta, ctx.to_device(D.ravel()) if hetero else None)
    norm = 1 + beta + 12 * alpha * (1.0 if D is None else float(D.max()))
    db = ctx.to_device(b)
    for guess in (np.zeros(G, np.float32), rng.random(G).astype(np.float32)):
        dx = ctx.to_device(guess)
        it, rel = pc.solve(db, dx, rtol=1e-6, max_iter=500)
        assert 0 < it <= 100 and rel <= 1e-6
        x = dx.numpy()
        gap = 10 * 2.0 ** -24 * norm * max(np.linalg.norm(guess), np.linalg.norm(x))
        assert np.linalg.norm(b - orc.apply7(x, shape, alpha, beta, D)) <= 1e-6 * np.linalg.norm(b) + gap


@pytest.mark.parametrize("shape", [(1, 1500, 1600), (1, 8, 16), (140, 136, 132), (32, 32, 32)])
def test_whole_quads_want_x_aligned(ctx, shape):
    """Whichever solver takes the grid."""
    nz, ny, nx = shape
    pc = nn.PCG(ctx, nx, ny, nz, 1.0, 0.1)
    b, x = ctx.to_device(np.ones(nx * ny * nz, np.float32)), ctx.to_device(np.zeros(nx * ny * nz + 4, np.float32))
    solve = nn.lib().nn_pcg_solve
    assert solve(pc.handle, b.ptr, x.value + 4, 1e-3, 100, None, None) == 1
    assert solve(pc.handle, b.ptr, x.value, 1e-3, 100, None, None) == 0
