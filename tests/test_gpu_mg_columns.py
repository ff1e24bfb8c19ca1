"""The multigrid's column kernels at the edges of their split: short and long
rows (one quad; more than half a block and more than a block of quads, where
row pairs of the restriction lie in different blocks), few rows, chunks of
planes cut short, a coarse level by columns.  Tolerance of one V-cycle as in
test_gpu_mg.py: 1e-4 of its largest magnitude, FP32 through the levels."""
import numpy as np
import pytest

import neuronephys_clean_gb300 as nn
from oracle import multigrid as mgo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hetero", [False, True])
@pytest.mark.parametrize("shape,levels", [((4, 4, 4), 2), ((6, 10, 44), 2), ((4, 6, 520), 2), ((4, 4, 1032), 2),
                                          ((5, 7, 12), 1), ((62, 34, 60), 2), ((256, 208, 160), 2)])
def test_vcycle_columns(ctx, shape, levels, hetero):
    rng = np.random.default_rng(2)
    D = rng.lognormal(0.0, 1.0, shape).astype(np.float32) if hetero else None
    alpha, beta = 20.0, 1e-3
    pc = nn.PCG(ctx, shape[2], shape[1], shape[0], alpha, beta, ctx.to_device(D.ravel()) if hetero else None)
    mg = nn.MultigridPCG(pc, levels)
    r = rng.standard_normal(int(np.prod(shape))).astype(np.float32)
    dz = ctx.empty((r.size,), np.float32)
    mg.apply(ctx.to_device(r), dz)
    ref = mgo.vcycle(mgo.hierarchy(shape, alpha, beta, D, levels=levels), r.reshape(shape).astype(np.float64)).ravel()
    np.testing.assert_allclose(dz.numpy(), ref, rtol=0, atol=1e-4 * np.abs(ref).max())
