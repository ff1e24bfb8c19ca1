"""The solver's autotuners on fields that are solved on the chip in one launch:
nothing to try, so no simulation periods are run and no setting changes."""
import numpy as np
import pytest

import neuronephys_clean_gb300 as nn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("overlap", [0, 1])
def test_nothing_is_tried(ctx, batch, overlap):
    c = nn.default_config(3000)
    c.seed, c.grid, c.timescale, c.par_overlap = 7, 0 if batch else 48, 50, overlap
    s = nn.Simulation(ctx, c)
    if batch:
        s.set_instances(np.array([0, 1000, 3000]), np.array([20, 33], np.int32))
    s.generate_network(nn.default_net_spec(nn.NN_NET_ER))
    s.init_state(-65.0, 5.0, 15.0)
    s.step(50)
    ctx.synchronize()
    before = ctx.kernel_launches
    shape, ms = s.autotune_solver(5)
    assert ctx.kernel_launches - before <= 2  # the right-hand side and a solve
    assert 0 < ms < 1 and shape == s.autotune_solver(5)[0]
    assert shape == 2048 if batch else shape in (4, 6, 8, 12, 16, 24, 32)


def test_batch_keeps_its_setting(ctx):
    bp = nn.BatchedPCG(ctx, [20, 33], 1e-3, 1e-4)
    G = int(bp.offsets[-1])
    b, x = ctx.to_device(np.random.default_rng(0).random(G).astype(np.float32)), ctx.empty((G,), np.float32)
    for cells in (512, 4096):
        bp.set_cells_per_block(cells)
        assert bp.autotune(b, x, 5)[0] == cells
