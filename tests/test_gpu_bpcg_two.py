"""The batched PCG of two launches an iteration, which serves batches that the
resident solve does not take: every block layout, instances at the edges of the
blocks, and sides beyond the resident solve's.

Tolerance: as of the batched PCG's other tests, 1e-5 of the FP64 solution
(relative residual 1e-6, smallest eigenvalue above 1)."""
import ctypes as C

import numpy as np
import pytest

import neuronephys_clean_gb300 as nn

pytestmark = pytest.mark.gpu


def _launches(ctx, f):
    before = ctx.kernel_launches
    f()
    return ctx.kernel_launches - before


def _check(ctx, orc, bp, sides, unit, beta, resident, some=None):
    rng = np.random.default_rng(3)
    G = int(bp.offsets[-1])
    b = (0.01 * rng.random(G)).astype(np.float32)
    b[rng.integers(0, G, max(1, G // 300))] += 1.0
    db, dx = ctx.to_device(b), ctx.to_device(np.zeros(G, np.float32))
    got = []
    n = _launches(ctx, lambda: got.append(bp.solve(db, dx, 1e-6, 5000)))
    assert got[0][1] == 0
    assert (n == 1) == resident
    x = dx.numpy()
    for k in range(len(sides)) if some is None else some:
        g, lo, hi = sides[k], bp.offsets[k], bp.offsets[k + 1]
        ref = orc.pcg7(b[lo:hi], np.zeros(hi - lo), (g, g, g), unit * g * g, beta, rtol=1e-12)[0]
        assert np.linalg.norm(x[lo:hi] - ref) <= 1e-5 * np.linalg.norm(ref), k
    its, bad = bp.solve(db, dx, 1e-3, 10)
    assert bad == 0 and np.all(its == 0)


@pytest.mark.parametrize("cells", [512, 1024, 2048, 4096])
def test_two_launch_layouts(ctx, orc, monkeypatch, cells):
    sides, unit, beta = [1, 16, 24, 8, 33, 12, 2], 4e-3, 1e-4
    monkeypatch.setenv("NN_PCG_TWO_KERNEL", "1")
    bp = nn.BatchedPCG(ctx, sides, unit, beta)
    bp.set_cells_per_block(cells)
    _check(ctx, orc, bp, sides, unit, beta, False)


def test_two_launch_autotune(ctx, orc, monkeypatch):
    """(Instances that converge within the trial's ten iterations give no time.)"""
    sides, unit, beta = [16, 24, 33], 4e-3, 1e-4
    monkeypatch.setenv("NN_PCG_TWO_KERNEL", "1")
    bp = nn.BatchedPCG(ctx, sides, unit, beta)
    G = int(bp.offsets[-1])
    b = ctx.to_device(np.random.default_rng(1).random(G).astype(np.float32))
    cpb, ms = bp.autotune(b, ctx.empty((G,), np.float32), 8)
    assert cpb in (512, 1024, 2048, 4096) and ms > 0
    _check(ctx, orc, bp, sides, unit, beta, False)


def test_side_beyond_the_resident_solve(ctx, orc):
    sides, unit, beta = [130, 9], 1e-4, 1e-4
    _check(ctx, orc, nn.BatchedPCG(ctx, sides, unit, beta), sides, unit, beta, False)


@pytest.mark.parametrize("sides,resident", [([8] * 300, True), ([8] * 1000, False), ([16] * 100, True),
                                            ([16] * 600, False), ([24] * 60, True), ([64] * 2 + [9] * 50, True),
                                            ([20] * 8 + [2] * 9000, False), ([128] * 4, True)])
def test_form_of_a_batch(ctx, orc, sides, resident):
    """Many small instances, and instances that each need the whole chip."""
    unit, beta = 1e-3, 1e-4
    n = len(sides)
    _check(ctx, orc, nn.BatchedPCG(ctx, sides, unit, beta), sides, unit, beta, resident, {0, 1, n // 2, n - 1})


def test_resident_batch_holds_no_vectors(ctx):
    """A resident batch keeps buffers of the chip's size (x in use, and faces of
    32 bytes a quad, twice: some 25 MB), not the four vectors of all instances
    that the two-launch form works on."""
    cuda = C.CDLL("libcuda.so.1")

    def free():
        f, t = C.c_size_t(0), C.c_size_t(0)
        assert cuda.cuMemGetInfo_v2(C.byref(f), C.byref(t)) == 0
        return f.value

    sides = [100] * 16
    nn.BatchedPCG(ctx, sides, 1e-3, 1e-4).close()  # loads the kernels
    ctx.synchronize()
    before = free()
    bp = nn.BatchedPCG(ctx, sides, 1e-3, 1e-4)
    assert before - free() < 4 * int(bp.offsets[-1])  # one vector
    bp.close()
