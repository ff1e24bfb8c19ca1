"""The leapfrog step's rate functions near their singularities, at the switch
between series and quotient, and far out, against the reference's FP64
expressions in numpy.

The gate after one step from gate 0 at dt is a dt / (dt/2 (a + b) + 1): with
dt = 1e-3 it is the opening rate up to factors known in FP64, so a rate that
is the rounding of its FP64 expression gives the gate to the roundings of the
FP32 update: at most six, each 2^-24 relative."""
import numpy as np
import pytest

import neuronephys_clean_gb300 as nn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 64, 65, 4097])
def test_opening_rates(ctx, n):
    edges = [-35.0, -50.0, -30.0, 0.0, 55.0, 120.0, -120.0, -399.0, 399.0, -401.0, 450.0]
    near = [c + s * d for c in (-35.0, -50.0) for s in (-1, 1)
            for d in (4e-6, 1e-4, 2.4e-3, 2.6e-3, 0.1, 3.49, 3.51)]
    rng = np.random.default_rng(n)
    V = np.concatenate([edges, near, rng.uniform(-110, 60, 4096)]).astype(np.float32)[:n]
    e = nn.HHEphys(ctx, n, dt=1e-3)
    e.set("V", V)
    e.simulate_ephys()
    v, dt = V.astype(np.float64), float(np.float32(1e-3))
    f32 = lambda x: x.astype(np.float32).astype(np.float64)  # noqa: E731
    with np.errstate(all="ignore"):
        am = np.where(V == -35, 1.0, (3.5 + 0.1 * v) / -np.expm1(-3.5 - 0.1 * v))
        an = np.where(V == -50, 0.1, (0.5 + 0.01 * v) / -np.expm1(-5 - 0.1 * v))
        bm = 4 * np.exp(-(v + 60) / 18)
        bn = 0.125 * np.exp(-(v + 60) / 80)
        ah, bh = 0.07 * np.exp(-v / 20 - 3), 1 / (np.exp(-3 - 0.1 * v) + 1)
        for name, a, b in (("M", am, bm), ("N", an, bn), ("H", ah, bh)):
            ref = f32(a) * dt / (dt / 2 * (a + b) + 1)
            ok = np.isfinite(ref) & (np.abs(ref) > 1e-30) & (np.abs(ref) < 1e30)
            # bm, bn and ah are FP32 exponentials of FP32 arguments: their error, 2^-22 |argument| or so,
            # enters the gate in proportion to their share of it
            arg = 1 + np.abs(v) / 10
            tol = 6 * 2.0 ** -24 + 2.0 ** -22 * arg * np.minimum(1.0, dt * b + (name == "H"))
            got = e.get(name).astype(np.float64)
            assert np.all(np.abs(got - ref)[ok] <= (tol * np.abs(ref))[ok]), name
