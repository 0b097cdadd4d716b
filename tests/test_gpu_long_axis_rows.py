"""The roundtrip passes of long 1-D axes with everything a step can put between two sandwiches: potential
and CAP tables, laser phases, the step mask and reductions with axis and grid weights, on even and odd
splits (64 x 128 points, 256 x 256 and 512 x 256), both gauges, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8192, 65536, 131072])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 2e-5)])
def test_masked_runs_with_observables(qnd_lib, n, precision, tol):
    from tdse_nd_mpi_b200 import Grid

    dr, steps = (0.1,), 4
    g, o = Grid(1, (n,), dr, "BM4", 0.05, precision=precision), O.OracleCtx(1, (n,), dr, "BM4", 0.05)
    x = g.axis_r(0)
    mask = np.where(np.abs(x) > 0.4 * n * dr[0], 0.98, 1.0)
    for q in (g, o):
        q.set_potential("H_1D")
        q.set_cap(0.05, 5.0)
        q.set_gradv(0, x / (x * x + 2.0) ** 1.5)
        q.set_mask_axis(0, mask)
    psi0 = O.smooth_state((n,), dr, 7)
    F = np.random.default_rng(n).standard_normal((steps, g.s, 1)) * 0.05
    names = ["norm", "dipole_r", "accel"]
    a, st = psi0.copy(), g.state(psi0)
    want, got = o.run_length(a, F, names), g.run_length(st, F, names)
    assert np.linalg.norm(st.download() - a) <= tol * np.linalg.norm(a)
    assert np.all(np.abs(got - want) <= tol * np.max(np.abs(want), axis=0).clip(1e-3))
    a, st = psi0.copy(), g.state(psi0)
    alpha = np.zeros((steps, 1))
    want, got = o.run_velocity(a, F, alpha, names), g.run_velocity(st, F, alpha, names)
    assert np.linalg.norm(st.download() - a) <= tol * np.linalg.norm(a)
    assert np.all(np.abs(got - want) <= tol * np.max(np.abs(want), axis=0).clip(1e-3))
