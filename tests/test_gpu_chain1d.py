"""1-D chains in one launch against the oracle at every line length of the chain kernel and the lengths
just outside it: both gauges and imaginary time with Gram-Schmidt, chains longer than one launch, the
step mask and reductions between steps."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

DR = (0.15,)


def rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / max(np.linalg.norm(np.ravel(b)), 1e-300))


def _pair(n, integ, precision="fp64"):
    from tdse_nd_mpi_b200 import Grid

    g, o = Grid(1, (n,), DR, integ, 0.05, precision=precision), O.OracleCtx(1, (n,), DR, integ, 0.05)
    for x in (g, o):
        x.set_potential("H_1D")
        x.set_cap(0.05, 2.0)
    return g, o


@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024, 2048, 4096, 8192])
@pytest.mark.parametrize("integ,steps", [("Verlet", 5), ("BM4", 150)])
def test_real_time_chains(qnd_lib, n, integ, steps):
    if steps > 100 and n > 1024:
        steps = 80  # BM4 with observables: 7 sandwiches a step, more than one launch's 512 from 74 steps on
    g, o = _pair(n, integ)
    psi0 = O.smooth_state((n,), DR, n)
    F = np.random.default_rng(n).standard_normal((steps, g.s, 1)) * 0.05
    names = ["norm", "dipole_r"]
    a, st = psi0.copy(), g.state(psi0)
    want = o.run_length(a, F, names)
    got = g.run_length(st, F, names)
    assert rel(st.download(), a) < 1e-12 * max(1, steps / 10)
    assert np.all(np.abs(got - want) <= 1e-11 * np.max(np.abs(want), axis=0))  # the dipole crosses zero
    alpha = np.random.default_rng(1).standard_normal((steps, 1)) * 0.05
    a, st = psi0.copy(), g.state(psi0)
    want = o.run_velocity(a, F, alpha, names)
    got = g.run_velocity(st, F, alpha, names)
    assert rel(st.download(), a) < 1e-12 * max(1, steps / 10)
    assert np.all(np.abs(got - want) <= 1e-11 * np.max(np.abs(want), axis=0))  # the dipole crosses zero


@pytest.mark.parametrize("n", [64, 128, 512, 4096])
def test_mask_between_steps(qnd_lib, n):
    """A masked run of many steps equals one call per step (the mask after each step)."""
    g, _ = _pair(n, "BM4")
    g.set_mask_axis(0, np.linspace(0.9, 1.0, n))
    psi0 = O.smooth_state((n,), DR, 2)
    F = np.random.default_rng(5).standard_normal((9, g.s, 1)) * 0.05
    for run in (g.run_length, g.run_velocity):
        one, many = g.state(psi0), g.state(psi0)
        kw = {"alpha": np.zeros((1, 1))} if run == g.run_velocity else {}
        rows1 = [run(one, F[k:k + 1], names=["norm"], **kw)[0] for k in range(9)]
        kw = {"alpha": np.zeros((9, 1))} if kw else {}
        rows = run(many, F, names=["norm"], **kw)
        assert rel(many.download(), one.download()) < 1e-13
        np.testing.assert_allclose(rows, np.array(rows1), rtol=1e-12)


@pytest.mark.parametrize("n", [64, 128, 256, 4096])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 2e-4)])
def test_imaginary_time_states(qnd_lib, n, precision, tol):
    """Six states, so that a Gram-Schmidt call has more than one batch of projections, over more steps
    than one block; FP32 states carry a few 1e-7 per step."""
    g, o = _pair(n, "BM4", precision)
    rng = np.random.default_rng(n)
    guesses = [O.smooth_state((n,), DR, k) + 0.05 * rng.standard_normal(n) for k in range(6)]
    steps = 140 if n == 128 else 12
    want = [v.astype(np.complex128).copy() for v in guesses]
    states = [g.state(v) for v in guesses]
    for j in range(6):
        o.imag_state(want, j, steps)
        g.imag_propagate(states, j, steps)
        assert rel(states[j].download(), want[j]) < tol


@pytest.mark.parametrize("n", [128, 4096])
@pytest.mark.parametrize("precision,tol", [("fp64", 5e-15), ("mixed", 3e-6)])
@pytest.mark.parametrize("steps", [119, 120, 511, 512])
def test_lists_of_sandwiches(qnd_lib, n, precision, tol, steps):
    """The last short and first long list of a launch (Verlet: steps + 1 sandwiches), the last list of one
    launch and the first of two: the run in one call equals the run in two halves, whose boundary rounds
    the state's factors once more (FP32: the dithered roundings of a launch differ, a random walk of
    2^-24 over two transforms of up to 12 levels a step, seven times that allowed)."""
    g, _ = _pair(n, "Verlet", precision)
    psi0 = O.smooth_state((n,), DR, 4)
    F = np.random.default_rng(steps).standard_normal((steps, 1, 1)) * 0.05
    one, two = g.state(psi0), g.state(psi0)
    g.run_length(one, F)
    g.run_length(two, F[:steps // 2])
    g.run_length(two, F[steps // 2:])
    assert rel(two.download(), one.download()) <= tol * np.sqrt(steps)
    g.close()
