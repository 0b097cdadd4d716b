"""Velocity-gauge runs as chunk-wide chains (observables between the two factors of a step boundary, the
mask after every step): against the oracle step by step, chunk boundaries, graph replays and both parities
of the sandwich count."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

NAMES = ["dipole_r", "norm", "accel"]


@pytest.mark.parametrize("shape,integ,steps", [
    ((32, 64), "Verlet", 300), ((64, 16), "BM4", 5), ((8, 16, 32), "RKN4", 4), ((8, 16, 32), "Verlet", 7),
    ((4, 8192), "Verlet", 3), ((16,), "Verlet", 5), ((16384,), "BM4", 3), ((1024, 64), "BM4", 3)])
@pytest.mark.parametrize("masked", [False, True])
def test_velocity_run_vs_oracle(qnd_lib, shape, integ, steps, masked):
    from tdse_nd_mpi_b200 import Grid

    dim, dr = len(shape), (0.25,) * len(shape)
    g, o = Grid(dim, shape, dr, integ, 0.02), O.OracleCtx(dim, shape, dr, integ, 0.02)
    rng = np.random.default_rng(steps)
    V = rng.standard_normal(shape)
    for q in (g, o):
        (q.set_vpot if q is o else q.set_potential)(V)
        q.set_cap(0.05, 1.0)
        for j in range(dim):
            q.set_gradv(j, np.random.default_rng(j).standard_normal(shape))
            if masked:
                q.set_mask_axis(j, np.linspace(0.95, 1.0, shape[j]))
    psi0 = O.smooth_state(shape, dr, 3)
    A = rng.standard_normal((steps, g.s, dim)) * 0.05
    alpha = rng.standard_normal((steps, dim)) * 0.05
    a, st = psi0.copy(), g.state(psi0)
    want, got = o.run_velocity(a, A, alpha, NAMES), g.run_velocity(st, A, alpha, NAMES)
    grow = max(1.0, steps / 10)
    assert np.linalg.norm(st.download() - a) <= 1e-12 * grow * np.linalg.norm(a)
    assert np.all(np.abs(got - want) <= 1e-11 * grow * np.max(np.abs(want), axis=0))
    b, st2 = psi0.copy(), g.state(psi0)  # without observables the boundary factors merge
    o.run_velocity(b, A, alpha, [])
    g.run_velocity(st2, A, alpha, [])
    assert np.linalg.norm(st2.download() - b) <= 1e-12 * grow * np.linalg.norm(b)
    g.close()


@pytest.mark.parametrize("integ", ["Verlet", "RKN4"])
@pytest.mark.parametrize("shape", [(32, 64), (16384,)])
@pytest.mark.parametrize("masked", [False, True])
def test_no_memory_for_the_boundary_factor(qnd_lib, integ, shape, masked, monkeypatch):
    """Where a context holds only the tables that a single step needs, a run of several steps still goes
    through (step by step), with the same state to rounding."""
    from tdse_nd_mpi_b200 import QndError

    def run(steps):
        from tdse_nd_mpi_b200 import Grid

        dim = len(shape)
        g = Grid(dim, shape, (0.3,) * dim, integ, 0.05)
        r2 = sum(np.reshape(g.axis_r(j) ** 2, [-1 if k == j else 1 for k in range(dim)]) for j in range(dim))
        g.set_potential(-1.0 / np.sqrt(r2 + 0.5))
        if masked:
            for j in range(dim):
                g.set_mask_axis(j, np.linspace(0.97, 1.0, shape[j]))
        st = g.state(np.exp(-0.5 * r2) + 0j)
        A = np.random.default_rng(2).standard_normal((5, g.s, dim)) * 0.05
        try:
            g.run_velocity(st, A[:steps])
            return st.download()
        finally:
            g.close()

    want = run(5)
    for tables in range(1, 12):
        monkeypatch.setenv("QND_FAIL_TABLES_ABOVE", str(tables))
        try:
            run(1)
            break
        except QndError as e:
            assert e.code == 3
    got = run(5)
    # the same operators, the factor of a boundary as one product or two
    assert np.linalg.norm(got - want) <= 1e-13 * np.linalg.norm(want)
