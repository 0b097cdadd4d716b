"""qnd_step_length in the momentum representation, whose first and last sandwiches take the changes of
representation in: against to_r, run_length and to_p of the same steps, for every pass length of both
transform forms, both end axes (odd and even sandwich counts), 2 and 3 dimensions, chunk boundaries."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 4), (16, 64), (128, 32), (1024, 16), (8, 2048), (32, 4096), (8, 32, 16), (16, 2, 4, 8)])
@pytest.mark.parametrize("integ,steps", [("Verlet", 1), ("BM4", 1), ("BM4", 130)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 2e-6)])
def test_step_matches_transforms_and_run(qnd_lib, shape, integ, steps, precision, tol):
    from tdse_nd_mpi_b200 import Grid

    dim = len(shape)
    g = Grid(dim, shape, (0.3,) * dim, integ, 0.05, precision=precision)
    rng = np.random.default_rng(steps)
    g.set_potential(rng.standard_normal(shape))
    psi = O.seeded_state(shape, 5)
    E = rng.standard_normal((steps, g.s, dim)) * 0.05
    a, b = g.state(psi), g.state(psi)
    g.integration_step_length(a, E)
    g.to_r(b)
    g.run_length(b, E)
    g.to_p(b)
    want = b.download()
    # unitary steps: rounding grows with the number of steps
    assert np.linalg.norm(a.download() - want) <= tol * max(1, steps / 4) * np.linalg.norm(want)
    g.close()
