"""Rounding of the FP64 transforms at every line length, so at every stage structure (radix 16 with a
last stage of 2, 4, 8 or 16), contiguous and strided, against numpy's FFT of white noise."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 4, 8, 16, 32, 64, 128, 256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("axis", [0, 1])
def test_unitary_transform_rounding(qnd_lib, n, axis):
    from tdse_nd_mpi_b200 import Grid

    shape = (n, 32) if axis == 0 else (32, n)
    grid = Grid(2, shape, (0.2, 0.3), "Verlet", 0.05)
    psi = O.seeded_state(shape, n + axis)
    st = grid.state(psi)
    grid.to_p(st)
    got = st.download()
    want = np.fft.fftn(psi, norm="ortho")
    # a relative error of a few roundings per butterfly level: 2^-53 times 2 sqrt(log2 N) expected in
    # the 2-norm (random signs), 8 times the level count allowed
    levels = np.log2(n) + 5
    assert np.linalg.norm(got - want) <= 8 * levels * 2.0**-53 * np.linalg.norm(want)
    grid.to_r(st)
    assert np.linalg.norm(st.download() - psi) <= 16 * levels * 2.0**-53 * np.linalg.norm(psi)
    # the largest single error, against the largest value's size
    assert np.max(np.abs(got - want)) <= 32 * levels * 2.0**-53 * np.max(np.abs(want))
    grid.close()


@pytest.mark.parametrize("n", [16, 32, 256, 512, 1024, 4096])
@pytest.mark.parametrize("axis", [0, 1])
def test_transform_rounding_is_the_expected_walk(qnd_lib, n, axis):
    """Three times the expected error: about two units in the last place per butterfly level (the factor,
    formed by up to three squarings, and the sum), adding up as a random walk over the levels."""
    from tdse_nd_mpi_b200 import Grid

    shape = (n, 32) if axis == 0 else (32, n)
    grid = Grid(2, shape, (0.2, 0.3), "Verlet", 0.05)
    psi = O.seeded_state(shape, 3 * n + axis)
    st = grid.state(psi)
    grid.to_p(st)
    want = np.fft.fftn(psi, norm="ortho")
    assert np.linalg.norm(st.download() - want) <= 6 * np.sqrt(np.log2(n) + 5) * 2.0**-53 * np.linalg.norm(want)
    grid.close()
