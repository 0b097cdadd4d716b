"""Final spectra over the kept momenta alone: no momentum, fewer than one block's run, and more than
the blocks of the energy distribution take at their shortest run, with bins past one block's threads."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prmax,ne", [((1e-9, 5.0), 40), ((0.3, 0.5), 17), ((0.9, 50.0), 300), ((50.0, 50.0), 300)])
def test_spectra_of_kept_momenta(qnd_lib, prmax, ne):
    from tdse_nd_mpi_b200 import Grid

    shape, dr, rmask, de = (64, 256), (0.3, 0.2), (2.0, 5.0), 0.02
    grid = Grid(2, shape, dr, "BM4", 0.05)
    psi = O.smooth_state(shape, dr, 3) * np.exp(1j * 0.7 * O.seeded_state(shape, 4).real)
    want, counts, data = O.final_spectra_numpy(psi, dr, rmask, prmax, de, ne)
    ped, got_counts, pmd = grid.final_spectra(grid.state(psi), rmask, prmax, de, ne)
    assert list(got_counts) == list(counts)
    # sums of at most 16384 non-negative terms in another order, exp to a few units in the last place
    np.testing.assert_allclose(ped, want, rtol=0, atol=1e-11 * np.max(np.abs(want)))
    assert pmd.shape == data.shape
    np.testing.assert_allclose(pmd[:, 0], data[:, 0], rtol=0, atol=1e-12 * data[:, 0].max())


def test_spectra_without_a_kept_momentum(qnd_lib):
    from tdse_nd_mpi_b200 import Grid

    grid = Grid(1, (64,), (0.3,), "BM4", 0.05)
    psi = O.smooth_state((64,), (0.3,), 3)
    ped, counts, pmd = grid.final_spectra(grid.state(psi), (2.0, 5.0), (-1.0,), 0.02, 9)
    assert counts == [0] and pmd.shape == (0, 2)
    assert np.all(ped == 0.0)
