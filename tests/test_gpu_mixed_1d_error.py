"""Mixed-precision 1-D runs stay as near to FP64 as the pass kernels' 16 values per thread put them, at
lengths on both sides of the chain kernel's and the long axis' limits: a few 1e-7 per step."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 128, 256, 512, 2048, 4096, 8192, 32768, 65536])
def test_mixed_run_against_fp64(qnd_lib, n):
    from tdse_nd_mpi_b200 import Grid

    dr, steps = (0.176,), 16
    out = {}
    psi0 = O.smooth_state((n,), dr, 3)
    E = np.random.default_rng(4).standard_normal((steps, 6, 1)) * 0.05
    for precision in ("fp64", "mixed"):
        g = Grid(1, (n,), dr, "BM4", 0.05, precision=precision)
        g.set_potential("H_1D")
        st = g.state(psi0)
        rows = g.run_length(st, E, ["norm", "dipole_r"])
        out[precision] = (st.download(), rows)
        g.close()
    ref, rows = out["fp64"]
    # 14 transforms a step, 16 steps: rounding of 2^-24 per butterfly level, adding up as a random walk
    # over 224 transforms of up to 16 levels (6e-8 * sqrt(224 * 16) = 3.6e-6), three times that allowed
    assert np.linalg.norm(out["mixed"][0] - ref) <= 1.1e-5 * np.linalg.norm(ref)
    assert np.max(np.abs(out["mixed"][1] - rows) / np.max(np.abs(rows), axis=0)) <= 1.1e-5
