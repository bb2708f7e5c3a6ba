"""The PCG solver's forms for radial lines that are too long for shared memory:
couplings staged up to NX = 517, the anchor and the update up to 1551, line
tiles of SOLVE_WITH_HYPRE up to 440 and block Jacobi's forward results up to
168.  Checked like the shorter lines: against a sparse direct solve and the
scaled FP64 sweeps."""
import pytest

import test_gpu_sweep_paths as paths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(520, 6, 5), (1552, 4, 4)])
def test_hypre(dims):
    paths.test_hypre_tiles(dims)


def test_pcg():
    paths.test_pcg_lines((520, 6, 5))
