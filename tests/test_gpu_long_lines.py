"""The PCG solver on radial lines that are too long for shared memory (line tiles
of SOLVE_WITH_HYPRE fit up to NX = 440, block Jacobi's forward results up to
168, pieces of 517 radii of the couplings and of 1551 of the anchor and the
update), and on strips of lines cut into pieces: one radius in the last piece,
fewer columns than a strip has, a piece per strip.  Checked like the other
lines: against a sparse direct solve and the scaled FP64 sweeps."""
import pytest

import test_gpu_sweep_paths as paths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(520, 6, 5), (1552, 4, 4)])
def test_hypre(dims):
    paths.test_hypre_tiles(dims)


@pytest.mark.parametrize("dims", [(520, 6, 5), (520, 36, 152)])
def test_pcg(dims):
    paths.test_pcg_lines(dims)


@pytest.mark.parametrize("dims", [(15, 4, 4), (33, 34, 5)])
def test_strips_hypre(dims):
    paths.test_hypre_tiles(dims)


@pytest.mark.parametrize("dims", [(15, 4, 4), (33, 34, 5), (49, 70, 30), (65, 40, 160), (91, 64, 60)])
def test_strips_pcg(dims):
    paths.test_pcg_lines(dims)
