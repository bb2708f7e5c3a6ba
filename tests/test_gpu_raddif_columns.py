"""ttfld_raddif in one launch on columns that differ: the boundary values that
RADIATIVEBOUND writes behind each colour (both colours of a column) are read by
the neighbouring columns, which other blocks own.  UPPERBND differs from column
to column (BOUNDS takes it from the density), the top is fixed (IBDRAD = 4, 7)
or moves on with every application (IBDRAD = 9, III = 2), and the grids go from
one short round of cells per block to several.

Bars, as for the uniform columns: E_R bitwise where no pow() enters, relative
L2 <= 1e-12 where the moving top reads the stellar heating; the same iterations;
repeated calls equal bit for bit.
"""
import numpy as np
import pytest

from conftest import fld_from_shell, rel_l2
from test_oracle import rad_oracle

pytestmark = pytest.mark.gpu


def shell(dims, uneven, seed=4, lowest=None):
    """A shell whose density falls below BOUNDS' 1e-9 at another radius in
    every column (uneven; from cell `lowest` or NX/2 on), or nowhere
    (UPPERBND = NX-1)."""
    from ttcode_gb300.synthetic import make_shell
    sh = make_shell(*dims, seed=seed, delt=100.0)
    if uneven:
        nx, ny, nz = dims
        first = np.random.default_rng(seed).integers(lowest or nx // 2, nx + 1, (ny, nz))
        rh = sh.fields["RH"][2:nx + 2, 2:ny + 2, 2:nz + 2]
        rh[np.arange(1, nx + 1)[:, None, None] >= first[None]] = 5e-10
    return sh


# coefficients in shared memory (the first two) and not (about 620,000 cells)
@pytest.mark.parametrize("dims", [(24, 16, 12), (41, 32, 30), (90, 96, 72)])
@pytest.mark.parametrize("ibdrad,uneven", [(4, True), (7, True), (9, True), (9, False)])
def test_boundary_values_wait_for_their_readers(dims, ibdrad, uneven):
    sh = shell(dims, uneven)
    o = rad_oracle(sh, ibdrad, 1e-10, 11)
    ub = np.asarray(o.f("UPPERBND"))[2:-2, 2:-2]
    assert (np.unique(ub).size > 4) == uneven
    t0 = o.f("T").copy()
    rc = o.call("raddif", 0.0, 0.0, 1, 0)
    f = fld_from_shell(sh, itmax=11)
    f.set_params(ibdrad=ibdrad, iii=2)
    f.stellarinput_heating()
    first = None
    for _ in range(4):
        f.upload("T", t0)
        st = f.raddif(0.0, 0.0, 1, 0)
        er = f.download("ER")
        assert st.status == rc and st.sor_iter == int(o.get("sor_iter"))
        if ibdrad == 9:
            assert rel_l2(er, o.f("ER")) <= 1e-12
        else:
            assert np.array_equal(er, o.f("ER"))
        if first is None:
            first = er
        assert np.array_equal(er, first)
    f.close()


@pytest.mark.parametrize("dims", [(9, 4, 5), (24, 16, 12)])
@pytest.mark.parametrize("ibdrad", [4, 7, 9])
def test_columns_with_their_top_at_the_first_cell(dims, ibdrad):
    """UPPERBND = 1: the cell i = 1 belongs to both radial boundaries, and
    RADIATIVEBOUND writes the bottom first, then the top.  Every cell of such a
    column is a boundary cell, and these are compared: the limiter of its faces
    is the one at UPPERBND - 1 = 0, where the reference forms none, so that the
    cells beside the column differ."""
    sh = shell(dims, True, lowest=1)
    o = rad_oracle(sh, ibdrad, 1e-10, 11)
    at = np.zeros(o.f("ER").shape, bool)
    at[2:, 2:-2, 2:-2] = np.asarray(o.f("UPPERBND"))[None, 2:-2, 2:-2] == 1
    assert at.any()
    rc = o.call("raddif", 0.0, 0.0, 1, 0)
    f = fld_from_shell(sh, itmax=11)
    f.set_params(ibdrad=ibdrad, iii=2)
    f.stellarinput_heating()
    st = f.raddif(0.0, 0.0, 1, 0)
    got, want = f.download("ER")[at], o.f("ER")[at]
    assert st.status == rc and st.sor_iter == int(o.get("sor_iter"))
    # IBDRAD = 9: exp() and pow() within some ulp of libm's
    assert np.all(np.abs(got - want) <= (1e-12 * want if ibdrad == 9 else 0.0))
    f.close()
