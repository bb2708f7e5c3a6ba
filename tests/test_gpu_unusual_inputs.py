"""Inputs outside the ordinary that the entry points take, against the oracle:
columns without irradiation whose MU_STAR is not positive."""
import numpy as np
import pytest

from conftest import fld_from_shell, oracle_from_shell

pytestmark = pytest.mark.gpu


def same_with_nan(got, want, tol):
    """Equal to a relative tol elementwise (products of subnormal exponentials
    apart, below 1e-290), NaN and infinities in the same places."""
    assert np.array_equal(np.isnan(got), np.isnan(want))
    fin = np.isfinite(want)
    assert np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)])
    assert np.all(np.abs(got[fin] - want[fin]) <= tol * np.abs(want[fin]) + 1e-290)


@pytest.mark.parametrize("mu", [-0.05, -0.0, 0.0, 1e-7])
def test_heating_of_columns_without_irradiation(mu):
    """TINCIDENT = 0 with MU_STAR of any sign: STELLARINPUT is 0 or, where the
    exponential overflows or 0 / 0 is formed, NaN (pprad.f:481-484)."""
    from ttcode_gb300.synthetic import make_shell
    sh = make_shell(24, 16, 12, seed=6)
    dark = np.zeros(sh.fields["MU_STAR"].shape, bool)
    dark[4:9] = True
    sh.fields["MU_STAR"][dark] = mu
    sh.fields["TINCIDENT"][dark] = 0.0
    o = oracle_from_shell(sh)
    assert o.call("stellarinput_heating") == 0
    f = fld_from_shell(sh)
    f.stellarinput_heating()
    got, want = f.download("STELLARINPUT"), np.asarray(o.f("STELLARINPUT"))[2:26]
    assert np.isnan(want).any() == (mu <= 0)
    same_with_nan(got, want, 1e-12)  # exp() may differ from libm in the last bit
    f.close()
