"""Inputs outside the ordinary that the entry points take, against the oracle:
columns without irradiation whose MU_STAR is not positive, opacity tables
whose nodes do not increase."""
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


def test_opacity_table_with_unsorted_nodes():
    """BurrowsOPC takes the first node above T and rho in the table's order
    (pprphy.f:1050, 1087), whatever that order is."""
    import oracle as orc
    from ttcode_gb300.fld import FLD
    from ttcode_gb300.synthetic import make_shell
    sh = make_shell(24, 16, 12, seed=7)
    lt, lr = np.linspace(1.69, 3.7, 50), np.linspace(-12.0, -1.9, 50)
    rng = np.random.default_rng(7)
    kr, kp, ka = (np.asfortranarray(rng.uniform(-4.0, 2.0, (50, 50))) for _ in range(3))
    for nodes, (a, b) in ((lt, (36, 43)), (lt, (38, 39)), (lr, (28, 45)), (lr, (36, 40)), (lt, (2, 3))):
        nodes[[a, b]] = nodes[[b, a]]
    o = oracle_from_shell(sh, start=False)
    assert orc._load().ttor_set_opacity_table(o.h, 50, 50, *[a.ctypes.data for a in (lt, lr, kr, kp, ka)]) == 0
    f = FLD(sh.grid, dict(sh.params, kappa_model=2))
    f.set_opacity_table(lt, lr, kr, kp, ka)
    f.load_shell(sh)
    o.set("iii", 1)
    f.set_params(iii=1)
    assert o.call("bounds") == 0 and o.call("kappa") == 0
    f.bounds()
    f.kappa()
    for n in ("XKAPR", "XKAPP", "XKAPA", "DXKAPP_DT", "DXKAPA_DT"):
        # log10 within 2 ulp, weights of up to about 20 beyond the bracket, 10^
        same_with_nan(f.download(n), np.asarray(o.f(n)), 1e-11)
    f.close()
