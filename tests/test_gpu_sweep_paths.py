"""The persistent FP64 sweeps and the PCG line passes on both sides of their
dispatch rules: grids whose coefficients stay in shared memory (to about
540,000 cells) and larger ones, the smallest grid, rows of odd length, solves
that stop within the first sweeps, values kept for putting back or not, lines
that fit in shared memory and longer ones, tiles that are not full.  Against
the oracle bit for bit, or against a sparse direct solve."""
import ctypes

import numpy as np
import pytest
import scipy.sparse.linalg as spla

from conftest import fld_from_shell, oracle_from_shell, rel_l2
from test_oracle import hypre_matrix, rad_oracle

pytestmark = pytest.mark.gpu

SYSTEM = ("SOR_A", "SOR_B", "SOR_C", "SOR_D", "SOR_E", "SOR_F", "SOR_G", "RHS_ER")
EVALS = ("EVAL1", "EVAL2", "EVAL3", "EVAL4", "EVAL5", "EVAL6", "EVAL7", "EVAL8", "EVAL_1_6")


def random_system(dims, seed):
    """A diagonally dominant system (no couplings into the radial and theta
    ghosts) and a right-hand side."""
    rng = np.random.default_rng(seed)
    s = {n: -rng.random(dims) for n in SYSTEM[1:7]}
    for n, axis, at in (("SOR_B", 0, 0), ("SOR_C", 0, -1), ("SOR_F", 2, 0), ("SOR_G", 2, -1)):
        sl = [slice(None)] * 3
        sl[axis] = at
        s[n][tuple(sl)] = 0.0
    s["SOR_A"] = 1.02 * sum(-s[n] for n in SYSTEM[1:7]) + rng.random(dims)
    s["RHS_ER"] = rng.standard_normal(dims)
    return {n: np.asfortranarray(a) for n, a in s.items()}


def pair(dims, seed=1, poles=False):
    from oracle import Oracle
    from ttcode_gb300.fld import FLD
    from ttcode_gb300.synthetic import make_shell
    sh = make_shell(*dims, seed=seed, poles=poles)
    sh.params["sorparam"] = 1.2
    f = FLD(sh.grid, sh.params)
    o = Oracle(*dims)
    for k, v in sh.params.items():
        if k != "kappa_model":
            o.set(k, v)
    for n, a in random_system(dims, seed).items():
        f.upload(n, a)
        o.f(n)[...] = a
    return f, o


# the smallest grid; odd radial counts; more blocks than rows allow; both
# sides of the shared-memory limit
@pytest.mark.parametrize("dims", [(4, 4, 4), (5, 6, 7), (33, 10, 5), (160, 6, 4), (64, 96, 80), (67, 112, 80)])
@pytest.mark.parametrize("poles", [False, True])
def test_exact_sweeps_and_stop(dims, poles):
    f, o = pair(dims, poles=poles)
    zero = np.zeros_like(o.f("DELTA_ER"))
    for n in (1, 2, 5):
        f.upload("DELTA_ER", zero)
        o.f("DELTA_ER")[...] = 0.0
        r, _ = f.sor_sweeps(n)
        assert o.call("sor_sweeps", n) == 0
        assert np.array_equal(f.download("DELTA_ER"), o.f("DELTA_ER")), n
        assert abs(r - o.get("global_rnorm")) <= 1e-12 * o.get("global_rnorm")
    # solves that stop after a few sweeps: the iterate is that of the sweep at
    # which the oracle's norm first meets the rule
    f.set_solver("sor64_exact")
    for eps, itmax in ((0.5, 1000), (1e-3, 1000), (1e-30, 3)):
        f.set_params(epsmat=eps, itmax=itmax)
        st = f.solve_system()
        o.f("DELTA_ER")[...] = 0.0
        ratios = []
        for _ in range(st.sor_iter):
            assert o.call("sor_sweeps", 1) == 0
            ratios.append(o.get("global_rnorm") / o.get("global_rhsnorm"))
        assert np.array_equal(f.download("DELTA_ER"), o.f("DELTA_ER")), (eps, st.sor_iter)
        assert all(q > eps for q in ratios[:-1])
        assert (ratios[-1] <= eps and st.status == 0) or (st.sor_iter == itmax and st.status == 1)
    f.close()


@pytest.mark.parametrize("dims", [(4, 4, 4), (37, 10, 5), (64, 128, 80), (128, 128, 80)])
@pytest.mark.parametrize("poles", [False, True])
def test_scaled_sweeps(dims, poles):
    """The scaled FP64 form from and to the same iterates (its rounding is its own)."""
    f, o = pair(dims, seed=2, poles=poles)
    f.set_params(epsmat=1e-11)
    f.set_solver("sor64_exact")
    ref = f.solve_system()
    x = f.download("DELTA_ER")
    f.set_solver("sor64_fast")
    st = f.solve_system()
    assert st.status == 0 and abs(st.sor_iter - ref.sor_iter) <= 1
    assert rel_l2(f.download("DELTA_ER"), x) <= 1e-10
    f.close()


@pytest.mark.parametrize("dims", [(4, 4, 4), (41, 12, 9), (64, 64, 64), (96, 112, 64)])
def test_noalloc_is_the_context_solve(dims):
    """The allocation-free solve, with and without room to keep the values a
    stopped sweep has replaced: the context's solve bit for bit."""
    import torch
    from ttcode_gb300 import _ffi
    f, _ = pair(dims, seed=3)
    L = _ffi.lib()
    f.set_params(epsmat=1e-6)
    f.set_solver("sor64_exact")
    ref = f.solve_system()
    nx, ny, nz = dims
    ptrs = [L.ttfld_device_ptr(f.h, _ffi.FIELDS[n]) for n in SYSTEM]
    x = torch.zeros((nz + 4, ny + 4, nx + 4), dtype=torch.float64, device="cuda")
    it = ctypes.c_int()
    rc = L.ttfld_sor_solve_noalloc(*ptrs, x.data_ptr(), nx, ny, nz, 1.2, 1e-6, 1, 1000,
                                   torch.cuda.current_stream().cuda_stream, ctypes.byref(it), None, None)
    assert rc == 0 and it.value == ref.sor_iter
    assert np.array_equal(x.cpu().numpy().transpose(2, 1, 0), f.download("DELTA_ER"))
    f.close()


@pytest.mark.parametrize("dims,ibdrad", [((9, 4, 5), 7), ((9, 4, 5), 9), ((90, 96, 72), 4)])
def test_raddif_in_one_launch(dims, ibdrad):
    from ttcode_gb300.synthetic import make_shell
    sh = make_shell(*dims, seed=4)
    o = rad_oracle(sh, ibdrad, 1e-10, 11)
    rc = o.call("raddif", 0.0, 0.0, 1, 0)
    f = fld_from_shell(sh, eps=1e-10, itmax=11)
    f.set_params(ibdrad=ibdrad, iii=2)
    f.stellarinput_heating()
    st = f.raddif(0.0, 0.0, 1, 0)
    assert st.status == rc and st.sor_iter == int(o.get("sor_iter"))
    er = f.download("ER")
    if ibdrad == 9:  # exp() of the heating in the moving top
        assert rel_l2(er, o.f("ER")) <= 1e-12
    else:
        assert np.array_equal(er, o.f("ER"))
    f.close()


# lines whose forward results fit in shared memory (NX <= 168) and longer
# ones, columns that do not fill a warp's 32
@pytest.mark.parametrize("dims", [(12, 6, 5), (168, 12, 10), (172, 10, 7), (40, 64, 33)])
def test_pcg_lines(dims):
    from ttcode_gb300.synthetic import make_shell
    f = fld_from_shell(make_shell(*dims, seed=5, delt=100.0))
    f.set_solver("pcg", tol=1e-10)
    f.coupled_energy_eqs(True)
    f.set_params(epsmat=1e-13, itmax=200000)
    f.set_solver("sor64_fast")
    f.begin_step(new_run=True)
    f.solve_system()
    ref = f.download("DELTA_ER")
    f.set_solver("pcg", tol=1e-11)
    st = f.solve_system()
    assert st.status == 0
    assert rel_l2(f.download("DELTA_ER"), ref) <= 1e-9
    f.close()


# tiles of one colour in shared memory, several groups a block, and lines too
# long for it (NX > 440), whose tiles lie in global memory
@pytest.mark.parametrize("dims", [(12, 6, 5), (24, 10, 7), (5, 128, 80), (460, 8, 6)])
def test_hypre_tiles(dims):
    from ttcode_gb300.synthetic import make_shell
    sh = make_shell(*dims, seed=6, delt=100.0)
    f = fld_from_shell(sh)
    f.set_solver("pcg", tol=1e-10)
    f.coupled_energy_eqs(True)
    o = oracle_from_shell(sh)
    for n in EVALS + ("RHS_ER", "UPPERBND"):
        o.f(n)[...] = f.download(n)
    assert o.call("fill_hypre_system") == 0
    x_ref = spla.spsolve(hypre_matrix(o).tocsc(), o.f("HYP_RHS").ravel(order="F")).reshape(dims, order="F")
    st = f.solve_with_hypre(tol=1e-12, maxit=10000)
    nx, ny, nz = dims
    assert st.status == 0
    assert rel_l2(f.download("DELTA_ER")[2:nx + 2, 2:ny + 2, 2:nz + 2], x_ref) <= 1e-8
    f.close()
