"""Contexts of different sizes on one device, in turn and from two host threads:
each solves as it does alone, bit for bit.  Launch shapes belong to a context,
and the shared-memory limit of a kernel, which all contexts share, is not moved
by any of them."""
import threading

import numpy as np
import pytest

from conftest import fld_from_shell

pytestmark = pytest.mark.gpu

# FP32 coefficients in shared memory (three sizes of it) and not; the FP64
# ones in shared memory in the first two
SIZES = [(24, 16, 12), (40, 64, 32), (53, 90, 47), (128, 128, 80)]


def context(dims):
    """A context that holds the system of an implicit step."""
    from ttcode_gb300.synthetic import make_shell
    f = fld_from_shell(make_shell(*dims, seed=dims[0], delt=100.0))
    f.set_solver("mixed", tol=1e-10)
    f.coupled_energy_eqs(True)
    return f


def solve(f, solver):
    if solver != "hypre":
        f.set_solver(solver, tol=1e-10)
    f.begin_step(new_run=True)
    st = f.solve_with_hypre(tol=1e-8, maxit=1000) if solver == "hypre" else f.solve_system()
    return st.sor_iter, st.status, f.download("DELTA_ER")


def same(a, b):
    return a[:2] == b[:2] and np.array_equal(a[2], b[2])


def in_turn_and_at_once(sizes, solvers, rounds):
    fs = [context(d) for d in sizes]
    ref = []
    for f in fs:
        ref.append({s: solve(f, s) for s in solvers})
    for s in solvers:
        for _ in range(2):
            for f, r in zip(fs, ref):
                assert same(solve(f, s), r[s]), (f.grid.nx, s)
    for m in range(len(fs) - 1):
        wrong, start = [], threading.Barrier(2)

        def work(q):
            try:
                start.wait(30)
                for _ in range(rounds):
                    for s in solvers:
                        if not same(solve(fs[q], s), ref[q][s]):
                            wrong.append((sizes[q], s))
            except Exception as e:  # the other thread's result tells nothing without it
                wrong.append((sizes[q], repr(e)))

        ts = [threading.Thread(target=work, args=(q,)) for q in (m, m + 1)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert not wrong, wrong
    for f in fs:
        f.close()


def test_product_solves():
    in_turn_and_at_once(SIZES, ["mixed"], 25)


def test_other_solvers():
    in_turn_and_at_once([(24, 16, 12), (40, 64, 32), (96, 112, 64)], ["sor64_exact", "sor64_fast", "pcg", "hypre"], 8)
