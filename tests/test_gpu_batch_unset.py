"""A solve of a batch that was never set is a lattice of Q = 0 without objects:
under a field it moves like any other (no active-site count, so it never
converges).  Against the oracle within the bounds of every batch path."""
import numpy as np
import pytest

from cases import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ls", [(2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0)], ids=["one", "multi"])
@pytest.mark.parametrize("precision", ["FP32", "FP64"])
def test_unset_solve_moves(qmin, oracle, precision, Ls):
    prec, tol = (qmin.FP32, 2e-5) if precision == "FP32" else (qmin.FP64, 1e-9)
    E = (0.0, 0.6, 0.8, 1.0, 1.0, 0.5)
    ss = [oracle.System(L, Ls=Ls, E=E) for L in ((7, 9, 8), (12, 5, 6))]
    ss[0].random_nematic(3)
    ss[1].Q[:] = 0.0
    b = qmin.Batch([s.L for s in ss], prec)
    p = ss[0].p
    b.set_params(p.A, p.B, p.C, p.L1, p.L2, p.L3, multi_constant=p.multi_constant, E=E)
    b.set_solve(0, ss[0].Q, ss[0].types, [])
    b.fire_init()
    r = b.fire_run(8)
    assert r["iterations"].tolist() == [8, 8] and np.isinf(r["forceMax"][1])
    for k, s in enumerate(ss):
        s.fire(8)
        assert np.abs(s.Q).max() > 0
        assert rel_err(b.get_solve(k), s.Q) <= tol, k
    b.close()
