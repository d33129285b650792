"""Types that leave an object's neighbours unmarked (type 0): those sites read
the object's Q like any other, whatever its size.  Object sites of planar
anchoring hold a unit vector, whose components may be 1 and more is accepted;
the FP64 forces and FIRE against the oracle within 1e-12 and 1e-9, FP32 within
1e-4 in forceMax and 2e-5 in Q, single lattices and batches."""
import numpy as np
import pytest

from cases import gpu_lattice, rel_err

pytestmark = pytest.mark.gpu


def system(oracle, Ls, value):
    s = oracle.System((9, 8, 11), Ls=Ls)
    s.random_nematic(6)
    s.add_sphere((4.0, 4.0, 5.0), 1.2, 1, 2.0)
    s.types[s.types < 0] = 0
    inside = s.types > 0
    assert 0 < inside.sum() < 40
    s.Q[inside] = 0.0
    s.Q[inside, 1] = value
    s.Q[inside, 3] = -value
    return s


@pytest.mark.parametrize("Ls", [(2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0)], ids=["one", "multi"])
@pytest.mark.parametrize("value", [0.4, 1.0, -1.5, 3.0])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_forces_beside_an_unmarked_object(qmin, oracle, precision, value, Ls):
    prec, tol, tol_f, tol_q = (qmin.FP64, 1e-12, 1e-9, 1e-9) if precision == "FP64" else (qmin.FP32, 2e-5, 1e-4, 2e-5)
    s = system(oracle, Ls, value)
    lat = gpu_lattice(qmin, s, prec)
    b = qmin.Batch([s.L, s.L], prec)
    b.set_params(s.p.A, s.p.B, s.p.C, s.p.L1, s.p.L2, s.p.L3, multi_constant=s.p.multi_constant)
    for k in range(2):
        b.set_solve(k, s.Q, s.types, [(s.objs[j].kind, s.objs[j].W, s.objs[j].S0) for j in range(s.nobj)])
    lc = s.types <= 0
    assert rel_err(lat.force()[lc], s.force()[lc]) <= tol
    lat.set_fire_kernel(qmin.FIRE_SPLIT)
    if any(Ls[1:]):
        lat.set_fire_variant(0)
    ro = s.fire(6)
    for run, get in ((lat, lambda: lat.get_state()[0]), (b, lambda: b.get_solve(1))):
        run.fire_init()
        r = run.fire_run(6)
        f = np.atleast_1d(r["forceMax"])[-1]
        assert abs(f - ro["forceMax"]) <= tol_f * ro["forceMax"]
        assert rel_err(get()[lc], s.Q[lc]) <= tol_q
