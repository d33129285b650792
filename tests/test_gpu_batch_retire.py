"""Solves of one batch that retire at different, odd and even, iteration counts:
each stops where its own minimize() stops, keeps its state while the others go
on, and never passes max_iterations.  Against each solve's oracle run: the
iteration counts equal (the oracle's forceMax stays 1e-3 away from the cutoff
at every iteration, ten times what FP32 may differ), forceMax and Q within the
bounds of every batch path (FP32 1e-4 and 2e-5, FP64 1e-9)."""
import numpy as np
import pytest

from cases import rel_err

pytestmark = pytest.mark.gpu

BOXES = [(3, 3, 3), (33, 5, 4), (9, 8, 12), (17, 11, 9), (5, 6, 20), (24, 10, 5), (8, 9, 10), (12, 6, 13), (6, 7, 5),
         (20, 21, 7)]
CUTOFF, MOST = 0.36, 48


def systems(oracle, Ls):
    out = []
    for k, L in enumerate(BOXES):
        s = oracle.System(L, Ls=Ls)
        s.random_nematic(20 + k)
        if k % 2:
            s.add_wall(2, 0, 0, 5.3)
        if k % 3 and min(L) >= 5:
            s.add_sphere(tuple(0.5 * x for x in L), 1.9, k % 2, 1.5)
        out.append(s)
    return out


@pytest.mark.parametrize("Ls", [(2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0)], ids=["one", "multi"])
@pytest.mark.parametrize("precision", ["FP32", "FP64"])
def test_solves_retire_on_their_own(qmin, oracle, precision, Ls):
    prec, tol_f, tol_q = (qmin.FP32, 1e-4, 2e-5) if precision == "FP32" else (qmin.FP64, 1e-9, 1e-9)
    ss = systems(oracle, Ls)
    starts = [s.Q.copy() for s in ss]
    runs = [s.fire(MOST, fcut=CUTOFF, trace=True) for s in ss]
    assert all(np.abs(r["trace"][:, 0] / CUTOFF - 1).min() > 1e-3 for r in runs)
    counts = [r["iterations"] for r in runs]
    assert max(counts) == MOST and min(counts) <= MOST - 12 and len({n & 1 for n in counts}) == 2 and len(set(counts)) >= 6
    b = qmin.Batch([s.L for s in ss], prec)
    p = ss[0].p
    b.set_params(p.A, p.B, p.C, p.L1, p.L2, p.L3, p.L4, multi_constant=p.multi_constant)
    for rep in range(20):
        for k, s in enumerate(ss):
            b.set_solve(k, starts[k], s.types, [(s.objs[j].kind, s.objs[j].W, s.objs[j].S0) for j in range(s.nobj)])
        b.fire_init(force_cutoff=CUTOFF)
        r = b.fire_run(MOST)
        assert r["iterations"].tolist() == counts, rep
        for k, s in enumerate(ss):
            assert abs(r["forceMax"][k] - runs[k]["forceMax"]) <= tol_f * runs[k]["forceMax"], (rep, k)
            assert rel_err(b.get_solve(k), s.Q) <= tol_q, (rep, k)
    b.close()
