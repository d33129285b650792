"""The FP32 batch iteration on tiles: boxes at the edges of the tile cut (one
site row more or less than a tile, sides below the tile, long thin boxes),
one-constant and multi-constant, solves retiring after odd and even iteration
counts and a resumed run, against each solve's FP64 oracle run within FP32
accuracy (forceMax 1e-4, Q 2e-5, as every FP32 batch)."""
import numpy as np
import pytest

from cases import rel_err

pytestmark = pytest.mark.gpu

BOXES = [(3, 3, 3), (33, 5, 4), (32, 9, 17), (17, 31, 9), (64, 10, 5), (65, 7, 6), (9, 40, 12), (5, 6, 70)]


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


@pytest.mark.parametrize("Ls", [(2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0), (2.32, 1.0, 0.5, 0.3, 0)],
                         ids=["one", "multi", "multi_l4"])
def test_tiles_follow_the_oracle(qmin, oracle, Ls):
    ss = systems(oracle, Ls)
    b = qmin.Batch([s.L for s in ss], qmin.FP32)
    p = ss[0].p
    b.set_params(p.A, p.B, p.C, p.L1, p.L2, p.L3, p.L4, multi_constant=p.multi_constant)
    for rep in range(2):  # the second pass sets the same types again
        for k, s in enumerate(ss):
            b.set_solve(k, s.Q, s.types, [(s.objs[j].kind, s.objs[j].W, s.objs[j].S0) for j in range(s.nobj)])
        b.fire_init()
        b.fire_run(7)
        r = b.fire_run(12)
        got = [b.get_solve(k) for k in range(len(ss))]
    for k, s in enumerate(ss):
        V = np.zeros((s.N, 5))
        ro = s.fire(12, V=V)
        assert r["iterations"][k] == 12
        assert abs(r["forceMax"][k] - ro["forceMax"]) <= 1e-4 * ro["forceMax"], k
        assert rel_err(got[k], s.Q) <= 2e-5, k
    b.close()


def test_types_changed_between_runs(qmin, oracle):
    """Another geometry in the same handle: classes and lists follow the types."""
    ss = systems(oracle, (2.32, 1.0, 0.5, 0, 0))[:4]
    b = qmin.Batch([s.L for s in ss], qmin.FP32)
    p = ss[0].p
    b.set_params(p.A, p.B, p.C, p.L1, p.L2, p.L3, p.L4, multi_constant=p.multi_constant)
    for step in range(2):
        for k, s in enumerate(ss):
            if step:
                s.random_nematic(50 + k)
                s.add_wall(0, 1, 0, 3.0)
            b.set_solve(k, s.Q, s.types, [(s.objs[j].kind, s.objs[j].W, s.objs[j].S0) for j in range(s.nobj)])
        b.fire_init()
        r = b.fire_run(9)
        for k, s in enumerate(ss):
            Q = b.get_solve(k)
            ro = s.fire(9)
            assert abs(r["forceMax"][k] - ro["forceMax"]) <= 1e-4 * ro["forceMax"], (step, k)
            assert rel_err(Q, s.Q) <= 2e-5, (step, k)
    b.close()
