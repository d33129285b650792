"""The FP64 batch iteration (bulk sites in 64-bit fixed point, listed sites in
items of their own) against each solve's oracle run, 1e-9 as every FP64 path:
boxes from the smallest to several items, both metric modes, fields inside and
outside the fixed-point range side by side in one batch, a
resumed run."""
import numpy as np
import pytest

from cases import rel_err

pytestmark = pytest.mark.gpu

BOXES = [(3, 3, 3), (33, 5, 4), (9, 40, 12), (17, 31, 9), (5, 6, 70), (64, 10, 5), (40, 41, 37)]


def systems(oracle, Ls, metric_mode):
    out = []
    for k, L in enumerate(BOXES):
        s = oracle.System(L, Ls=Ls, metric_mode=metric_mode)
        s.random_nematic(20 + k)
        if k == 2:
            s.Q += 0.4 * np.random.default_rng(k).standard_normal(s.Q.shape)  # beyond the range
        elif k == 3:
            s.Q *= 1e-3  # below it
        if k % 2:
            s.add_wall(2, 0, 0, 5.3)
        if k % 3 and min(L) >= 5:
            s.add_sphere(tuple(0.5 * x for x in L), 1.9, k % 2, 1.5)
        out.append(s)
    return out


@pytest.mark.parametrize("metric_mode", [0, 1])
@pytest.mark.parametrize("Ls", [(2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0), (2.32, 1.0, 0.5, 0.3, 0)],
                         ids=["one", "multi", "multi_l4"])
def test_solves_follow_the_oracle(qmin, oracle, Ls, metric_mode):
    ss = systems(oracle, Ls, metric_mode)
    b = qmin.Batch([s.L for s in ss], qmin.FP64, metric_mode)
    p = ss[0].p
    b.set_params(p.A, p.B, p.C, p.L1, p.L2, p.L3, p.L4, multi_constant=p.multi_constant)
    for k, s in enumerate(ss):
        b.set_solve(k, s.Q, s.types, [(s.objs[j].kind, s.objs[j].W, s.objs[j].S0) for j in range(s.nobj)])
    b.fire_init()
    b.fire_run(4)
    r = b.fire_run(9)
    for k, s in enumerate(ss):
        V = np.zeros((s.N, 5))
        ro = s.fire(9, V=V)
        assert r["iterations"][k] == 9
        assert abs(r["forceMax"][k] - ro["forceMax"]) <= 1e-9 * ro["forceMax"], k
        assert rel_err(b.get_solve(k), s.Q) <= 1e-9, k
    b.close()
