"""New geometries of a batch are taken in groups of solves (about four million
sites each): solves of several groups, of one group together, and solves whose
types change between runs so that their lists grow, shrink and grow, run as the
same lattice in a handle of its own does.  Both are within 2e-5 (FP32) and 1e-9
(FP64) of the oracle; the bounds here are twice those."""
import numpy as np
import pytest

from cases import gpu_lattice, rel_err

pytestmark = pytest.mark.gpu

BOXES = [(96, 100, 104), (5, 6, 20), (120, 97, 101), (3, 3, 3), (17, 11, 9), (110, 108, 99), (33, 5, 4), (101, 100, 98),
         (9, 8, 12)]


@pytest.mark.parametrize("Ls", [(2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0)], ids=["one", "multi"])
@pytest.mark.parametrize("precision", ["FP32", "FP64"])
def test_geometries_in_groups(qmin, oracle, precision, Ls):
    prec, tol_f, tol_q = (qmin.FP32, 2e-4, 4e-5) if precision == "FP32" else (qmin.FP64, 2e-9, 2e-9)
    b = qmin.Batch(BOXES, prec)
    b.set_chunk_shape(0)

    def system(k, walls):
        s = oracle.System(BOXES[k], Ls=Ls)
        s.random_nematic(30 + k)
        for plane in walls:
            if plane < BOXES[k][2]:
                s.add_wall(2, plane, k % 2, 5.3)
        return s

    p = system(3, ()).p
    b.set_params(p.A, p.B, p.C, p.L1, p.L2, p.L3, p.L4, multi_constant=p.multi_constant)
    walls = [(0,) if k % 3 else () for k in range(len(BOXES))]
    for step in ({}, {0: (0, 7), 1: (4,), 5: (0, 50), 6: ()}, {0: (), 2: (3,)}, {0: (1, 20, 60), 8: (0, 6)}):
        for k, w in step.items():
            walls[k] = w
        ss = [system(k, w) for k, w in enumerate(walls)]
        for k, s in enumerate(ss):
            b.set_solve(k, s.Q, s.types, [(s.objs[j].kind, s.objs[j].W, s.objs[j].S0) for j in range(s.nobj)])
        b.fire_init()
        r = b.fire_run(3)
        for k, s in enumerate(ss):
            lat = gpu_lattice(qmin, s, prec)
            lat.set_fire_kernel(qmin.FIRE_SEPARATE)
            lat.fire_init()
            rl = lat.fire_run(3)
            assert abs(r["forceMax"][k] - rl["forceMax"]) <= tol_f * rl["forceMax"], (step, k)
            assert rel_err(b.get_solve(k), lat.get_state()[0]) <= tol_q, (step, k)
            lat.close()
    b.close()
