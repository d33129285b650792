"""Where the fixed-point form hands over to FP64, |Q| = 1 at any LC site: one
site with exactly 1 (outside; as a fixed-point number it would be another
value), with the number below it (inside), and with values between 3/4 and 1,
single lattices and batches against the oracle, 1e-12 for a force and 1e-9
after FIRE, as every FP64 path."""
import numpy as np
import pytest

from cases import gpu_lattice, rel_err

pytestmark = pytest.mark.gpu

VALUES = {"one": 1.0, "minus_one": -1.0, "below_one": np.nextafter(1.0, 0.0), "above_three_quarters": 0.76,
          "two": 2.0, "large": 7.5}


@pytest.mark.parametrize("Ls", [(2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0)], ids=["one", "multi"])
@pytest.mark.parametrize("name", list(VALUES) + ["upper_quarter"])
@pytest.mark.parametrize("L", [(14, 11, 10), (48, 44, 50)], ids=["small", "force_only_in_fixed_point"])
def test_one_value(qmin, oracle, L, name, Ls):
    s = oracle.System(L, Ls=Ls)
    s.random_nematic(8)
    s.add_wall(2, 0, 0, 5.3)
    s.add_sphere(tuple(0.5 * x for x in L), 2.2, 1, 2.0)
    site = int(np.flatnonzero(s.types == 0)[len(s.types) // 5])
    if name == "upper_quarter":
        rng = np.random.default_rng(4)
        lc = s.types <= 0
        s.Q[lc] = rng.uniform(0.75, 1.0, (lc.sum(), 5)) * rng.choice([-1.0, 1.0], (lc.sum(), 5))
    else:
        s.Q[site, 3] = VALUES[name]
    lat = gpu_lattice(qmin, s, qmin.FP64)
    assert rel_err(lat.force(), s.force()) <= 1e-12
    b = qmin.Batch([s.L], qmin.FP64)
    b.set_params(s.p.A, s.p.B, s.p.C, s.p.L1, s.p.L2, s.p.L3, multi_constant=s.p.multi_constant)
    b.set_solve(0, s.Q, s.types, [(s.objs[j].kind, s.objs[j].W, s.objs[j].S0) for j in range(s.nobj)])
    lat.set_fire_kernel(qmin.FIRE_SPLIT)
    if any(Ls[1:]):
        lat.set_fire_variant(0)
    ro = s.fire(3)
    for run, Q in ((lat, lambda: lat.get_state()[0]), (b, lambda: b.get_solve(0))):
        run.fire_init()
        r = run.fire_run(3)
        assert abs(np.atleast_1d(r["forceMax"])[0] - ro["forceMax"]) <= 1e-9 * ro["forceMax"]
        assert rel_err(Q(), s.Q) <= 1e-9
