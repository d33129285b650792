"""FP32 L-BFGS on the products of its pairs (m <= 8; the passes beyond): follows
the oracle within FP32 accuracy (1e-4 in forceMax and Q, as every FP32
minimiser), a resumed run continues bit for bit, and a run that ends inside a
captured chunk leaves the forces at the last Q."""
import numpy as np
import pytest

from cases import gpu_lattice, rel_err

pytestmark = pytest.mark.gpu


def system(oracle, L=(21, 18, 15), Ls=(2.32, 1.0, 0.5, 0, 0)):
    s = oracle.System(L, Ls=Ls)
    s.random_nematic(7)
    s.add_wall(2, 0, 0, 5.3)
    s.add_sphere((10, 9, 8), 3.2, 1, 2.0)
    return s


@pytest.mark.parametrize("Ls", [(2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0)], ids=["one", "multi"])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6, 7, 8, 9])
def test_follows_the_oracle_and_resumes(qmin, oracle, m, Ls):
    s = system(oracle, Ls=Ls)
    lat, split = (gpu_lattice(qmin, s, qmin.FP32) for _ in range(2))
    ro = s.lbfgs(29, eta=5e-4, m=m)
    r = lat.lbfgs_run(29, eta=5e-4, m=m)
    assert r["iterations"] == 29
    assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-4 * ro["forceMax"]
    Q, _, F = lat.get_state(Q=True, F=True)
    assert rel_err(Q, s.Q) <= 1e-4
    assert split.lbfgs_run(3, eta=5e-4, m=m)["iterations"] == 3
    assert split.lbfgs_run(12, eta=5e-4, m=m, reset=False)["iterations"] == 12
    assert split.lbfgs_run(29, eta=5e-4, m=m, reset=False) == r
    for x, y in zip(split.get_state(Q=True, F=True), (Q, None, F)):
        if y is not None:
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("run", ["adam", "nesterov", "gd", "lbfgs"])
def test_forces_after_a_part_of_a_chunk(qmin, oracle, run, prec):
    s = system(oracle)
    lat = gpu_lattice(qmin, s, prec)
    getattr(lat, run + "_run")(5)
    F = lat.get_state(Q=False, F=True)[2]
    np.testing.assert_array_equal(F, lat.force())
