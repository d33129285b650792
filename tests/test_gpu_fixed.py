"""The FP64 form's fixed-point path (predictor with Q 2^56, deep-site force)
against the oracle: forces to 1e-12 normwise and FIRE to 1e-9, as every FP64
path, on the smallest and on odd boxes, for both metric modes and forms, with
fields and objects, and outside the fixed-point range, where the FP64 kernels
take over."""
import numpy as np
import pytest

from cases import gpu_lattice, rel_err

pytestmark = pytest.mark.gpu

ONE, MULTI = (2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0)


def system(oracle, L, Ls, metric_mode=0, objects=False, E=None, H=None, field="random"):
    s = oracle.System(L, Ls=Ls, metric_mode=metric_mode, E=E, H=H)
    s.random_nematic(11)
    rng = np.random.default_rng(5)
    if field == "small":
        s.Q *= 1e-3
    elif field == "wide":
        s.Q += 0.4 * rng.standard_normal(s.Q.shape)
    elif field == "one_wide":
        s.Q[s.Q.shape[0] // 2, 1] = 0.76
    elif field == "edge":
        s.Q[s.Q.shape[0] // 2] = [np.nextafter(0.75, 0), 0.1, -np.nextafter(0.75, 0), -0.2, 0.125]
    if objects:
        s.add_wall(2, 0, 0, 5.3)
        s.add_sphere(tuple(0.5 * x for x in L), 2.2, 1, 2.0)
    return s


@pytest.mark.parametrize("Ls", [ONE, MULTI], ids=["one", "multi"])
@pytest.mark.parametrize("L,objects", [((3, 3, 3), False), ((5, 3, 4), False), ((33, 29, 31), True), ((64, 3, 7), False),
                                       ((12, 40, 9), True)])
@pytest.mark.parametrize("metric_mode", [0, 1])
def test_force_and_fire(qmin, oracle, L, objects, Ls, metric_mode):
    s = system(oracle, L, Ls, metric_mode, objects, H=(0.3, 0.1, -0.4, 1.0, 1.0, 0.5))
    lat = gpu_lattice(qmin, s, qmin.FP64, metric_mode)
    assert rel_err(lat.force(), s.force()) <= 1e-12
    lat.set_fire_kernel(qmin.FIRE_SPLIT)
    if any(Ls[1:]):
        lat.set_fire_variant(0)
    lat.fire_init()
    r, ro = lat.fire_run(12), s.fire(12)
    assert lat.fire_tuning()["path"] == "split"
    assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-9 * ro["forceMax"]
    assert rel_err(lat.get_state()[0], s.Q) <= 1e-9


@pytest.mark.parametrize("Ls", [ONE, MULTI], ids=["one", "multi"])
@pytest.mark.parametrize("field", ["small", "wide", "one_wide", "edge"])
def test_range(qmin, oracle, field, Ls):
    s = system(oracle, (14, 11, 10), Ls, objects=True, field=field)
    lat = gpu_lattice(qmin, s, qmin.FP64)
    assert rel_err(lat.force(), s.force()) <= 1e-12
    lat.set_fire_kernel(qmin.FIRE_SPLIT)
    if any(Ls[1:]):
        lat.set_fire_variant(0)
    lat.fire_init()
    r, ro = lat.fire_run(6), s.fire(6)
    assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-9 * ro["forceMax"]
    Q, V, F = lat.get_state(V=True, F=True)
    assert rel_err(Q, s.Q) <= 1e-9
    # a field that enters and leaves the range from call to call
    lat.set_positions(0.2 * s.Q)
    F = lat.force()
    assert rel_err(F, s.force(0.2 * s.Q)) <= 1e-12
