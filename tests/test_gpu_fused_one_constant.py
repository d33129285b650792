"""One-constant FP32 lattices through the split fused iteration (boundary sites
listed, the bulk on tiles): against the oracle within FP32 accuracy (1e-4 in
forceMax, 2e-5 in Q, as every FP32 FIRE path) on lattices smaller than a tile,
not a multiple of one and larger, with and without listed sites, and a resumed
run within the same bounds."""
import pytest

from cases import gpu_lattice, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,objects", [((3, 3, 3), False), ((5, 4, 7), False), ((33, 29, 31), True), ((64, 9, 17), True),
                                       ((70, 66, 6), False)])
def test_follows_the_oracle_and_resumes(qmin, oracle, L, objects):
    s = oracle.System(L, Ls=(2.32, 0, 0, 0, 0))
    s.random_nematic(13)
    if objects:
        s.add_wall(2, 0, 0, 5.3)
        s.add_sphere(tuple(0.5 * x for x in L), 2.2, 1, 2.0)
    lat, split = (gpu_lattice(qmin, s, qmin.FP32) for _ in range(2))
    ro = s.fire(13)
    for x in (lat, split):
        x.set_fire_kernel(qmin.FIRE_SPLIT)
        x.fire_init()
    r = lat.fire_run(13)
    assert lat.fire_tuning()["path"] == "split"
    assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-4 * ro["forceMax"]
    Q = lat.get_state()[0]
    assert rel_err(Q, s.Q) <= 2e-5
    split.fire_run(6)
    r2 = split.fire_run(13)
    assert r2["iterations"] == r["iterations"] == 13
    assert abs(r2["forceMax"] - r["forceMax"]) <= 1e-4 * ro["forceMax"]
    assert rel_err(split.get_state()[0], Q) <= 2e-5
