"""Which strategies an FP32 one-constant lattice chooses among: with listed sites
all of them are candidates (a wall every five planes makes two sites of five
listed, and the split path, the fastest without objects, is then the slowest).
Timing them leaves the state as it was: the run agrees with the oracle to the
FP32 bounds, the second of two runs too."""
import pytest

from cases import gpu_lattice, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [0, 5, 48])
def test_choice_among_all(qmin, oracle, every):
    s = oracle.System((34, 40, 48), Ls=(2.32, 0, 0, 0, 0))
    s.random_nematic(6)
    for plane in range(0, 48, every) if every else ():
        s.add_wall(2, plane, 0, 5.3)
    qmin.lib().qmin_tuning_cache_clear()
    lat = gpu_lattice(qmin, s, qmin.FP32)
    lat.fire_init()
    r, ro = lat.fire_run(6), s.fire(6)
    ms = lat.fire_tuning()["candidates_ms"]
    timed = {k.split("_")[0] for k in ms}
    assert timed == ({"separate", "fused", "tiled", "split"} if every else {"separate", "split"}), ms
    assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-4 * ro["forceMax"]
    assert rel_err(lat.get_state()[0], s.Q) <= 2e-5
    lat.fire_init()
    r, ro = lat.fire_run(5), s.fire(5)
    assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-4 * ro["forceMax"]
    assert rel_err(lat.get_state()[0], s.Q) <= 2e-5
    lat.close()
    qmin.lib().qmin_tuning_cache_clear()
