"""The strategy of an FP64 lattice does not hang on where its field is at the
first run: a quench from noise below the fixed-point range, and a field with one
value above it, take the strategy that a nematic start takes.  (96 x 80 x 88,
where the fixed-point force is more than twice as fast as any other candidate.)"""
import numpy as np
import pytest

from cases import gpu_lattice, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ls", [(2.32, 0, 0, 0, 0), (2.32, 1.0, 0.5, 0, 0)], ids=["one", "multi"])
@pytest.mark.parametrize("start", ["noise", "wide"])
def test_choice_outside_the_range(qmin, oracle, start, Ls):
    s = oracle.System((96, 80, 88), Ls=Ls)
    s.random_nematic(5)
    s.add_wall(2, 0, 0, 5.3)
    nematic = s.Q.copy()
    choices = []
    for field in ("nematic", start):
        s.Q[:] = nematic
        if field == "noise":
            s.Q[s.types <= 0] *= 1e-3
        elif field == "wide":
            s.Q[s.N // 2, 1] = 1.5
        qmin.lib().qmin_tuning_cache_clear()
        lat = gpu_lattice(qmin, s, qmin.FP64)
        lat.fire_init()
        r, ro = lat.fire_run(5), s.fire(5)
        t = lat.fire_tuning()
        choices.append((t["path"], t["variant"]))
        assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-9 * ro["forceMax"]
        assert rel_err(lat.get_state()[0], s.Q) <= 1e-9
        lat.close()
    qmin.lib().qmin_tuning_cache_clear()
    assert choices[0] == ("split", 0) and choices[1] == choices[0], choices
