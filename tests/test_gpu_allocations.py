"""What a handle allocates and when, and what a call does when the device has no
room for it."""
import pytest

import malloc_shim

pytestmark = pytest.mark.gpu


def test_fixed_point_force_asks_for_no_planes(qmin, oracle, tmp_path):
    """Q 2^56 goes into the staging buffer of uploads: creation allocates the
    state alone, and neither a force evaluation nor a FIRE run any further
    planes but the tuner's second state set."""
    malloc_shim.run("""
        L = (50, 50, 50)
        s = oracle.System(L, Ls=(2.32, 0, 0, 0, 0))
        s.random_nematic(4)
        planes = 5 * 8 * (s.N + (-s.N) % 32)
        lat = qmin.Lattice(L, qmin.FP64)
        assert sum(n == planes for n in sizes()) == 3, "Q, V, F"
        lat.set_params(s.p.A, s.p.B, s.p.C, s.p.L1)
        lat.set_objects([])
        lat.set_state(s.Q, s.types)
        assert sum(n == planes for n in sizes()) == 4, "the staging buffer"
        assert rel_err(lat.force(), s.force()) <= 1e-12
        assert sum(n >= planes for n in sizes()) == 4
        lat.fire_init()
        r, ro = lat.fire_run(9), s.fire(9)
        assert lat.fire_tuning()["path"] == "split"
        assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-9 * ro["forceMax"]
        assert sum(n >= planes for n in sizes()) == 7, "the second set"
        Q, V, F = lat.get_state(V=True, F=True)
        assert rel_err(Q, s.Q) <= 1e-9 and rel_err(F, s.force()) <= 1e-9
    """, tmp_path)
