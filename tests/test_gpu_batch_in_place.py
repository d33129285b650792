"""An FP32 multi-constant batch without room for a second state set (the
allocations of its planes answer out of memory) runs in place: solves of uneven
boxes, near walls and spheres, retire at the oracle's iteration counts with its
forceMax and Q, within the bounds of every FP32 batch (1e-4 and 2e-5); with room
again the same batch runs on two sets to the same bounds."""
import pytest

import malloc_shim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("passed", [0, 2])
def test_no_room_for_a_second_set(qmin, oracle, tmp_path, passed):
    malloc_shim.run(f"""
        from test_gpu_batch_retire import CUTOFF, MOST, systems
        ss = systems(oracle, (2.32, 1.0, 0.5, 0, 0))
        starts = [s.Q.copy() for s in ss]
        runs = [s.fire(MOST, fcut=CUTOFF) for s in ss]
        b = qmin.Batch([s.L for s in ss], qmin.FP32)
        p = ss[0].p
        b.set_params(p.A, p.B, p.C, p.L1, p.L2, p.L3, p.L4, multi_constant=p.multi_constant)
        b.set_chunk_shape(0)  # the tuner has a copy of V, as large
        planes = sizes()[0]
        assert planes >= 20 * sum(s.N for s in ss) and sizes().count(planes) == 3, "Q, V, F"
        for room in (False, False, True):
            since = shim.shim_made()
            shim.shim_fail(planes, planes, {passed}, 0 if room else 100)
            for k, s in enumerate(ss):
                b.set_solve(k, starts[k], s.types, [(s.objs[j].kind, s.objs[j].W, s.objs[j].S0) for j in range(s.nobj)])
            b.fire_init(force_cutoff=CUTOFF)
            r = b.fire_run(MOST)
            assert sizes(since).count(planes) == 3, "the second set, asked for at each run until there is one"
            assert r["iterations"].tolist() == [x["iterations"] for x in runs]
            for k, s in enumerate(ss):
                assert abs(r["forceMax"][k] - runs[k]["forceMax"]) <= 1e-4 * runs[k]["forceMax"], (room, k)
                assert rel_err(b.get_solve(k), s.Q) <= 2e-5, (room, k)
        b.close()
    """, tmp_path)
