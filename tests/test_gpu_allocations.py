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
        lat.set_fire_kernel(qmin.FIRE_SPLIT)
        lat.fire_init()
        r, ro = lat.fire_run(9), s.fire(9)
        assert lat.fire_tuning()["path"] == "split"
        assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-9 * ro["forceMax"]
        assert sum(n >= planes for n in sizes()) == 7, "the second set"
        Q, V, F = lat.get_state(V=True, F=True)
        assert rel_err(Q, s.Q) <= 1e-9 and rel_err(F, s.force()) <= 1e-9
    """, tmp_path)


def test_no_room_for_the_fixed_point_form(qmin, oracle, tmp_path):
    """A one-constant FP64 handle without the fixed-point form (the allocation of
    its flags answers out of memory) runs the FP64 kernels, also after a handle of
    the same shape has left the fixed-point strategy in the process."""
    malloc_shim.run("""
        def system():
            s = oracle.System((33, 17, 21), Ls=(2.32, 0, 0, 0, 0))
            s.random_nematic(4)
            s.add_wall(2, 0, 0, 5.3)
            return s
        for room in (True, False, True):
            s = system()
            lat = gpu_lattice(qmin, s, qmin.FP64)
            lat.set_fire_kernel(qmin.FIRE_SPLIT)  # the separate kernels where there is none
            shim.shim_fail(8, 8, 0, 0 if room else 1000)
            lat.fire_init()
            r, ro = lat.fire_run(9), s.fire(9)
            shim.shim_fail(8, 8, 0, 0)
            assert lat.fire_tuning()["path"] == ("split" if room else "separate"), (room, lat.fire_tuning())
            assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-9 * ro["forceMax"]
            assert rel_err(lat.get_state()[0], s.Q) <= 1e-9
            lat.close()
    """, tmp_path)


def test_checkpoint_into_a_handle_with_a_field_map(qmin, oracle, tmp_path):
    """The strategy of a checkpoint that a handle cannot launch (fixed point under
    a spatially varying field) is tuned afresh."""
    import numpy as np

    from cases import gpu_lattice, rel_err
    s = oracle.System((33, 17, 21), Ls=(2.32, 0, 0, 0, 0))
    s.random_nematic(4)
    s.add_wall(2, 0, 0, 5.3)
    a, b = gpu_lattice(qmin, s, qmin.FP64), gpu_lattice(qmin, s, qmin.FP64)
    H = np.random.default_rng(2).standard_normal((s.N, 3))
    a.set_field_map(H, 1.0, 1.0, 0.5)
    a.set_field_map(None, 1.0, 1.0, 0.5)  # off; the field constants are part of a checkpoint
    a.set_fire_kernel(qmin.FIRE_SPLIT)
    a.fire_init()
    a.fire_run(5)
    assert a.fire_tuning()["path"] == "split"
    a.checkpoint_save(str(tmp_path / "c"))
    b.set_field_map(H, 1.0, 1.0, 0.5)
    b.checkpoint_load(str(tmp_path / "c"))
    s.fire(5)
    s.set_field_map(H, 1.0, 1.0, 0.5)
    b.fire_init()
    r, ro = b.fire_run(9), s.fire(9)
    assert b.fire_tuning()["path"] == "separate"
    assert abs(r["forceMax"] - ro["forceMax"]) <= 1e-9 * ro["forceMax"]
    assert rel_err(b.get_state()[0], s.Q) <= 1e-9


@pytest.mark.parametrize("precision", ["FP32", "FP64"])
@pytest.mark.parametrize("passed", [0, 1, 2])
def test_second_set_that_did_not_fit(qmin, oracle, tmp_path, precision, passed):
    """A run that found room for only some of the second set's planes answers
    QMIN_ENOMEM, and so does the next; with room the handle runs as ever."""
    malloc_shim.run(f"""
        L, passed, prec = (24, 9, 11), {passed}, qmin.{precision}
        s = oracle.System(L, Ls=(2.32, 1.0, 0.5, 0, 0))
        s.random_nematic(4)
        planes = 5 * (4 if prec == qmin.FP32 else 8) * (s.N + (-s.N) % 32)
        tol_f, tol_q = (1e-4, 2e-5) if prec == qmin.FP32 else (1e-9, 1e-9)
        lat = gpu_lattice(qmin, s, prec)
        for kind in ("lattice", "batch"):
            if kind == "lattice":
                run = lambda: (lat.fire_init(), lat.fire_run(7))[1]
                Q = lambda: lat.get_state()[0]
            elif prec == qmin.FP32:
                b = qmin.Batch([L], prec)
                s = oracle.System(L, Ls=(2.32, 0, 0, 0, 0))  # multi-constant batches run without it
                b.set_params(s.p.A, s.p.B, s.p.C, s.p.L1)
                b.set_chunk_shape(0)
                s.random_nematic(4)
                b.set_solve(0, s.Q, s.types, [])
                run = lambda: (b.fire_init(), b.fire_run(7))[1]
                Q = lambda: b.get_solve(0)
            else:
                continue
            for k in range(2):
                shim.shim_fail(planes, planes, passed if k == 0 else 0, 100)
                try:
                    run()
                    raise SystemExit("no error")
                except qmin.QminError as e:
                    assert e.code == qmin.QMIN_ENOMEM, e
            shim.shim_fail(planes, planes, 0, 0)
            r = run()
            ro = s.fire(7)
            f = r["forceMax"] if kind == "lattice" else r["forceMax"][0]
            assert abs(f - ro["forceMax"]) <= tol_f * ro["forceMax"]
            assert rel_err(Q(), s.Q) <= tol_q
    """, tmp_path)
