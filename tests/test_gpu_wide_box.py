"""A flat box of more tiles than the usual buffer of per-block sums has places
(2048 x 2048 x 3: 16384 tiles of 32 x 8 or 16 x 16, one z chunk each, listed
sites beside them): the periodic repetition of a 32 x 16 x 3 lattice, whose
oracle run it follows within the bounds of every lattice path (FP64 1e-9, FP32
1e-4 in forceMax and 2e-5 in Q)."""
import numpy as np
import pytest

from cases import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,strategy,variant", [("FP32", "AUTO", None), ("FP32", "TILED", None), ("FP32", "SPLIT", 4),
                                                        ("FP32", "SPLIT", 9), ("FP64", "SPLIT", 2), ("FP64", "SPLIT", 0)])
def test_follows_the_small_lattice(qmin, oracle, precision, strategy, variant):
    s = oracle.System((32, 16, 3), Ls=(2.32, 1.0, 0.5, 0, 0))
    s.random_nematic(3)
    s.add_wall(2, 0, 0, 5.3)
    reps = (2048 // 16, 2048 // 32)

    def wide(a):
        a = a.reshape(3, 16, 32, -1)
        return np.ascontiguousarray(np.tile(a, (1, reps[0], reps[1], 1)).reshape(3 * 2048 * 2048, -1))

    lat = qmin.Lattice((2048, 2048, 3), getattr(qmin, precision))
    p = s.p
    lat.set_params(p.A, p.B, p.C, p.L1, p.L2, p.L3, p.L4, multi_constant=1)
    lat.set_objects([(s.objs[0].kind, s.objs[0].W, s.objs[0].S0)])
    lat.set_state(wide(s.Q), wide(s.types)[:, 0])
    lat.set_fire_kernel(getattr(qmin, "FIRE_" + strategy))
    if variant is not None:
        lat.set_fire_variant(variant)
    lat.fire_init()
    r, ro = lat.fire_run(4), s.fire(4)
    tol_f, tol_q = (1e-4, 2e-5) if precision == "FP32" else (1e-9, 1e-9)
    # forceMax is |F| / N: the root of the number of copies less
    assert abs(r["forceMax"] * np.sqrt(reps[0] * reps[1]) - ro["forceMax"]) <= tol_f * ro["forceMax"]
    Q = lat.get_state()[0].reshape(3, reps[0], 16, reps[1], 32, 5)
    got = np.stack([Q[:, 0, :, 0], Q[:, -1, :, -1], Q[:, 37, :, 11]])
    want = np.broadcast_to(s.Q.reshape(3, 16, 32, 5), got.shape)
    assert rel_err(got, want) <= tol_q
    lat.close()
