"""One-constant FP32 iterations add f.f, v.v and f.v of every site as exactly as
FP64 would: on a uniform field of one component without a cubic term every site
has the same force, f.f is one rounded square, and forceMax is that of N equal
terms to 1e-12 (a plain FP32 sum over a column of 16 or more planes is 1e-8 off
and more)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", ["AUTO", "SPLIT", "SEPARATE", "FUSED", "TILED"])
@pytest.mark.parametrize("L", [(40, 24, 50), (96, 88, 90)])
def test_sum_of_equal_terms(qmin, L, strategy):
    N = L[0] * L[1] * L[2]
    lat = qmin.Lattice(L, qmin.FP32)
    lat.set_params(-0.172, 0.0, 1.73, 2.32)
    lat.set_objects([])
    Q = np.zeros((N, 5))
    Q[:, 1] = 0.2871
    lat.set_state(Q, np.zeros(N, dtype=np.int32))
    lat.set_fire_kernel(getattr(qmin, "FIRE_" + strategy))
    lat.fire_init()
    r = lat.fire_run(1)
    F = lat.get_state(F=True)[2].astype(np.float32)
    assert (F[:, 1] == F[0, 1]).all() and F[0, 1] != 0 and not F[:, [0, 2, 3, 4]].any()
    term = np.float64(F[0, 1] * F[0, 1])  # FP32 product, rounded once
    want = np.sqrt(N * term) / N
    assert abs(r["forceMax"] - want) <= 1e-12 * want, (lat.fire_tuning(), r["forceMax"] / want - 1)
    lat.close()
