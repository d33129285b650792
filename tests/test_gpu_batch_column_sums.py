"""FP32 batches add f.f, v.v and f.v of every site as exactly as FP64 would: on a
uniform field of one component without a cubic term every site has the same
force, and forceMax is that of N equal terms to 1e-12 (a plain FP32 sum over the
16 planes of an item is 1e-8 off)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [(40, 24, 50), (160, 152, 156)])
def test_sum_of_equal_terms(qmin, L):
    N = L[0] * L[1] * L[2]
    b = qmin.Batch([L], qmin.FP32)
    b.set_params(-0.172, 0.0, 1.73, 2.32)
    b.set_chunk_shape(0)
    Q = np.zeros((N, 5))
    Q[:, 1] = 0.2871
    b.set_solve(0, Q, np.zeros(N, dtype=np.int32), [])
    b.fire_init()
    r = b.fire_run(1)
    F = b.get_solve(0, F=True)[1].astype(np.float32)
    assert (F[:, 1] == F[0, 1]).all() and F[0, 1] != 0 and not F[:, [0, 2, 3, 4]].any()
    want = np.sqrt(N * np.float64(F[0, 1] * F[0, 1])) / N  # the term: an FP32 product, rounded once
    assert abs(r["forceMax"][0] - want) <= 1e-12 * want, r["forceMax"][0] / want - 1
    b.close()
