"""The tcgen05 weight gradient of the 3^3 convolutions (tensor path 1) against
the mma.sync one (path 0), layer by layer: rows of one and of several 64-voxel
segments, the last one cut at 8 to 56 voxels, the smallest grid, several
samples.  Both sum the same BF16 products in FP32, after passes whose
activations differ by their own rounding: the bound of the layer-wise
comparison with FP64 (6e-2 normwise, cosine 0.998)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L", [(1, (8, 8, 8)), (2, (72, 24, 16)), (1, (136, 8, 16)), (3, (56, 40, 8)), (1, (64, 32, 24)),
                                 (1, (248, 16, 8))])
def test_layers_match_mma_sync(qmin, B, L):
    rng = np.random.default_rng(3)
    n = L[0] * L[1] * L[2]
    x = torch.as_tensor(rng.standard_normal((B, n, 16)).astype(np.float32) * 0.5).cuda()
    tgt = torch.as_tensor((0.3 * rng.standard_normal((B, n, 5))).astype(np.float32)).cuda()
    grads = []
    for path in (0, 1):
        net = qmin.WarmNet(B, L, train=True)
        p = np.random.default_rng(17).standard_normal(net.get_params().size).astype(np.float32) * 0.05
        net.set_params(p)
        net.set_tensor_path(path)
        xv, _y, m = net.torch_views()
        xv.copy_(x.reshape(xv.shape))
        m.fill_(1)
        torch.cuda.synchronize()
        net.forward()
        net.backward(tgt.data_ptr())
        grads.append(net.get_params(grads=True)[1].astype(np.float64))
        net.close()
    for i, (ws, _bs, spec) in enumerate(qmin.warmnet_param_slices()):
        a, b = grads[1][ws], grads[0][ws]
        rel = np.linalg.norm(a - b) / np.linalg.norm(b)
        assert rel <= 6e-2 and a @ b >= 0.998 * np.linalg.norm(a) * np.linalg.norm(b), (i, spec, rel)
