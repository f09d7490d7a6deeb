"""Kernels at the sizes where their tiling can go wrong: edges of tiles,
remainders, the smallest and largest of each dispatch range, against the oracle
or a plain FP64 restatement."""
import ctypes as ct

import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 31, 32, 33, 45, 46, 64, 65, 4096, 9728, 9729, 20001])
def test_training_gradient_at_tile_edges(bem, B):
    """Tiles of 32 samples, one CTA below 46 samples (room for two partial
    gradients), several tiles per CTA above 9,728. FP32 sums of B terms: 1e-5
    of the gradient's norm, as for a single size elsewhere."""
    torch = pytest.importorskip("torch")
    from oracle import mlp
    rng = np.random.default_rng(B)
    p = mlp.init(5).astype(np.float32)
    X = rng.standard_normal((B, 24)).astype(np.float32)
    y = rng.integers(0, 5, B).astype(np.uint8)
    pd, Xd, yd = (torch.from_numpy(a).cuda() for a in (p, X, y))
    # guard values behind the work area: the partial gradients stay inside it
    work = torch.full((B * 265 + 64,), 7.0, device="cuda")
    g = torch.zeros(6085, device="cuda")
    loss = torch.zeros(1, device="cuda")
    ptr = [ct.c_void_p(t.data_ptr()) for t in (pd, Xd, yd, g, loss, work)]
    got = []
    for _ in range(2):
        assert bem.lib().bem_mlp_grad(ptr[0], ptr[1], ptr[2], B, ptr[3], ptr[4], ptr[5], None) == 0
        torch.cuda.synchronize()
        got.append(g.cpu().numpy().copy())
    assert np.array_equal(got[0], got[1])
    assert (work[B * 265:] == 7.0).all()
    ref = mlp.grad(p.astype(np.float64), X.astype(np.float64), y.astype(int))
    assert np.linalg.norm(got[0] - ref) < 1e-5 * np.linalg.norm(ref)
    assert abs(float(loss.item()) - mlp.loss(p.astype(np.float64), X, y.astype(int))) < 1e-5
