"""H-matrix products: the launch shapes of small and large meshes, and the error
of the complex-FP32 arithmetic."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _product(bem, s, which, x, arith, acc=None):
    torch = pytest.importorskip("torch")
    y = torch.full_like(x, np.nan) if acc is None else acc.clone()
    torch.cuda.synchronize()
    assert bem.lib().bem_hmatvec_device_ex(s._h, which, ct.c_void_p(x.data_ptr()),
                                           ct.c_void_p(y.data_ptr()), x.shape[0],
                                           int(acc is not None), arith) == 0
    torch.cuda.synchronize()
    return y


def _waves(torch, rng, shape):
    return torch.from_numpy(rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).cuda()


@pytest.mark.parametrize("n,leaves", [(1283, (190, 608)), (3500, (608, 10**9))])
@pytest.mark.parametrize("precision", [0, 1])
def test_products_with_one_and_two_ctas_per_leaf(bem, meshes, n, leaves, precision):
    """Leaves of fewer than 8 rows: on 152 SMs a leaf of the smaller mesh takes a
    cluster of two CTAs, one of the larger mesh a single CTA. Products against the
    dense expansion of the stored blocks; tolerances as for the other shapes (FP64
    and two-float sums 1e-12, FP32 products 2e-6)."""
    torch = pytest.importorskip("torch")
    tri = meshes.box(n_target=n, seed=5)[:n]
    n = tri.shape[0]
    s = bem.Solver(precision=precision, leaf_size=8, aca_tol=1e-5, wave_speed=343.0, density=1.2,
                   near_fp64=0)
    s.set_mesh(tri)
    s.set_bc(np.zeros(n), np.ones(n))
    s.assemble(500.0)
    info = s.partition()
    rows = np.unique(info[info[:, 4] == 0][:, 0])  # every leaf has its own near block
    assert leaves[0] <= len(rows) < leaves[1]
    rng = np.random.default_rng(n)
    D = torch.from_numpy(s.dense(1)).cuda()
    for R in (1, 2, 3, 4, 8):
        x, y0 = _waves(torch, rng, (R, n)), _waves(torch, rng, (R, n))
        ref = (D @ x.T).T
        for arith, tol in ((0, 1e-12), (1, 2e-6), (2, 1e-12))[:1 if precision == 0 else 3]:
            for acc in (None, y0):
                want = ref if acc is None else ref + acc
                err = torch.linalg.vector_norm(_product(bem, s, 1, x, arith, acc) - want, dim=1)
                assert (err < tol * torch.linalg.vector_norm(want, dim=1)).all(), (R, arith)
    s.close()


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("R", [1, 3, 4, 8])
def test_fp32_product_error(bem, meshes, which, R):
    """The complex-FP32 product of the 20,480-element sphere against FP64 products
    of the same stored matrix. Sums that start anew with every block are 0.99e-7 to
    1.02e-7 off; sums over the columns of many blocks have to be as close."""
    torch = pytest.importorskip("torch")
    tri = meshes.icosphere(5, 1.0)
    n = tri.shape[0]
    s = bem.Solver(precision=1, aca_tol=1e-5, wave_speed=343.0, density=1.2)
    s.set_mesh(tri)
    s.set_bc(np.zeros(n), np.ones(n))
    s.assemble(1500.0)
    x = _waves(torch, np.random.default_rng(R), (R, n))
    ref = _product(bem, s, which, x, 0)
    err = torch.linalg.vector_norm(_product(bem, s, which, x, 1) - ref)
    assert err < 1.02e-7 * torch.linalg.vector_norm(ref)
    s.close()
