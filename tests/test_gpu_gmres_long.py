"""GMRES cycles of many hundred steps: the rotations and the triangular solve of
one cycle beyond what a thread prefetches and what fits in shared memory."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("restart", [1500, 1600])
def test_one_cycle_of_many_hundred_steps(bem, meshes, restart):
    """A box whose walls have admittances of random phase and magnitudes over ten
    orders: the dense restatement takes nearly as many steps as there are elements.
    Cycles that fit in the triangular solve's shared memory and that do not; two
    right-hand sides that end at different steps. The residual estimate has to be
    the true residual; the error is below 1e-10 times the conditioning (4e3), 1e-6."""
    tri = meshes.box(n_target=1100, seed=9)
    n = tri.shape[0]
    rng = np.random.default_rng(1)
    a = 7.0 * np.exp(3.0 * rng.standard_normal(n)) * np.exp(2j * np.pi * rng.random(n))
    s = bem.Solver(aca_tol=1e-7, gmres_tol=1e-10, gmres_restart=restart, gmres_maxit=1600,
                   use_preconditioner=0)
    s.set_mesh(tri)
    s.set_bc(a, np.ones(n))
    s.assemble(400.0)
    A = s.dense(1)
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    B[:, 1] = A @ np.eye(n)[3]  # a few hundred steps less
    x, info = s.gmres(B)
    assert info["status"] == 0
    assert 520 < info["iterations"] <= n
    true = np.linalg.norm(B - A @ x, axis=0) / np.linalg.norm(B, axis=0)
    assert true.max() < 1.1e-10
    assert rel(x, np.linalg.solve(A, B)) < 1e-6
    x1, info1 = s.gmres(B[:, 0])
    assert abs(info1["iterations"] - info["iterations"]) <= 1
    estimate, true1 = info1["rel_residual"], np.linalg.norm(B[:, 0] - A @ x1) / np.linalg.norm(B[:, 0])
    assert estimate < 1e-10 and abs(estimate - true1) < 1e-11
    s.close()
