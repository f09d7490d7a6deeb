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


@pytest.mark.parametrize("M", [1, 63, 65, 997, 4095, 4097])
@pytest.mark.parametrize("freq", [300.0, 2500.0, 9000.0])
def test_field_at_tile_edges(bem, meshes, orc, M, freq):
    """Point tiles of 64 and 256, short element chunks, and the three forms of
    the FP64 phase (k rho below 0.35, below 1 and above, rho ~ 0.02 m). FP64
    differs from the oracle by the rounding of k r (about 200 at most): 1e-11
    norm-wise; FP32 integrand 2e-5."""
    tri = meshes.box(n_target=1200, seed=7)[:-3]
    n = tri.shape[0]
    rng = np.random.default_rng(M)
    phi = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    dphi = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    pts = rng.uniform(-0.4, 0.8, (M, 3))
    some = np.unique(np.r_[0, M - 1, rng.integers(0, M, 40)])  # points the oracle evaluates
    ref, _ = orc.field(tri, freq, pts[some], phi, dphi, c=343.0, rho=1.2)
    for precision, tol in ((0, 1e-11), (1, 2e-5)):
        s = bem.Solver(precision=precision, wave_speed=343.0, density=1.2)
        s.set_mesh(tri)
        pf, _ = s.field(freq, pts, phi, dphi)
        assert rel(pf[some], ref) < tol
        assert np.isfinite(pf).all()
        s.close()


@pytest.mark.parametrize("body,n,leaf", [("box", 12, 32), ("box", 320, 32), ("box", 323, 64),
                                         ("box", 1283, 100), ("sphere", 1280, 24),
                                         ("pencil", 2560, 32)])
def test_products_at_tile_edges(bem, meshes, body, n, leaf):
    """H-matrix products of 1 to 11 vectors in every arithmetic against the
    dense expansion of the stored blocks: no admissible block, leaves above 32
    rows, rows beyond 256 columns, odd sizes. FP64 and two-float sums of up to
    2,560 terms: 1e-12 norm-wise; FP32 products (6e-8 each): 2e-6."""
    torch = pytest.importorskip("torch")
    tri = {"box": lambda: meshes.box(n_target=max(n, 12), seed=5)[:n],
           "sphere": lambda: meshes.icosphere(3, 1.0),
           "pencil": lambda: meshes.pencil(n_target=n)}[body]()
    n = tri.shape[0]
    rng = np.random.default_rng(n)
    for precision in (0, 1):
        s = bem.Solver(precision=precision, leaf_size=leaf, aca_tol=1e-5, wave_speed=343.0,
                       density=1.2, near_fp64=0)
        s.set_mesh(tri)
        s.set_bc(np.zeros(n), np.ones(n))
        s.assemble(500.0)
        D = torch.from_numpy(s.dense(1)).cuda()
        for R in (1, 2, 3, 4, 5, 7, 8, 11):
            x = torch.from_numpy(rng.standard_normal((R, n)) + 1j * rng.standard_normal((R, n))).cuda()
            y0 = torch.from_numpy(rng.standard_normal((R, n)) + 0j).cuda()
            ref = (D @ x.T).T
            for arith, tol in ((0, 1e-12), (1, 2e-6), (2, 1e-12)):
                if precision == 0 and arith:
                    continue
                for acc in (0, 1):
                    y = y0.clone() if acc else torch.full_like(x, np.nan)
                    torch.cuda.synchronize()
                    assert bem.lib().bem_hmatvec_device_ex(
                        s._h, 1, ct.c_void_p(x.data_ptr()), ct.c_void_p(y.data_ptr()), R, acc,
                        arith) == 0
                    torch.cuda.synchronize()
                    want = ref + y0 if acc else ref
                    err = torch.linalg.vector_norm(y - want, dim=1)
                    assert (err < tol * torch.linalg.vector_norm(want, dim=1)).all(), (R, arith, acc)
        s.close()


@pytest.mark.parametrize("n,leaf,rank", [(12, 32, 2), (36, 32, 2), (300, 32, 2), (701, 20, 3),
                                         (1283, 32, 2), (2600, 28, 5)])
@pytest.mark.parametrize("precision", [0, 1])
def test_substitution_at_super_edges(bem, meshes, orc, n, leaf, rank, precision):
    """The dataflow sweeps against the oracle's leaf-by-leaf solves with one
    diagonal block, several, ragged ones, and 1 to 11 right-hand sides (1, 2, 4
    and 8 per pass, remainders). FP64 factors: rounding times the conditioning of
    the diagonal blocks, 1e-11; FP32 factors: 1e-4, as for the other FP32 sweep
    test. One right-hand side does not depend on the others beside it."""
    tri = meshes.box(n_target=max(n, 12), seed=3)[:n]
    n = tri.shape[0]
    s = bem.Solver(aca_tol=1e-6, precision=precision, precond_rank=rank, leaf_size=leaf)
    s.set_mesh(tri)
    s.set_bc(np.zeros(n), np.ones(n))
    s.assemble(300.0)
    s.hlu_build()
    assert s.hlu_sweep_kind() == 1
    Ll, Ld, _ = s.hlu_export(0)
    Ul, Ud, _ = s.hlu_export(1)
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, 11)) + 1j * rng.standard_normal((n, 11))
    ref = np.stack([orc.upper_solve(n, Ul, Ud, orc.lower_solve(n, Ll, Ld, B[:, q]))
                    for q in range(11)], axis=1)
    for R in (1, 2, 3, 5, 8, 11):
        X = s.hlu_solve(B[:, :R])
        for q in range(R):
            assert rel(X[:, q], ref[:, q]) < (1e-11, 1e-4)[precision], (R, q)
    s.close()


@pytest.mark.parametrize("n", [12, 130, 1300])
@pytest.mark.parametrize("restart", [4, 300, 1600])
def test_gmres_cycles_against_dense(bem, meshes, n, restart):
    """GMRES against the dense solve of the assembled matrix: short cycles, one
    cycle, cycles too long for the triangular solve's shared memory; one and
    three right-hand sides, one of them zero. The relative residual is below
    1e-10, so the error is below that times the conditioning (~1e2): 1e-7."""
    tri = meshes.box(n_target=max(n, 12), seed=9)[:n]
    n = tri.shape[0]
    s = bem.Solver(aca_tol=1e-7, gmres_tol=1e-10, gmres_restart=restart, gmres_maxit=1600)
    s.set_mesh(tri)
    s.set_bc(np.zeros(n), np.ones(n))
    s.assemble(400.0)
    A = s.dense(1)
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    B[:, 1] = 0.0
    x1, i1 = s.gmres(B[:, 0])
    x3, i3 = s.gmres(B)
    ref = np.linalg.solve(A, B)
    assert i1["status"] == 0 and i3["status"] == 0
    assert rel(x1, ref[:, 0]) < 1e-7
    assert rel(x3, ref) < 1e-7 and np.abs(x3[:, 1]).max() == 0.0
    assert rel(A @ x1, B[:, 0]) < 1.1e-10
    s.close()


@pytest.mark.parametrize("freq", [200.0, 440.0, 1400.0])
@pytest.mark.parametrize("wall", ["rigid", "soft", "mixed"])
def test_fp64_entries_in_each_phase_range(bem, meshes, orc, freq, wall):
    """Near-field blocks (regular, near-singular and singular rules) with the
    three forms of the phase (k rho below 0.35, below 1 and above; rho ~ 0.08 m)
    and columns that need one or both pairs of operators. Differences from the
    oracle are the rounding of k r (60 at most) and of the terms of N, which
    cancel by less than 1e3: 1e-12 of a block's largest entry. The far blocks
    together hold theirs to a hundred times the ACA tolerance."""
    tri = meshes.icosphere(3, 1.0)[:-1]
    n = tri.shape[0]
    i = np.arange(n)
    a = {"rigid": 0 * i, "soft": 1 + 0 * i, "mixed": (i % 3 == 1) * 0.7j + (i % 3 == 2) * 2.0}[wall] + 0j
    b = {"rigid": 1 + 0 * i, "soft": 0 * i, "mixed": 1 + 0 * i}[wall] + 0j
    s = bem.Solver(leaf_size=32, aca_tol=1e-6, wave_speed=343.0)
    s.set_mesh(tri)
    s.set_bc(a, b)
    s.assemble(freq)
    P = orc.Problem(tri, 32, s.config.eta)
    perm = P.perm
    exact = P.dense(2 * np.pi * freq / 343.0, s.config.coupling, a[perm], b[perm])
    info = s.partition()
    for which in (0, 1):
        D = s.dense(which)
        far = np.zeros(2)
        for r0, m, c0, nn, adm in info:
            ref = exact[which][r0:r0 + m, c0:c0 + nn]
            got = D[r0:r0 + m, c0:c0 + nn]
            if adm:
                far += [np.linalg.norm(got - ref) ** 2, np.linalg.norm(ref) ** 2]
            else:
                assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()
        assert far[0] < 1e-8 * far[1]
    s.close()


@pytest.mark.parametrize("n", [1, 3, 31, 32, 33, 64])
@pytest.mark.parametrize("precision", [0, 1])
def test_leaf_factorization_sizes(bem, meshes, n, precision):
    """One diagonal leaf: its factors are exact, below and above the 32 rows that
    fit in registers. Rounding times a condition number of at most 1e3: 1e-11
    with FP64 factors, 1e-4 with FP32 ones."""
    tri = meshes.box(n_target=200, seed=5)[:n]
    s = bem.Solver(precision=precision, precond_rank=2, leaf_size=64)
    s.set_mesh(tri)
    s.set_bc(np.zeros(n), np.ones(n))
    s.assemble(300.0)
    s.hlu_build()
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    assert rel(s.hlu_solve(s.hmatvec(1, x)).ravel(), x) < (1e-11, 1e-4)[precision]
    s.close()
