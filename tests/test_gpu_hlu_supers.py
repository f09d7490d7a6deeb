"""The dense inverses of the H-LU sweeps' diagonal blocks: what they hold where
the factors hold nothing, and how they are built beside other handles."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from conftest import ROOT, rel

pytestmark = pytest.mark.gpu


def _plate(n, axis):
    """2 n^2 triangles of the unit square through the origin normal to `axis`,
    with exact coordinates: no element sees another one of its own plate."""
    u, v = [a for a in range(3) if a != axis]
    g = np.arange(n + 1) / n
    tri = []
    for i in range(n):
        for j in range(n):
            c = np.zeros((4, 3))
            c[:, u] = g[[i, i + 1, i + 1, i]]
            c[:, v] = g[[j, j, j + 1, j + 1]]
            tri += [c[[0, 1, 2]].ravel(), c[[0, 2, 3]].ravel()]
    return np.array(tri)


def _factors(s):
    return [s.hlu_export(which)[:2] for which in (0, 1)]


def _leafwise(orc, factors, n, B):
    (Ll, Ld), (Ul, Ud) = factors
    return np.stack([orc.upper_solve(n, Ul, Ud, orc.lower_solve(n, Ll, Ld, B[:, q]))
                     for q in range(B.shape[1])], axis=1)


def _absent(factors, info, n, span):
    """Far blocks within `span` rows and columns of each other that no leaf of
    either factor covers."""
    held = np.zeros((n, n), bool)
    for leaves, _ in factors:
        for r0, m, c0, nn, *_ in leaves:
            held[r0:r0 + m, c0:c0 + nn] = True
    return sum(1 for r0, m, c0, nn, adm in info
               if adm and max(r0 + m, c0 + nn) - min(r0, c0) <= span
               and not held[r0:r0 + m, c0:c0 + nn].any())


@pytest.mark.parametrize("precision,rank", [(0, 8), (0, 2), (1, 2)])
def test_blocks_without_a_leaf_are_zero(bem, orc, precision, rank):
    """Rigid plates at a right angle, coupling 0: far blocks inside a plate are
    exactly zero, so the host factorization drops their leaves. One handle
    factorizes a full matrix (soft walls) first, then the rigid one at two
    frequencies: the sweeps are those of the factors (FP64 1e-11, FP32 1e-4, as
    for the other tests of the sweeps against the leaf-by-leaf solves)."""
    tri = np.vstack([_plate(24, 0), _plate(24, 2) + np.tile([0.25, 0.0, 0.0], 3)])
    n = tri.shape[0]
    s = bem.Solver(precision=precision, aca_tol=1e-6, leaf_size=32, coupling=0, hlu_device=0,
                   precond_rank=rank, precond_tol=1e-8)
    s.set_mesh(tri)
    rng = np.random.default_rng(4)
    B = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    for k, (a, b, freq) in enumerate([(1.0, 0.0, 300.0), (0.0, 1.0, 300.0), (0.0, 1.0, 500.0)]):
        s.set_bc(np.full(n, a), np.full(n, b))
        s.assemble(freq)
        s.hlu_build()
        assert s.hlu_sweep_kind() == 1
        factors = _factors(s)
        assert (_absent(factors, s.partition(), n, 128) > 0) == (k > 0)
        assert rel(s.hlu_solve(B), _leafwise(orc, factors, n, B)) < (1e-11, 1e-4)[precision], k
    s.close()


def test_factorizations_in_threads(bem, meshes):
    """Factors of a body with diagonal blocks of hundreds of rows while other
    threads factorize a tiny one: a launch's shared memory does not depend on
    what other handles launched last."""
    def handle(tri):
        s = bem.Solver(precision=1, precond_rank=2, leaf_size=32, aca_tol=1e-5)
        s.set_mesh(tri)
        s.set_bc(np.zeros(len(tri)), np.ones(len(tri)))
        s.assemble(300.0)
        return s

    large = handle(meshes.icosphere(3, 1.0))
    small = [handle(meshes.box(n_target=12, seed=3)[:12]) for _ in range(3)]
    done, errors = threading.Event(), []

    def rebuild(s):
        try:
            while not done.is_set():
                s.hlu_build()
        except Exception as e:  # noqa: BLE001 -- reported below
            errors.append(e)

    threads = [threading.Thread(target=rebuild, args=(s,)) for s in small]
    for t in threads:
        t.start()
    try:
        for _ in range(200):
            large.hlu_build()
    except Exception as e:  # noqa: BLE001
        errors.append(e)
    done.set()
    for t in threads:
        t.join()
    assert not errors
    for s in (large, *small):
        s.close()


def test_sweeps_without_room_for_inverses(tmp_path):
    """With less device memory than the inverses take (a cap on the library's
    allocations, in child processes) the factors are built all the same and the
    leaf-by-leaf sweeps solve with them. The least cap that is enough is found
    by bisection; there the inverses have no room."""
    code = r"""
import importlib, sys, numpy as np
sys.path.insert(0, sys.argv[1])
bem = importlib.import_module("3d_bem_gb300")
meshes = importlib.import_module("3d_bem_gb300.meshes")
tri = meshes.icosphere(3, 1.0); n = tri.shape[0]
s = bem.Solver(precision=0, aca_tol=1e-5, precond_rank=2, leaf_size=32)
s.set_mesh(tri); s.set_bc(np.zeros(n), np.ones(n))
try:
    s.assemble(300.0); s.hlu_build()
    b = np.random.default_rng(1).standard_normal(n) + 0j
    x = s.hlu_solve(b)
except bem.BemError as e:
    print("STATUS", e.status)
else:
    np.save(sys.argv[2], x)
    print("KIND", s.hlu_sweep_kind())
"""
    def run(mib):
        out = str(tmp_path / f"x{mib}.npy")
        env = dict(os.environ)
        env.pop("BEM_DEVICE_MEM_CAP", None)
        if mib:
            env["BEM_DEVICE_MEM_CAP"] = str(mib << 20)
        r = subprocess.run([sys.executable, "-c", code, ROOT, out], env=env, capture_output=True,
                           text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        word, value = r.stdout.split()
        if word == "STATUS":
            assert int(value) == 2  # BEM_ENOMEM
            return None, None
        return int(value), np.load(out)

    kind, x = run(0)
    assert kind == 1
    lo, hi = 0, 512
    while hi - lo > 2:
        mid = (lo + hi) // 2
        if run(mid)[0] is None:
            lo = mid
        else:
            hi = mid
    kind, y = run(hi)
    assert kind == 0
    assert rel(y, x) < 1e-11


def test_inverses_in_batches(bem, meshes, orc):
    """40,960 elements: the dense blocks of all supers (about 13 million values)
    are inverted in two batches. FP32 factors: 1e-4, as for the other tests."""
    tri = meshes.pencil(n_target=40960)
    n = tri.shape[0]
    s = bem.Solver(precision=1, aca_tol=1e-4, precond_rank=2, leaf_size=32, wave_speed=343.0)
    s.set_mesh(tri)
    s.set_bc_impedance(meshes.wall_admittance(n))
    s.assemble(1000.0)
    s.hlu_build()
    assert s.hlu_sweep_kind() == 1
    rng = np.random.default_rng(2)
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    assert rel(s.hlu_solve(B), _leafwise(orc, _factors(s), n, B)) < 1e-4
    s.close()


@pytest.mark.parametrize("body", ["sphere", "box", "pencil"])
def test_fp32_sweeps_as_accurate_as_leaf_by_leaf(bem, meshes, orc, body):
    """8 vectors through FP32 factors against the exact solve with the same
    factors. Substitution leaf by leaf in complex FP32, in the order of the
    schedule, is 1.28e-7 to 1.33e-7 off on these bodies: products with the
    inverses have to be as close."""
    tri = {"sphere": lambda: meshes.icosphere(3, 1.0),
           "box": lambda: meshes.box(n_target=1280, exact=True),
           "pencil": lambda: meshes.pencil(n_target=20480)}[body]()
    n = tri.shape[0]
    s = bem.Solver(precision=1, aca_tol=1e-5, precond_rank=2, wave_speed=343.0, density=1.2)
    s.set_mesh(tri)
    if body == "pencil":
        s.set_bc_impedance(meshes.wall_admittance(n))
    else:
        s.set_bc(np.zeros(n), np.ones(n))
    s.assemble({"sphere": 300.0, "box": 700.0, "pencil": 1500.0}[body])
    s.hlu_build()
    assert s.hlu_sweep_kind() == 1
    rng = np.random.default_rng(3)
    B = rng.standard_normal((n, 8)) + 1j * rng.standard_normal((n, 8))
    X, ref = s.hlu_solve(B), _leafwise(orc, _factors(s), n, B)
    assert np.linalg.norm(X - ref) < 1.33e-7 * np.linalg.norm(ref)
    s.close()


def test_sweep_trace(bem, meshes, tmp_path, monkeypatch):
    """BEM_DF_TRACE: one line per lower sweep of up to 8 vectors, and the same
    solution."""
    tri = meshes.icosphere(3, 1.0)
    n = tri.shape[0]
    s = bem.Solver(precision=1, aca_tol=1e-5, precond_rank=2)
    s.set_mesh(tri)
    s.set_bc(np.zeros(n), np.ones(n))
    s.assemble(300.0)
    s.hlu_build()
    rng = np.random.default_rng(6)
    B = rng.standard_normal((n, 9)) + 1j * rng.standard_normal((n, 9))
    X = s.hlu_solve(B)
    path = tmp_path / "sweeps.txt"
    monkeypatch.setenv("BEM_DF_TRACE", str(path))
    assert np.array_equal(s.hlu_solve(B), X)
    monkeypatch.delenv("BEM_DF_TRACE")
    lines = path.read_text().split("\n")[:-1]
    assert len(lines) == 2
    for line, R in zip(lines, (8, 1)):
        assert line.startswith("df L sweep: levels ") and f" R {R} " in line
        words = line.split()
        levels, total = int(words[words.index("levels") + 1]), float(words[words.index("total_us") + 1])
        per = [float(words[words.index(w) + 1]) for w in ("row", "diag", "dot")]
        assert levels > 1 and all(0 < v < 1e4 for v in per)
        assert total == pytest.approx(levels * sum(per), rel=0.01)
    s.close()


def test_sweep_trace_of_a_solve(bem, meshes, tmp_path, monkeypatch):
    """BEM_DF_TRACE in a preconditioned solve: the sweeps of its GMRES steps are
    traced too, those launched after convergence leave no line."""
    tri = meshes.icosphere(2, 1.0)
    n = tri.shape[0]
    s = bem.Solver(aca_tol=1e-5, gmres_tol=1e-9, use_preconditioner=1, precond_rank=2)
    s.set_mesh(tri)
    s.set_bc(np.zeros(n), np.ones(n))
    p = s.solve(300.0, np.ones(n))[2]
    path = tmp_path / "sweeps.txt"
    monkeypatch.setenv("BEM_DF_TRACE", str(path))
    q, info = s.solve(300.0, np.ones(n))[2:]
    monkeypatch.delenv("BEM_DF_TRACE")
    assert np.array_equal(p, q)
    lines = path.read_text().split("\n")[:-1]
    assert len(lines) >= info["iterations"] + 1  # the right-hand side and every step
    assert all(float(x.split("total_us")[1].split()[0]) > 0 for x in lines)
    s.close()
