"""The integrator's dense factorisation and solve on given matrices: the team
forms against the one-thread factorisation and the solve that divides, bit for
bit, at the edges of what the solve by reciprocals covers and beyond them; and
the adjoint's factorisation at species counts on either side of a warp."""

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = [pytest.mark.gpu, pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")]


@pytest.fixture(scope="module")
def lc(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("linear_checks") / "linear_checks.so")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-Xcompiler", "-fPIC",
                        "-shared", "-diag-suppress", "177,550", "-I", os.path.join(ROOT, "pelephysics_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "linear_checks.cu"), "-o", so], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(so)
    vp, i = C.c_void_p, C.c_int
    L.lc_factor_solve.argtypes = [i, i, i, vp, vp, i, i, vp, vp, vp, vp, vp]
    L.lc_adjoint.argtypes = [i, vp, C.c_double, i, vp, i, vp, vp]
    return L


def matrices(n, fp32, rng):
    """name -> matrix (A[i, j])."""
    unit = lambda: np.eye(n) + 0.3 * rng.normal(size=(n, n)) / np.sqrt(n)  # noqa: E731
    out = {"newton": unit(), "full": rng.normal(size=(n, n))}
    ties = np.sign(rng.normal(size=(n, n)))
    ties[0] = 1.0
    out["ties"] = ties + 2.0 * np.diag(rng.integers(0, 2, n))
    out["sparse"] = unit() * (rng.uniform(size=(n, n)) < 0.3) + np.eye(n)
    low = np.tril(unit())
    out["all ones"] = low * (1 - np.eye(n)) * 1e-2 + np.diag(np.full(n, 2.0 - 2.0 ** (-23 if fp32 else -52)))
    if not fp32:
        for e in (399, 401, -399, -401, 600, -600):
            a = np.tril(1e-3 * rng.normal(size=(n, n)), -1) + np.eye(n)
            a[:, n // 2] = 0.0
            a[n // 2, n // 2] = 2.0 ** e
            out[f"diagonal 2^{e}"] = a
    tiny = 1e-42 if fp32 else 1e-310  # its reciprocal is not finite
    a = unit()
    a[:, 0] = tiny * np.linspace(1.0, 0.1, n)
    a[0, 1::2] = 0.0
    out["multipliers not finite, half of the pivot row zero"] = a
    a = a.copy()
    a[0, 1:] = 0.0  # a zero times an infinite multiplier is left out of the update
    out["multipliers not finite, pivot row zero"] = a
    a = unit()
    a[n - 1, 0] = np.inf
    out["infinite entry"] = a
    a = unit()
    a[0, 0] = np.nan
    out["nan entry"] = a
    a = unit()
    a[:, n // 2] = 0.0
    out["zero column"] = a
    a = unit()
    a[:, 0] = np.nan
    out["nan column"] = a
    return out


def right_hand_sides(n, rng):
    b = [rng.normal(size=n), np.zeros(n), np.eye(n)[0], np.eye(n)[n - 1]]
    for e in (-499, -501, 499, 501, 1000, -1000, -1060):
        v = rng.normal(size=n)
        v[rng.integers(0, n)] *= 2.0 ** e
        b.append(v)
        b.append(rng.normal(size=n) * 2.0 ** e)
    for w in (np.inf, np.nan):
        v = rng.normal(size=n)
        v[n // 3] = w
        b.append(v)
    return np.array(b)


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("team,n", [(16, 10), (16, 22), (32, 10), (32, 22), (32, 32), (32, 33), (32, 54), (32, 89),
                                    (64, 54), (128, 54), (128, 89), (256, 89)])
def test_team_forms_give_the_one_thread_bits(cuda, lc, team, n, fp32):
    torch = cuda
    rng = np.random.default_rng(100 * n + team)
    mats = matrices(n, fp32, rng)
    A = np.array([m.T for m in mats.values()])  # column-major
    b = np.array([right_hand_sides(n, rng) for _ in mats])
    m, r = b.shape[:2]
    dev = lambda a, t: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device="cuda")  # noqa: E731
    empty = lambda *s, t=torch.float64: torch.zeros(s, dtype=t, device="cuda")  # noqa: E731
    dA, db = dev(A, torch.float64), dev(b, torch.float64)
    ret, piv = empty(m, 2, t=torch.int32), empty(m, 2, n, t=torch.int32)
    lu, dinv0, x = empty(m, 2, n, n), empty(m), empty(m, 2, r, n)
    assert lc.lc_factor_solve(team, fp32, n, *(t.data_ptr() for t in (dA, db)), m, r,
                              *(t.data_ptr() for t in (ret, piv, lu, dinv0, x))) == 0
    torch.cuda.synchronize()
    ret, piv, lu, dinv0, x = (t.cpu().numpy() for t in (ret, piv, lu, dinv0, x))
    for k, name in enumerate(mats):
        assert ret[k, 0] == ret[k, 1], name
        if name in ("zero column", "nan column"):
            assert ret[k, 0] != 0, name
        if name in ("newton", "full", "all ones", "infinite entry", "multipliers not finite, pivot row zero") or \
                name.startswith("diagonal"):
            assert ret[k, 0] == 0, name
        if ret[k, 0]:
            continue
        assert np.array_equal(piv[k, 0], piv[k, 1]), name
        assert np.array_equal(lu[k, 0], lu[k, 1], equal_nan=True), name
        # the register solve gives way beyond 2^+-400 on the diagonal, on a significand
        # of all ones (FP64) and on what is not finite, to the dividing one
        d = np.abs(np.diag(lu[k, 1].T))
        with np.errstate(all="ignore"):
            man, e = np.frexp(d)
            inside = np.all(np.isfinite(d) & (e - 1 >= -400) & (e - 1 <= 400) & (man != 1.0 - 2.0 ** -53))
        assert np.isnan(dinv0[k]) == (not inside), (name, dinv0[k])
        for q in range(r):
            assert np.array_equal(x[k, 0, q], x[k, 1, q], equal_nan=True), (name, q)
        if name in ("newton", "full", "ties", "sparse"):
            # |P A - L U| <= gamma_n |L| |U| componentwise (Higham, theorem 9.3), doubled for the product here
            a = A[k].T.astype(np.float32 if fp32 else np.float64).astype(np.float64)
            for j, p in enumerate(piv[k, 1]):
                a[[j, p]] = a[[p, j]]
            f = lu[k, 1].T
            Lo, U = np.tril(f, -1) + np.eye(n), np.triu(f)
            eps = 2.0 ** (-24 if fp32 else -53)
            assert np.all(np.abs(a - Lo @ U) <= 2.0 * (n + 1) * eps * (np.abs(Lo) @ np.abs(U)) + 1e-300), name


@pytest.mark.parametrize("ns", [9, 31, 32, 53, 64, 88])
@pytest.mark.parametrize("transpose", [0, 1])
def test_adjoint_factorisation(cuda, lc, ns, transpose):
    """n = ns + 1 unknowns: 33 and 65 have a row more than their species fill lanes."""
    torch = cuda
    n, m = ns + 1, 5
    rng = np.random.default_rng(ns)
    J = rng.normal(size=(m, n, n)) / np.sqrt(n)
    b = rng.normal(size=(m, n))
    dJ, db = (torch.as_tensor(np.ascontiguousarray(a), device="cuda") for a in (J.transpose(0, 2, 1), b))
    ret, x = torch.zeros(m, dtype=torch.int32, device="cuda"), torch.zeros_like(db)
    assert lc.lc_adjoint(ns, dJ.data_ptr(), 0.5, transpose, db.data_ptr(), m, ret.data_ptr(), x.data_ptr()) == 0
    torch.cuda.synchronize()
    assert not ret.any()
    for k in range(m):
        a = np.eye(n) - 0.5 * (J[k].T if transpose else J[k])
        # backward error of elimination with pivoting: n eps times a growth of at most ~10 here
        tol = 10 * n * n * 2.0 ** -53 * np.linalg.cond(a)
        ref = np.linalg.solve(a, b[k])
        assert np.linalg.norm(x[k].cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
