"""Mechanism tables beyond the compact records of the tuned kernels (RxRate,
JcEntry: three slots a phase space, five Gibbs or net-stoichiometry terms, and
so on) are taken, through the wide records, up to the limits of the latter;
rates, Jacobian and integration against the general path, which reads the
tables themselves."""

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests.helpers import premix_oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "pelephysics_b200")
GOLD = os.path.join(ROOT, "tests", "golden")
pytestmark = pytest.mark.skipif(shutil.which("nvcc") is None or not os.path.exists(os.path.join(PKG, "libppb200.so")),
                                reason="needs nvcc and the built engine")

# LiDryer: H2 O2 H2O H O OH HO2 H2O2 N2; the last reaction's reactants and products
H2, O2, H2O, OH, HO2, H2O2, N2 = 0, 1, 2, 5, 6, 7, 8
REACTIONS = {
    "four forward slots": ({H2: 1, OH: 2, N2: 1}, {H2O: 2, N2: 1}),
    "five reverse slots": ({H2: 1, H2O2: 1, N2: 1}, {H2: 1, O2: 1, H2O: 1, N2: 2}),
    "six Gibbs and net terms": ({H2: 1, H2O2: 1, N2: 1}, {O2: 1, H2O: 1, HO2: 1}),
    "two repeated species": ({H2: 2, H2O2: 2}, {H2O: 3}),
    "a repeated species behind two others": ({H2: 1, O2: 1, H2O: 2}, {H2O: 1, H2O2: 1, N2: 1}),
    "three moles fewer": ({H2: 1, O2: 1, H2O: 1, N2: 1}, {H2O2: 1}),
    "three moles more": ({H2O2: 1}, {H2: 1, O2: 1, H2O: 1, N2: 1}),
}
LAST = 20


@pytest.fixture(scope="module")
def tc(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("table_checks") / "table_checks.so")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "-Xcompiler", "-fPIC",
                        "-shared", "-diag-suppress", "177,550", "-I", os.path.join(PKG, "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "table_checks.cu"), "-o", so, "-L", PKG, "-lppb200", "-Xlinker",
                        "-rpath," + PKG], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = C.CDLL(so)
    vp, d, i = C.c_void_p, C.c_double, C.c_int
    L.tc_new.restype = vp
    L.tc_new.argtypes = [C.c_char_p]
    ip = C.POINTER(i)
    L.tc_reaction.argtypes = [vp, i, i, ip, ip, i, ip, ip, d, d, d]
    L.tc_coefficient.argtypes = [vp, i, d]
    L.tc_third.argtypes = L.tc_more_qss.argtypes = [vp, i]
    L.tc_pack.argtypes = L.tc_upload.argtypes = L.tc_free.argtypes = [vp]
    L.tc_rates.argtypes = [vp, vp, vp, vp, i, i]
    L.tc_rate_scale.argtypes = [vp, vp, vp, vp, i]
    L.tc_jacobian.argtypes = [vp, vp, vp, i, vp, i, i]
    L.tc_react.argtypes = [vp, i, vp, vp, vp, vp, vp, i, d]
    return L


class Mech:
    def __init__(self, tc, base, what):
        self.tc, self.h = tc, tc.tc_new(base.encode())
        if what in REACTIONS:
            self.reaction(LAST, *REACTIONS[what], 1e3)
        elif what == "a fractional coefficient":
            tc.tc_coefficient(self.h, LAST, -0.3)
        elif what == "300 third bodies":
            tc.tc_third(self.h, 300)
        elif what == "32 QSS species":
            tc.tc_more_qss(self.h, 28)
        else:
            assert what is None

    def reaction(self, r, f, p, A):
        arr = lambda v: (C.c_int * len(v))(*v)  # noqa: E731
        self.tc.tc_reaction(self.h, r, len(f), arr(list(f)), arr(list(f.values())), len(p), arr(list(p)),
                            arr(list(p.values())), A, 0.0, 500.0)

    def __enter__(self):
        return self

    def __exit__(self, *a):
        self.tc.tc_free(self.h)


CASES = [("LiDryer", w) for w in list(REACTIONS) + ["a fractional coefficient"]] + [
    ("heptane_lu_88sk", "300 third bodies"), ("CH4_lean_qss", "32 QSS species")]


@pytest.mark.parametrize("base,what", CASES)
def test_tables_pack(tc, base, what):
    """On the CPU: the packing takes the tables."""
    with Mech(tc, base, what) as m:
        assert tc.tc_pack(m.h) == 0


def test_tables_beyond_the_wide_records_are_refused(tc):
    with Mech(tc, "LiDryer", None) as m:
        m.reaction(LAST, {H2: 2, O2: 1, OH: 2}, {H2O: 2, N2: 1}, 1.0)  # five forward slots
        assert tc.tc_pack(m.h) != 0


def _point(base):
    g = np.load(os.path.join(GOLD, f"point_{base}.npz"))
    return g["sc"], g["T"]


def _dev(torch, a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _rates(torch, m, sc, T, team):
    w = torch.zeros_like(sc)
    assert m.tc.tc_rates(m.h, sc.data_ptr(), T.data_ptr(), w.data_ptr(), len(T), team) == 0
    torch.cuda.synchronize()
    return w.cpu().numpy()


# The bars of the pointwise tests (tests/test_gpu_pointwise.py): FP64 on both
# sides, the sums in another order.
@pytest.mark.gpu
@pytest.mark.parametrize("base,what", CASES[:-1])
def test_rates_and_jacobian_match_the_general_path(cuda, tc, base, what):
    torch = cuda
    sc, T = (_dev(torch, a) for a in _point(base))
    n, N = sc.shape
    with Mech(tc, base, what) as m:
        assert tc.tc_upload(m.h) == 0
        scale = torch.zeros_like(sc)
        assert tc.tc_rate_scale(m.h, sc.data_ptr(), T.data_ptr(), scale.data_ptr(), n) == 0
        torch.cuda.synchronize()
        general, team = _rates(torch, m, sc, T, 1), _rates(torch, m, sc, T, 32)
        assert np.all(np.abs(team - general) <= 1e-12 * scale.cpu().numpy() + 1e-300)
        for consP in (0, 1):
            J = [torch.zeros((n, (N + 1) ** 2), dtype=torch.float64, device="cuda") for _ in range(2)]
            for out, lanes in zip(J, (1, 32)):
                assert tc.tc_jacobian(m.h, sc.data_ptr(), T.data_ptr(), consP, out.data_ptr(), n, lanes) == 0
            torch.cuda.synchronize()
            for ref, got in zip(*(j.cpu().numpy() for j in J)):
                assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref)
                big = np.abs(ref) > 1e-6 * np.abs(ref).max()
                assert np.all(np.abs(got - ref)[big] <= 1e-10 * np.abs(ref)[big])


@pytest.mark.gpu
def test_qss_species_without_reactions_change_nothing(cuda, tc):
    torch = cuda
    sc, T = (_dev(torch, a) for a in _point("CH4_lean_qss"))
    with Mech(tc, "CH4_lean_qss", None) as a, Mech(tc, "CH4_lean_qss", "32 QSS species") as b:
        assert tc.tc_upload(a.h) == 0 and tc.tc_upload(b.h) == 0
        assert np.array_equal(_rates(torch, a, sc, T, 32), _rates(torch, b, sc, T, 32))


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["four forward slots", "six Gibbs and net terms"])
def test_react_matches_the_plain_engine(cuda, oracle, tc, what):
    """The tuned kernel on a wide mechanism against the one-thread engine: the
    bars of the integration tests (T 1e-6 relative, Y 1e-8)."""
    torch = cuda
    rY, src, rX, rXs = premix_oracle(oracle, "LiDryer", 33, 4, 1300.0, 400.0, 0.5, 1.0)
    n, N = src.shape
    rY[:, [OH, HO2, H2O2]] = 1e-3 * rY[:, [O2]]
    rho = rY[:, :N].sum(1)
    M = oracle.Mech("LiDryer")
    rX = np.array([rho[c] * M.ckubms(rY[c, N], rY[c, :N] / rho[c]) for c in range(n)])

    def run(m, engine):
        y, s, x, xs = _dev(torch, rY.T), _dev(torch, src.T), _dev(torch, rX), _dev(torch, rXs)
        work = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
        assert tc.tc_react(m.h, engine, y.data_ptr(), s.data_ptr(), x.data_ptr(), xs.data_ptr(), work.data_ptr(), n,
                           1e-6) == 0
        torch.cuda.synchronize()
        assert not work[1:].any()
        return y.cpu().numpy().T

    with Mech(tc, "LiDryer", what) as m, Mech(tc, "LiDryer", None) as base:
        assert tc.tc_upload(m.h) == 0 and tc.tc_upload(base.h) == 0
        plain, tuned, without = run(m, 0), run(m, 1), run(base, 1)
    assert np.max(np.abs(tuned[:, N] / plain[:, N] - 1)) <= 1e-6
    assert np.max(np.abs(tuned[:, :N] - plain[:, :N]) / rho[:, None]) <= 1e-8
    # the reaction counts: without it the result is a hundred times the bar away
    assert np.max(np.abs(without[:, :N] - plain[:, :N]) / rho[:, None]) > 1e-6
