"""Launch forms of the BDF kernels.  Teams of one and of two lanes a species,
blocks of up to 12 warps and batches that leave lanes, warps and blocks idle
give the same bits.  Blocks of 16 warps round the energy of one temperature
solve an iteration differently, and 16-lane teams sum in another order where
there are more unknowns than lanes: these agree to what rounding grows to.
And the transport kernel at the edges of its tiles."""

import numpy as np
import pytest

from pelephysics_b200 import _lib, transport as tr
from pelephysics_b200.reactor import Reactor
from tests.helpers import premix_oracle

pytestmark = pytest.mark.gpu


def _react(mech, rY, src, rX, rXs, dt, **opts):
    r = Reactor(mech)
    r.init(1, rX.shape[0], **opts)
    y = rY.copy()
    r.react(y, src.copy(), rX.copy(), rXs.copy(), dt)
    stats = r.cell_stats(rX.shape[0])
    r.close()
    return y, stats


# 54 and 89 unknowns: two and three rows a lane, the last one part filled
@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("mech,lanes,T0,P,dt", [("dodecane_lu", 64, 1000.0, 40 * 1013250.0, 2e-6),
                                                ("grimech30", 64, 1300.0, 1013250.0, 1e-6),
                                                ("heptane_lu_88sk", 128, 900.0, 20 * 1013250.0, 1e-5)])
def test_two_lanes_a_species_change_no_bits(cuda, oracle, mech, lanes, T0, P, dt, fp32):
    cells = premix_oracle(oracle, mech, 5, 7, T0, 500.0, 0.5, 1.0, P=P)
    opts = dict(rtol=1e-8, atol=1e-12, max_order=5, lu_fp32=fp32, team_lanes=lanes)
    a, sa = _react(mech, *cells, dt, warps_per_block=lanes // 32, **opts)
    b, sb = _react(mech, *cells, dt, warps_per_block=lanes // 16, **opts)
    assert np.array_equal(a, b) and np.array_equal(sa, sb)


def test_a_team_the_mechanism_has_not_is_refused(cuda, oracle):
    for mech, lanes in (("dodecane_lu", 128), ("heptane_lu_88sk", 64), ("drm19", 64)):
        cells = premix_oracle(oracle, mech, 1, 7, 1300.0, 100.0, 0.5, 1.0)
        for integrator in ("ReactorCvode", "ReactorRK64"):
            r = Reactor(mech, integrator)
            r.init(1, 1, warps_per_block=lanes // 16, team_lanes=lanes)
            with pytest.raises(_lib.EngineError):
                r.react(*[c.copy() for c in cells], 1e-9)
            r.close()


# 10 and 22 unknowns: the update's lane groups from 32 rows down to one
@pytest.mark.parametrize("ncells", [1, 33])
@pytest.mark.parametrize("mech,dt", [("LiDryer", 1e-5), ("drm19", 1e-6)])
def test_block_sizes_change_no_bits(cuda, oracle, mech, dt, ncells):
    cells = premix_oracle(oracle, mech, ncells, 9, 1100.0, 700.0, 0.5, 1.0)
    opts = dict(rtol=1e-10, atol=1e-10, max_order=5)
    ref, st = _react(mech, *cells, dt, warps_per_block=8, **opts)
    for form in (dict(warps_per_block=1), dict(warps_per_block=4, register_budget=1), dict(warps_per_block=12)):
        y, s = _react(mech, *cells, dt, **form, **opts)
        assert np.array_equal(y, ref) and np.array_equal(s, st), form


@pytest.mark.parametrize("mech,dt", [("LiDryer", 1e-5), ("drm19", 1e-6)])
def test_fp32_block_sizes_change_no_bits(cuda, oracle, mech, dt):
    cells = premix_oracle(oracle, mech, 33, 9, 1100.0, 700.0, 0.5, 1.0)
    opts = dict(rtol=1e-10, atol=1e-10, max_order=5, lu_fp32=1)
    ref, st = _react(mech, *cells, dt, warps_per_block=8, **opts)
    for wpb in (1, 4, 12):
        y, s = _react(mech, *cells, dt, warps_per_block=wpb, **opts)
        assert np.array_equal(y, ref) and np.array_equal(s, st), wpb


# Through ignition at rtol = 1e-10 one bit of T grows to 1e-8 of the result
# (2-norm over the cells; ppb_bdf.cuh, UE): ten times that is the bar.
@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("mech,dt", [("LiDryer", 1e-4), ("drm19", 1e-5)])
def test_forms_of_other_roundings_agree(cuda, oracle, mech, dt, fp32):
    cells = premix_oracle(oracle, mech, 200, 5, 1000.0, 400.0, 0.5, 1.5)
    opts = dict(rtol=1e-10, atol=1e-10, max_order=5, lu_fp32=fp32)
    ref, _ = _react(mech, *cells, dt, warps_per_block=8, **opts)
    for form in (dict(warps_per_block=16), dict(warps_per_block=8, team_lanes=16),
                 dict(warps_per_block=1, team_lanes=16)):
        y, _ = _react(mech, *cells, dt, **form, **opts)
        for part in (slice(0, -1), slice(-1, None)):
            assert np.linalg.norm(y[:, part] - ref[:, part]) <= 1e-7 * np.linalg.norm(ref[:, part]), form


def _config(mech, **opts):
    r = Reactor(mech)
    r.init(1, 1, **opts)
    cfg = r.launch_config()[:3]
    r.close()
    return cfg


@pytest.mark.parametrize("mech,lanes,T0,P,dt", [("dodecane_lu", 64, 1000.0, 40 * 1013250.0, 2e-6),
                                                ("heptane_lu_88sk", 128, 900.0, 20 * 1013250.0, 1e-5)])
def test_a_fixed_team_keeps_its_lanes(cuda, oracle, mech, lanes, T0, P, dt):
    """team_lanes is the lanes of a cell whatever warps_per_block says; two
    lanes a species are asked for, and reported, as what they are."""
    for wpb in (1, 2, 4, 8):
        assert _config(mech, warps_per_block=wpb, team_lanes=lanes) == (lanes // 32, lanes, 1)
    two = dict(warps_per_block=lanes // 16, team_lanes=2 * lanes)
    assert _config(mech, **two) == (lanes // 16, 2 * lanes, 1)
    cells = premix_oracle(oracle, mech, 5, 7, T0, 500.0, 0.5, 1.0, P=P)
    opts = dict(rtol=1e-8, atol=1e-12, max_order=5)
    for fp32 in (0, 1):
        a, sa = _react(mech, *cells, dt, warps_per_block=1, team_lanes=lanes, lu_fp32=fp32, **opts)
        b, sb = _react(mech, *cells, dt, lu_fp32=fp32, **two, **opts)
        assert np.array_equal(a, b) and np.array_equal(sa, sb)


# five cells of 46,464 bytes in a block's 232,448
def test_the_largest_fp32_block_fits(cuda, oracle):
    cells = premix_oracle(oracle, "grimech30", 11, 3, 1300.0, 500.0, 0.5, 1.0)
    opts = dict(rtol=1e-8, atol=1e-12, max_order=5, lu_fp32=1)
    a, sa = _react("grimech30", *cells, 1e-6, warps_per_block=4, **opts)
    b, sb = _react("grimech30", *cells, 1e-6, warps_per_block=5, **opts)
    assert np.array_equal(a, b) and np.array_equal(sa, sb)


# tiles of 32 cells (16 for 88 species)
@pytest.mark.parametrize("n", [1, 15, 17, 33])
@pytest.mark.parametrize("mech", ["LiDryer", "drm19", "dodecane_lu", "heptane_lu_88sk"])
def test_transport_tile_edges(cuda, oracle, mech, n):
    torch = cuda
    N = oracle.Mech(mech).nsp
    rng = np.random.default_rng(n)
    T = rng.uniform(300.0, 3000.0, n)
    rho = 10.0 ** rng.uniform(-5, -1, n)
    Y = rng.uniform(size=(n, N)) ** 3
    Y /= Y.sum(1, keepdims=True)
    out = tr.transport(mech, torch.as_tensor(T, device="cuda"), torch.as_tensor(rho, device="cuda"),
                       torch.as_tensor(np.ascontiguousarray(Y.T), device="cuda"), tr.TR_ALL)
    D = out["D"].cpu().numpy().T
    rel = lambda a, b: np.max(np.abs(np.asarray(a) - b) / np.abs(b))  # noqa: E731
    for c in {0, n // 2, n - 1}:
        Dr, _, mur, xir, lamr = oracle.transport(mech, oracle.TR_ALL, T[c], rho[c], Y[c])
        # the bar of the transport tests: mixture sums in another order, the last bit of exp
        assert rel(D[c], Dr) <= 1e-13
        assert rel(out["mu"][c].item(), mur) <= 1e-13 and rel(out["lam"][c].item(), lamr) <= 1e-13
        assert rel(out["xi"][c].item(), xir) <= 1e-13
