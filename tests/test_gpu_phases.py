"""GPU parity of each PM phase against the FP64 oracle, through the C-ABI.

Bars: cell indices bit-exact; density bit-exact run to run and within 1e-6
of the oracle's max; forces within FIELD_RTOL (1e-5) of the oracle's max;
positions/velocities after a phase within float rounding.
"""
import ctypes

import numpy as np
import pytest

import hacc_gpm_b200 as H
from oracle import pm_oracle as O
from tests.helpers import FIELD_RTOL, lattice_state, params_text, rel_max_err

pytestmark = pytest.mark.gpu

F = ctypes.POINTER(ctypes.c_float)
SIZES = [16, 24, 32, 40, 48, 64, 80, 96, 120, 128, 160, 200]


def make(ng, np_side=None, rl=None, extra=""):
    return H.Simulation(H.parse_params(params_text(ng, np_side, rl, extra=extra)))


@pytest.mark.parametrize("ng", [32, 48])
def test_state_roundtrip_and_cells_bitexact(ng):
    x, v = lattice_state(ng, ng, disp=3.0, seed=ng)
    with make(ng) as s:
        s.load_state(x, v)
        x2, v2 = s.store_state()
        assert np.array_equal(x2, x) and np.array_equal(v2, v)
        cells = s.get_cells()
    i = np.trunc(x).astype(np.int64)  # cic_pm.cu:52-54 `int i = x`
    assert np.array_equal(cells, (i[:, 0] * ng + i[:, 1]) * ng + i[:, 2])


@pytest.mark.parametrize("ng", [32, 48])
def test_drift_matches_oracle(ng):
    x, v = lattice_state(ng, ng, disp=2.0, vel=3.0, seed=3)
    pf = np.float32(0.37)
    with make(ng) as s:
        s.load_state(x, v)
        s.drift(float(pf))
        xg, vg = s.store_state()
    xo = O.drift(x.astype(np.float64), v.astype(np.float64), float(pf), ng)
    err = np.abs(O.periodic_diff(xg, xo, ng)).max()
    assert err < 4 * np.finfo(np.float32).eps * ng
    assert np.array_equal(vg, v)


@pytest.mark.parametrize("ng,np_side", [(32, 32), (48, 48), (64, 32), (32, 64), (24, 48)])
def test_deposit_deterministic_and_matches_oracle(ng, np_side):
    x, v = lattice_state(np_side, ng, disp=1.5, seed=5)
    with make(ng, np_side) as s:
        s.load_state(x, v)
        s.cic()
        r1 = s.get_density()
        s.cic()
        r2 = s.get_density()
    assert np.array_equal(r1, r2)  # bit-exact run to run
    ro = O.cic_deposit(x.astype(np.float64), ng, O.cic_mass(ng, np_side))
    assert np.abs(r1 - ro).max() <= 1e-6 * ro.max()
    assert r1.astype(np.float64).sum() == pytest.approx(ro.sum(), rel=1e-7)


@pytest.mark.parametrize("ng,np_side,ncand", [(32, 32, 12), (64, 32, 8)])
def test_deposit_hot_cell_exact(ng, np_side, ncand, monkeypatch):
    """All particles in one cell (late-time clustering extreme): the 32-bit
    windows wrap, every candidate detects it and sends the block to the
    exact pass (the candidate that checks while flushing first takes its
    flushed values back out of the grid), and the integer accumulation stays
    exact."""
    for pos, cells in ((5.5, 8), (5.0, 1)):
        x = np.full((np_side ** 3, 3), pos, np.float32)
        v = np.zeros_like(x)
        for cand in range(ncand):
            monkeypatch.setenv("HGPM_DEPOSIT", str(cand))
            with make(ng, np_side) as s:
                s.load_state(x, v)
                s.cic()
                r = s.get_density()
            mass = (ng / np_side) ** 3
            assert np.count_nonzero(r) == cells, (pos, cand)
            assert r[5, 5, 5] == np.float32(np_side ** 3 * mass / cells), (pos, cand)


@pytest.mark.parametrize("ng", SIZES)
def test_solve_gradient_matches_oracle(ng):
    x, v = lattice_state(ng, ng, disp=1.2, seed=ng + 1)
    with make(ng) as s:
        s.load_state(x, v)
        s.cic()
        rho = s.get_density().astype(np.float64)
        s.solve_gradient()
        f = s.get_force()
    fo = O.solve_gradient(rho, ref_quirks=True)
    assert rel_max_err(f, fo) < FIELD_RTOL


@pytest.mark.parametrize("ng,np_side", [(48, 48), (64, 64), (80, 80), (128, 128), (320, 320), (768, 192)])
def test_tma_and_plain_strided_passes_bit_identical(ng, np_side, monkeypatch):
    """The persistent TMA-fed y passes and the plain strided kernels run the
    same per-line transform, so forces are bit-identical."""
    x, v = lattice_state(np_side, ng, disp=1.3, seed=ng + 7)
    out = []
    for flag in ("0", "1"):
        monkeypatch.setenv("HGPM_NO_TMA", flag)
        with make(ng, np_side) as s:
            s.load_state(x, v)
            s.cic()
            s.solve_gradient()
            out.append(s.get_force())
            s.sync()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("ng,np_side", [(256, 256), (512, 256), (1024, 128)])
def test_plane_cluster_passes_bit_identical(ng, np_side, monkeypatch):
    """The z and y passes as one kernel with a thread-block cluster per x
    plane (HGPM_PLANE=1) give the spectrum, the force formed on demand, the
    paired-potential kick and P(k) of the separate passes bit for bit."""
    rng = np.random.default_rng(ng + np_side)
    x = (rng.random((np_side ** 3, 3), dtype=np.float32) * np.float32(ng)).astype(np.float32)
    x = np.minimum(x, np.float32(ng) * np.float32(1 - 2 ** -23))
    v = rng.standard_normal((np_side ** 3, 3), dtype=np.float32)
    monkeypatch.setenv("HGPM_KICK", "7")
    ref = None
    for flag in ("0", "1"):
        monkeypatch.setenv("HGPM_PLANE", flag)
        with make(ng, np_side) as s:
            s.load_state(x, v)
            s.cic()
            pk = s.power_spectrum(nbins=64, log_bins=True)[1]
            s.cic()
            s.solve_gradient()
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            xs, vs = s.store_state()
            # the force grid formed on demand from the y-inverted spectrum
            # (not at 1024^3: 13 GB on the host)
            f = s.get_force() if ng <= 512 else None
            got = (pk, xs, vs, f)
        if ref is None:
            ref = got
            continue
        for a, b in zip(ref, got):
            assert (a is None and b is None) or np.array_equal(a, b), flag


@pytest.mark.parametrize("ng,np_side", [(32, 32), (64, 64), (128, 128), (80, 80), (96, 96), (192, 96),
                                        (256, 128), (384, 128), (512, 256)])
def test_fused_x_pass_variants_bit_identical(ng, np_side, monkeypatch):
    """The persistent TMA-fed Poisson x pass and the plain fused x pass (with
    its own or twice the columns per CTA) give bit-identical forces, and the
    next deposit after the solve starts from a zeroed accumulator."""
    x, v = lattice_state(np_side, ng, disp=1.1, seed=ng + 3)
    out = []
    for flag in ("0", "1", "2"):
        monkeypatch.setenv("HGPM_XTMA", flag)
        with make(ng, np_side) as s:
            s.load_state(x, v)
            s.cic()
            s.solve_gradient()
            f = s.get_force()
            s.cic()
            rho = s.get_density()
            s.sync()
        if out:
            assert np.array_equal(out[0][0], f) and np.array_equal(out[0][1], rho), flag
        else:
            out.append((f, rho))


@pytest.mark.parametrize("ng,np_side,disp", [(32, 32, 0.3), (64, 64, 0.3), (64, 64, 2.0), (64, 64, 6.0),
                                             (64, 32, 1.0), (48, 48, 1.0), (64, 32, 5.0)])
def test_deposit_configurations_bit_identical(ng, np_side, disp, monkeypatch):
    """Every deposit candidate (split, 32-bit and column windows, with and
    without x-half splitting, and the direct one without a window; the spill
    passes, reached with disp 2 to 6) gives the same int64 grid; 16^3 blocks
    (np = ng = 32, 48, 64) and 8^3 blocks (np < ng)."""
    x, v = lattice_state(np_side, ng, disp=disp, vel=1.0, seed=23)
    out = []
    n = 12 if np_side % 16 == 0 and ng <= np_side else 8
    for flag in range(n):
        monkeypatch.setenv("HGPM_DEPOSIT", str(flag))
        with make(ng, np_side) as s:
            assert s.tuned_choices()["deposit"] == flag
            s.load_state(x, v)
            s.cic()
            out.append(s.get_density())
    for o in out[1:]:
        assert np.array_equal(out[0], o)


@pytest.mark.parametrize("ng,np_side,disp", [(32, 32, 1.0), (48, 48, 1.0), (64, 32, 1.0), (32, 64, 1.0), (64, 64, 0.3),
                                             (64, 64, 4.0), (128, 128, 1.5)])
def test_kick_variants_bit_identical(ng, np_side, disp, monkeypatch):
    """Every kick candidate (flat global gathers with different CTA shapes
    and unit runs, the float4-window kick, the gathers of the real or the
    paired potential that form each corner's force as the gradient kernel
    does) runs the same FP32 arithmetic in the same order; disp 4 spreads
    blocks past the window caps (global-gather fallback); at 128^3 the grid
    has more blocks than resident CTAs."""
    x, v = lattice_state(np_side, ng, disp=disp, vel=1.0, seed=17)
    out = []
    for flag in ("0", "1", "2", "3", "4", "5", "6", "7"):
        monkeypatch.setenv("HGPM_KICK", flag)
        with make(ng, np_side) as s:
            s.load_state(x, v)
            s.cic()
            s.solve_gradient()
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            out.append(s.store_state())
    for o in out[1:]:
        assert np.array_equal(out[0][0], o[0]) and np.array_equal(out[0][1], o[1])


def test_solve_gradient_plane_wave_analytic():
    """Particles arranged so that rho = 1 + A cos(2 pi x/ng) exactly on the
    grid is not reachable with CIC; instead place a sheet and compare with
    the oracle's discrete operator, plus symmetry: F_y = F_z = 0."""
    ng = 32
    q = np.stack(np.meshgrid(np.arange(ng), np.arange(ng), np.arange(ng), indexing="ij"), -1).reshape(-1, 3)
    x = q.astype(np.float64)
    x[:, 0] = np.mod(x[:, 0] + 0.8 * np.sin(2 * np.pi * x[:, 0] / ng), ng)
    x = x.astype(np.float32)
    with make(ng) as s:
        s.load_state(x, np.zeros_like(x))
        s.cic()
        rho = s.get_density().astype(np.float64)
        s.solve_gradient()
        f = s.get_force()
    fo = O.solve_gradient(rho, ref_quirks=True)
    assert rel_max_err(f[0], fo[0]) < FIELD_RTOL
    assert np.abs(f[1]).max() < 1e-5 * np.abs(f[0]).max()
    assert np.abs(f[2]).max() < 1e-5 * np.abs(f[0]).max()


@pytest.mark.parametrize("ng", [32, 48])
def test_kick_and_fused_drifts_match_oracle(ng):
    x, v = lattice_state(ng, ng, disp=1.0, vel=1.0, seed=9)
    dt, fscal = 0.0123, 1.7
    pf_a, pf_b = np.float32(0.3), np.float32(0.25)
    with make(ng) as s:
        s.load_state(x, v)
        s.cic()
        s.solve_gradient()
        f = s.get_force().astype(np.float64)
        s.kick_drift(dt, fscal, float(pf_a), float(pf_b), 2)
        xg, vg = s.store_state()
    vo = O.interp_kick(x.astype(np.float64), v.astype(np.float64), f, dt, fscal)
    xo = O.drift(O.drift(x.astype(np.float64), vo, float(pf_a), ng), vo, float(pf_b), ng)
    assert rel_max_err(vg, vo) < 1e-6
    assert np.abs(O.periodic_diff(xg, xo, ng)).max() < 1e-5


def test_kick_only_leaves_positions():
    ng = 32
    x, v = lattice_state(ng, ng, seed=2)
    with make(ng) as s:
        s.load_state(x, v)
        s.cic()
        s.solve_gradient()
        s.kick_drift(0.01, 1.0, 0.0, 0.0, 0)
        xg, _ = s.store_state()
    assert np.array_equal(xg, x)


def test_errors_are_status_codes_not_crashes():
    ng = 32
    with make(ng) as s:
        with pytest.raises(H.HgpmError, match="no particle state"):
            s.cic()
        with pytest.raises(H.HgpmError, match="no deposited density"):
            s.solve_gradient()
        with pytest.raises(H.HgpmError):
            s.load_state(np.zeros((5, 3), np.float32), np.zeros((5, 3), np.float32))


@pytest.mark.parametrize("ng,np_side", [(64, 64), (64, 32)])
def test_autotune_leaves_state_and_results_unchanged(ng, np_side, tmp_path, monkeypatch):
    """hgpm_autotune times every candidate on the live state: the state is
    the same afterwards, the picks are valid, steps after tuning equal steps
    without it bit for bit, and a stored pick is applied to the next context
    of that size."""
    for k in ("HGPM_DEPOSIT", "HGPM_KICK", "HGPM_NO_TMA", "HGPM_XTMA", "HGPM_PLANE"):
        monkeypatch.delenv(k, raising=False)
    monkeypatch.setenv("HGPM_TUNE_CACHE", str(tmp_path / "tune.txt"))
    hp = H.parse_params(params_text(ng, np_side))
    x, v = lattice_state(np_side, ng, disp=2.0, vel=1.0, seed=29)

    def run(tune):
        with H.Simulation(hp) as s:
            s.load_state(x, v)
            picks = None
            if tune:
                picks = s.autotune(reps=2, store=True)
                x1, v1 = s.store_state()
                assert np.array_equal(x1, x) and np.array_equal(v1, v)
            ts = H.Timestepper(hp)
            ts.set_initial_z(hp.z_ini)
            ts.reverse_half_step()
            ts.advance_half_step()
            s.run_steps(ts, 3)
            return s.store_state(), picks

    (xa, va), picks = run(True)
    monkeypatch.setenv("HGPM_NO_TUNE_CACHE", "1")
    (xb, vb), _ = run(False)
    assert np.array_equal(xa, xb) and np.array_equal(va, vb)
    assert all(p["ms"] > 0 for p in picks.values())
    monkeypatch.delenv("HGPM_NO_TUNE_CACHE")
    with H.Simulation(hp) as s:
        got = s.tuned_choices()
    assert got == {k: p["choice"] for k, p in picks.items()}


def test_bounded_wait_time_out_reported_and_context_usable():
    """A bounded mbarrier wait that nothing completes sets the error flag;
    hgpm_sync reports it once and clears it, and the context stays usable:
    the next solve matches a fresh context's bit for bit."""
    ng = 32
    x, v = lattice_state(ng, ng, disp=1.0, seed=31)
    with make(ng) as s:
        s.load_state(x, v)
        s.sync()
        s.test_wait_timeout(1000)
        with pytest.raises(H.HgpmError, match="timed out"):
            s.sync()
        s.sync()  # the flag was cleared
        s.cic()
        s.solve_gradient()
        f1 = s.get_force()
        s.sync()
    with make(ng) as s:
        s.load_state(x, v)
        s.cic()
        s.solve_gradient()
        f2 = s.get_force()
    assert np.array_equal(f1, f2)


@pytest.mark.parametrize("ng,np_side", [(32, 32), (64, 32)])
def test_force_grid_on_demand_with_potential_kick(ng, np_side, monkeypatch):
    """With a kick that gathers the real or the paired potential the solve
    writes no force grid; hgpm_get_force forms it (for the paired potential
    from the potential's spectrum first), equal bit for bit to the grid the
    force-grid kick's solve writes, and the kick after it is unchanged."""
    x, v = lattice_state(np_side, ng, disp=1.5, vel=1.0, seed=37)
    out = []
    states = []
    for flag in ("0", "5", "7"):
        monkeypatch.setenv("HGPM_KICK", flag)
        with make(ng, np_side) as s:
            assert s.tuned_choices()["kick"] == int(flag)
            s.load_state(x, v)
            s.cic()
            s.solve_gradient()
            out.append(s.get_force())
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            states.append(s.store_state())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    for st in states[1:]:
        assert np.array_equal(states[0][0], st[0]) and np.array_equal(states[0][1], st[1])


@pytest.mark.parametrize("ng,np_side", [(96, 96), (120, 120), (256, 256), (256, 128), (320, 160)])
def test_kick_shares_bit_identical(ng, np_side, monkeypatch):
    """The potential-gathering kicks in 128-particle CTAs (up to 96^3), in
    several waves of CTAs (256^3) and in 8^3 blocks give the flat force-grid
    kick's state bit for bit."""
    rng = np.random.default_rng(ng + np_side)
    x = rng.random((np_side ** 3, 3), dtype=np.float32) * np.float32(ng * (1 - 2 ** -20))
    v = rng.standard_normal((np_side ** 3, 3), dtype=np.float32)
    out = []
    for flag in ("3", "5", "6", "7"):
        monkeypatch.setenv("HGPM_KICK", flag)
        with make(ng, np_side) as s:
            s.load_state(x, v)
            s.cic()
            s.solve_gradient()
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            out.append(s.store_state())
    for o in out[1:]:
        assert np.array_equal(out[0][0], o[0]) and np.array_equal(out[0][1], o[1])


@pytest.mark.parametrize("ng,np_side", [(96, 96), (128, 128), (40, 40), (120, 120), (256, 128), (320, 160)])
def test_default_deposit_on_each_side_of_its_rule(ng, np_side, monkeypatch):
    """The default deposit (direct below its rule's sides, windowed above)
    gives the split window's grid bit for bit, twice in a row."""
    x, v = lattice_state(np_side, ng, disp=2.5, vel=1.0, seed=41)
    out = []
    for flag in ("0", None):
        if flag is None:
            monkeypatch.delenv("HGPM_DEPOSIT", raising=False)
        else:
            monkeypatch.setenv("HGPM_DEPOSIT", flag)
        with make(ng, np_side) as s:
            s.load_state(x, v)
            for _ in range(2):
                s.cic()
                out.append(s.get_density())
    for o in out[1:]:
        assert np.array_equal(out[0], o)


@pytest.mark.parametrize("ng,np_side", [(16, 16), (24, 24), (40, 40), (48, 48), (120, 120), (160, 80), (200, 200),
                                        (240, 120), (320, 160), (400, 200), (480, 240), (640, 160), (768, 192),
                                        (800, 200), (960, 240), (1000, 200), (1024, 128)])
def test_x_pass_line_tiles_equal_tma(ng, np_side, monkeypatch):
    """The x pass in line tiles (whole tiles, and the left-over columns of
    several planes in one) and the TMA-fed one move the particles alike, bit
    for bit, at the grid sides of every tile size."""
    rng = np.random.default_rng(ng)
    x = rng.random((np_side ** 3, 3), dtype=np.float32) * np.float32(ng * (1 - 2 ** -20))
    v = rng.standard_normal((np_side ** 3, 3), dtype=np.float32)
    out = []
    for flag in ("1", "2"):
        monkeypatch.setenv("HGPM_XTMA", flag)
        with make(ng, np_side) as s:
            s.load_state(x, v)
            s.cic()
            s.solve_gradient()
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            out.append(s.store_state())
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert not np.array_equal(out[0][1], v)


@pytest.mark.parametrize("np_side,ng", [(32, 32), (40, 40), (64, 32), (24, 48)])
@pytest.mark.parametrize("off", [0, 1, 3])
def test_device_state_round_trip_at_any_alignment(np_side, ng, off):
    """Device float3 arrays at 16-byte aligned and at 4-byte aligned addresses
    (blocks of 16^3 and 8^3 particles) load and store the same particles, and
    the floats around them are left alone."""
    import torch

    n = np_side ** 3
    rng = np.random.default_rng(off + np_side)
    x = rng.random((n, 3), dtype=np.float32) * np.float32(ng * (1 - 2 ** -20))
    v = rng.standard_normal((n, 3), dtype=np.float32)
    xd, vd, xo, vo = (torch.full((3 * n + 8,), -7.0, device="cuda") for _ in range(4))
    xd[off:off + 3 * n] = torch.from_numpy(x.reshape(-1)).cuda()
    vd[off:off + 3 * n] = torch.from_numpy(v.reshape(-1)).cuda()
    torch.cuda.synchronize()
    with make(ng, np_side) as s:
        s.load_state(x, v)
        xh, vh = s.store_state()
        cells = s.get_cells()
        s.load_state_device(xd.data_ptr() + 4 * off, vd.data_ptr() + 4 * off)
        assert np.array_equal(s.get_cells(), cells)
        s.store_state_device(xo.data_ptr() + 4 * off, vo.data_ptr() + 4 * off)
        s.sync()
    i = np.floor(x).astype(np.int64)
    assert np.array_equal(cells, (i[:, 0] * ng + i[:, 1]) * ng + i[:, 2])
    assert np.array_equal(vh, v) and np.abs(xh - x).max() <= np.spacing(np.float32(ng))
    for got, want in ((xo, xh), (vo, vh)):
        got = got.cpu().numpy()
        assert np.array_equal(got[off:off + 3 * n], want.reshape(-1))
        assert (got[:off] == -7.0).all() and (got[off + 3 * n:] == -7.0).all()


@pytest.mark.parametrize("ng,np_side", [(16, 16), (24, 24), (40, 40), (120, 120), (160, 80), (200, 200), (240, 120),
                                        (400, 200), (480, 240), (640, 160), (800, 200), (960, 240), (1000, 200),
                                        (1024, 128)])
def test_y_pass_line_tiles_equal_tma(ng, np_side, monkeypatch):
    """The y passes in line tiles and the TMA-fed ones move the particles
    alike, bit for bit, at the grid sides of every tile size."""
    rng = np.random.default_rng(ng)
    x = rng.random((np_side ** 3, 3), dtype=np.float32) * np.float32(ng * (1 - 2 ** -20))
    v = np.zeros_like(x)
    out = []
    for flag in ("0", "1"):
        monkeypatch.setenv("HGPM_NO_TMA", flag)
        with make(ng, np_side) as s:
            assert s.tuned_choices()["y_pass"] == (1 if flag == "0" else 0)
            s.load_state(x, v)
            s.cic()
            s.solve_gradient()
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            out.append(s.store_state())
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert out[0][1].any()


@pytest.mark.parametrize("ng,np_side", [(16, 16), (24, 24), (48, 48), (120, 120), (160, 80), (200, 200), (320, 160),
                                        (512, 128), (640, 160)])
@pytest.mark.parametrize("nbins,log_bins", [(7, False), (221, False), (64, True), (1024, True)])
def test_power_spectrum_bins_equal_double_binning(ng, np_side, nbins, log_bins):
    """Mode counts at every tile size equal a count whose bins are formed in
    double for every mode, with few, many, linear and log-spaced bins."""
    import torch

    x, v = lattice_state(np_side, ng, disp=1.0, seed=ng)
    with make(ng, np_side) as s:
        rl = s.params.rl
        s.load_state(x, v)
        k, p, n = s.power_spectrum(nbins, log_bins)
    i = torch.arange(ng, device="cuda")
    d = 2 * np.pi / rl
    kf = (torch.where(i > ng // 2 - 1, i - ng, i).double() * d).float()
    kz = kf[:ng // 2 + 1].clone()
    s2 = kf[:, None, None] * kf[:, None, None] + kf[None, :, None] * kf[None, :, None]
    kmag = (s2 + kz[None, None, :] * kz[None, None, :]).sqrt().double()
    kmax = np.sqrt(3 * ((ng // 2) * (ng // 2) * d * d))
    if log_bins:
        fb = torch.log(kmag / d) / (np.log(kmax / d) / nbins)
    else:
        fb = (kmag - d) / ((kmax - d) / nbins)
    w = torch.full_like(kmag, 2.0)
    w[:, :, 0] = w[:, :, ng // 2] = 1.0
    w[0, 0, 0] = w[ng // 2, ng // 2, ng // 2] = 0.0
    b = torch.trunc(torch.nan_to_num(fb, nan=-2.0, neginf=-2.0))
    w *= (b >= 0) & (b < nbins) & (fb > -1)
    want = torch.zeros(nbins, dtype=torch.float64, device="cuda")
    want.index_add_(0, b.clamp(0, nbins - 1).long().reshape(-1), w.reshape(-1))
    got = torch.from_numpy(n).double().cuda()
    # a mode whose double quotient is an integer but for its last bits may
    # round to the other side of it in another order of operations
    edge = ((fb - fb.round()).abs() < 1e-12 * nbins).double() * (w > 0)
    assert (got - want).abs().sum() <= 4 * edge.sum()
    assert n.sum() == int(w.sum())
    assert np.isfinite(p).all() and (p[n > 0] > 0).all()


@pytest.mark.parametrize("ng,np_side", [(240, 80), (256, 64), (320, 80), (384, 96), (400, 80), (480, 96), (512, 64),
                                        (640, 64), (1000, 40)])
def test_solve_of_large_sides_matches_double_fft(ng, np_side):
    """Sides beyond the oracle's reach: the forces against a double-precision
    transform of the same density on the device."""
    import torch

    x, v = lattice_state(np_side, ng, disp=1.2, seed=ng + 1)
    with make(ng, np_side) as s:
        s.load_state(x, v)
        s.cic()
        rho = torch.from_numpy(s.get_density()).cuda().double().reshape(ng, ng, ng)
        s.solve_gradient()
        f = s.get_force()
    d = np.float32(2.0 * np.pi / np.float32(ng))  # the oracle's cosine arguments
    c = torch.from_numpy(np.cos(np.arange(ng).astype(np.float32) * d).astype(np.float64)).cuda()
    g = 0.5 / (c[:, None, None] + c[None, :, None] + c[None, None, : ng // 2 + 1] - 3.0)
    g[0, 0, 0] = 0.0
    phi = torch.fft.irfftn(torch.fft.rfftn(rho) * g, s=(ng, ng, ng))
    del rho, g
    for dim in range(3):
        want = 0.5 * (torch.roll(phi, 1, dim) - torch.roll(phi, -1, dim))
        err = (torch.from_numpy(np.ascontiguousarray(f[dim])).cuda().reshape(ng, ng, ng) - want).abs().max()
        assert float(err / want.abs().max()) < FIELD_RTOL
    del phi, want, err
    torch.cuda.empty_cache()


@pytest.mark.parametrize("ng,np_side,choice", [(32, 32, "9"), (32, 32, "8"), (64, 64, "8"), (40, 40, "4"), (64, 32, "1"),
                                               (64, 32, "0"), (128, 16, "0"), (48, 96, None), (128, 128, "8"),
                                               (160, 160, "8")])
def test_dense_cells_reach_the_solve(ng, np_side, choice, monkeypatch):
    """Half the particles in a few cells, far from their blocks' windows and
    thousands of units of weight in each: the forces match the oracle's on the
    exact density, and the next deposits start from a clean accumulator."""
    if choice is None:
        monkeypatch.delenv("HGPM_DEPOSIT", raising=False)
    else:
        monkeypatch.setenv("HGPM_DEPOSIT", choice)
    x, v = lattice_state(np_side, ng, disp=1.0, vel=0.0, seed=3)
    hot = x.copy()
    for k, at in enumerate(((1.5, 2.0, ng - 0.5), (0.0, 0.0, 0.0), (ng - 1.0, 3.25, 7.0), (5.0, 5.0, 5.0))):
        hot[k * 2::8] = at
    with make(ng, np_side) as s:
        s.load_state(hot, v)
        s.cic()
        rho = s.get_density()
        s.solve_gradient()
        f = s.get_force()
        s.load_state(x, v)
        s.cic()
        clean = s.get_density()
        s.cic()
        again = s.get_density()
    ro = O.cic_deposit(hot.astype(np.float64), ng, O.cic_mass(ng, np_side))
    assert rho.max() > 512 and np.abs(rho - ro).max() <= 1e-6 * ro.max()
    assert rel_max_err(f, O.solve_gradient(rho.astype(np.float64), ref_quirks=True)) < FIELD_RTOL
    rc = O.cic_deposit(x.astype(np.float64), ng, O.cic_mass(ng, np_side))
    assert np.abs(clean - rc).max() <= 1e-6 * rc.max() and np.array_equal(clean, again)


@pytest.mark.parametrize("ng,np_side", [(16, 16), (16, 32), (24, 24), (32, 32), (32, 16), (32, 64), (40, 40)])
def test_one_kernel_solve_equals_passes(ng, np_side):
    """The whole solve of a small box in one kernel and the separate passes
    (which run while the phases are timed) leave the same bits: the state after
    steps, the potential's force grid and an empty accumulator."""
    x, v = lattice_state(np_side, ng, disp=1.5, vel=0.2, seed=11)
    got = []
    for timed in (False, True):
        with make(ng, np_side) as s:
            s.enable_timing(timed)
            s.load_state(x, v)
            s.cic()
            s.solve_gradient()
            first = s.get_force()
            s.cic()
            rho = s.get_density()
            s.solve_gradient()
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            again = s.get_force()
            xo, vo = s.store_state()
        assert np.array_equal(first, again)
        got.append((first, rho, xo, vo))
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("np_side", [32, 40, 64, 96])
def test_store_to_pageable_and_pinned_arrays(np_side):
    """The state stored into pageable arrays (in chunks; 32 below one chunk, 40
    and 96 with a part of one left) and into page-locked ones is the state on
    the device."""
    import torch

    n = np_side ** 3
    x, v = lattice_state(np_side, np_side, disp=1.0, vel=0.5, seed=4)
    with make(np_side) as s:
        s.load_state(x, v)
        for _ in range(2):
            xp, vp = s.store_state()
            assert np.array_equal(xp, x) and np.array_equal(vp, v)
        xl, vl = (torch.full((n, 3), -7.0).pin_memory() for _ in range(2))
        assert s.L.hgpm_store_state(s._h, ctypes.cast(xl.data_ptr(), F), ctypes.cast(vl.data_ptr(), F)) == 0
        assert np.array_equal(xl.numpy(), x) and np.array_equal(vl.numpy(), v)


@pytest.mark.parametrize("ng", [16, 24, 32, 40, 48])
@pytest.mark.parametrize("reps", [2, 40])
def test_autotune_leaves_the_current_potential(ng, reps, monkeypatch):
    """Straight after hgpm_autotune the context holds the state it had, the
    potential of that state, and a kick without another solve moves the
    particles as in a context that was never tuned, bit for bit: at the sides
    that solve in one kernel too, whatever the repetitions."""
    for k in ("HGPM_DEPOSIT", "HGPM_KICK", "HGPM_NO_TMA", "HGPM_XTMA", "HGPM_PLANE"):
        monkeypatch.delenv(k, raising=False)
    monkeypatch.setenv("HGPM_NO_TUNE_CACHE", "1")
    x, v = lattice_state(ng, ng, disp=1.5, vel=0.2, seed=ng)
    got = []
    for tune, force_first in ((False, False), (True, False), (True, True)):
        with make(ng) as s:
            s.load_state(x, v)
            if tune:
                s.autotune(reps=reps)
                xt, vt = s.store_state()
                assert np.array_equal(xt, x) and np.array_equal(vt, v)
            else:
                s.cic()
                s.solve_gradient()
            if force_first:
                s.get_force()
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            xo, vo = s.store_state()
            got.append((s.get_force(), xo, vo))
    assert not np.array_equal(got[0][2], v)
    for a in got[1:]:
        for p, q in zip(got[0], a):
            assert np.array_equal(p, q)


def test_power_spectrum_with_every_number_of_bins():
    """P(k) runs with any number of bins, also where the tile and the
    histograms come to just under 48 KB.  In a process of its own and in
    ascending order: what a kernel may use is asked for once, so a larger
    spectrum before would hide a smaller one that is refused."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = """
from tests.helpers import lattice_state, params_text
import hacc_gpm_b200 as H
for ng, bins in ((48, range(1, 500, 3)), (64, range(1, 500, 3)), (200, range(190, 230)), (256, range(110, 140)),
                 (320, range(340, 370)), (512, range(110, 140))):
    with H.Simulation(H.parse_params(params_text(ng, 32))) as s:
        s.load_state(*lattice_state(32, ng))
        total = {int(s.power_spectrum(n)[2].sum()) for n in bins}
        assert len(total) == 1, (ng, total)
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("np_side", [40, 64, 96])
@pytest.mark.parametrize("new", [(True, True), (True, False), (False, True), (False, False)])
def test_store_to_arrays_with_and_without_pages(np_side, new):
    """Stores into arrays that have no pages yet (through page-locked chunks from
    a context's third such store on) and into arrays that have them (by the
    driver), one of each too, give the state on the device and leave the bytes
    around the arrays alone."""
    import mmap

    n = np_side ** 3
    x, v = lattice_state(np_side, np_side, disp=1.0, vel=0.5, seed=4)
    with make(np_side) as s:
        s.load_state(x, v)
        for _ in range(5):
            maps, out = [], []
            for fresh in new:
                m = mmap.mmap(-1, 12 * n + 8192, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
                a = np.frombuffer(m, np.float32)
                if not fresh:
                    a[:] = -7.0
                maps.append((m, a))
                out.append(a[5:5 + 3 * n])
            ptr = [ctypes.cast(a.ctypes.data, F) for a in out]
            assert s.L.hgpm_store_state(s._h, *ptr) == 0
            assert np.array_equal(out[0].reshape(n, 3), x) and np.array_equal(out[1].reshape(n, 3), v)
            for fresh, (m, a) in zip(new, maps):
                around = 0.0 if fresh else -7.0
                assert (a[:5] == around).all() and (a[5 + 3 * n:] == around).all()


@pytest.mark.parametrize("ng", [16, 24, 32])
def test_autotune_weighs_the_one_kernel_solve(ng, monkeypatch):
    """A tuned small box steps in three kernels, as an untuned one does: the
    deposit, the whole solve and the kick.  What the tuner finds for the y pass,
    the x pass or another kick alone does not give up the one-kernel solve,
    which takes about half of what five passes take at these sides."""
    for k in ("HGPM_DEPOSIT", "HGPM_KICK", "HGPM_NO_TMA", "HGPM_XTMA", "HGPM_PLANE"):
        monkeypatch.delenv(k, raising=False)
    monkeypatch.setenv("HGPM_NO_TUNE_CACHE", "1")
    x, v = lattice_state(ng, ng, disp=1.0, vel=0.2, seed=ng)
    for _ in range(8):
        with make(ng) as s:
            s.load_state(x, v)
            picks = s.autotune(reps=10)
            assert all(p["ms"] > 0 for p in picks.values())
            s.kernel_launches(reset=True)
            s.cic()
            s.solve_gradient()
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            assert s.kernel_launches() <= 4, picks  # a windowed deposit is two
            assert picks["kick"]["choice"] == 7 and picks["y_pass"]["choice"] == 0 and picks["x_pass"]["choice"] != 1


@pytest.mark.parametrize("ng,np_side", [(16, 16), (24, 24), (32, 32), (40, 40), (32, 64)])
@pytest.mark.parametrize("var,values", [("HGPM_XTMA", ("1", "2")), ("HGPM_NO_TMA", ("0", "1"))])
def test_line_tiles_of_small_sides_equal_tma(ng, np_side, var, values, monkeypatch):
    """The separate y and x passes in line tiles at the sides whose solve is one
    kernel otherwise: with the phases timed the passes run, and they move the
    particles as the TMA-fed ones do, bit for bit."""
    rng = np.random.default_rng(ng)
    x = rng.random((np_side ** 3, 3), dtype=np.float32) * np.float32(ng * (1 - 2 ** -20))
    v = rng.standard_normal((np_side ** 3, 3), dtype=np.float32)
    out = []
    for value in values:
        monkeypatch.setenv(var, value)
        with make(ng, np_side) as s:
            s.enable_timing(True)
            s.load_state(x, v)
            s.kernel_launches(reset=True)
            s.cic()
            s.solve_gradient()
            assert s.kernel_launches() >= 6  # a deposit and five passes
            s.kick_drift(0.0123, 1.7, 0.3, 0.25, 2)
            out.append(s.store_state())
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert not np.array_equal(out[0][1], v)


@pytest.mark.parametrize("ng", [16, 24, 200, 512, 1000, 1024])
@pytest.mark.parametrize("rounded", [True, False])
def test_green_quotient_equals_division(ng, rounded):
    """The Green's function's quotient is the float of the double division for
    every mode of a side, with the cosines of rounded arguments and the exact
    ones.  Its error before the last rounding is below 2^-88, so that none of
    the 10^9 modes is expected to round otherwise (2^-35 of them in double, of
    which 2^-29 in float)."""
    if rounded:
        cosq = np.cos((np.arange(ng, dtype=np.float32) * np.float32(2 * np.pi / ng)).astype(np.float64)) - 1.0
    else:
        cosq = -2.0 * np.sin(np.pi * np.arange(ng) / ng) ** 2
    cosq = np.ascontiguousarray(cosq)
    n, most = ctypes.c_int64(-1), ctypes.c_int64(-1)
    rc = H.lib().hgpm_test_green(ng, cosq.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), ctypes.byref(n),
                                 ctypes.byref(most))
    assert rc == 0 and n.value == 0 and most.value == 0, (rc, n.value, most.value)


@pytest.mark.parametrize("ng,kernels", [(32, 1), (64, 2)])
def test_force_grid_on_demand_counts_its_kernels(ng, kernels):
    """hgpm_kernel_launches counts kernels: the force grid formed after a solve is
    the gradient alone where the potential is copied out of the paired records,
    the z pass and the gradient elsewhere."""
    with make(ng) as s:
        s.load_state(*lattice_state(ng, ng))
        s.cic()
        s.solve_gradient()
        s.kernel_launches(reset=True)
        s.get_force()
        assert s.kernel_launches() == kernels


@pytest.mark.parametrize("np_side,ng,choice", [
    (48, 24, 9), (64, 32, 8), (64, 48, 8), (80, 40, 8), (96, 48, 8), (96, 96, 9), (24, 16, 5),
    (40, 24, 4), (40, 40, 5), (64, 80, 5), (80, 96, 4), (96, 128, 4), (96, 160, 5), (120, 128, 4), (128, 160, 4),
    (128, 192, 5), (160, 192, 1), (200, 240, 1)])
def test_deposit_of_boxes_around_the_direct_rule(np_side, ng, choice, monkeypatch):
    """Which deposit a box takes by its blocks and its particles a cell (adding
    straight to the grid loses where many particles meet in a cell), and that
    its density is the window deposit's, bit for bit, with the particles drawn
    together too."""
    for k in ("HGPM_DEPOSIT", "HGPM_KICK"):
        monkeypatch.delenv(k, raising=False)
    monkeypatch.setenv("HGPM_NO_TUNE_CACHE", "1")
    x, v = lattice_state(np_side, ng, disp=0.7, seed=3)
    c = np.float32(ng / 2)
    clumped = np.mod(c + (x - c) * np.float32(0.2), np.float32(ng)).astype(np.float32)
    clumped[clumped >= ng] = 0
    got = []
    for force in (None, "0"):
        if force is not None:
            monkeypatch.setenv("HGPM_DEPOSIT", force)
        with make(ng, np_side) as s:
            assert s.tuned_choices()["deposit"] == (choice if force is None else 0)
            rho = []
            for state in (x, clumped):
                s.load_state(state, v)
                s.cic()
                rho.append(s.get_density())
        got.append(rho)
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
