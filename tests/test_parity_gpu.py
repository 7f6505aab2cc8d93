"""Parity of the CUDA engine (through the C-ABI) with the CPU oracle.

Every case runs the same seeded inputs through liblbmx.so on cuda:0 and
through the FP64 restatement of the reference step, then compares the
density, force-corrected velocity (the reference's d_rho / d_u) and the
post-collision populations.

Tolerances: FP32 storage |diff| <= 2e-5 on populations, rho and u
(single-precision rounding carried over a few hundred steps; the
reference's own FP32 arithmetic differs from FP64 by the same order).
16-bit offset storage is checked against FP32 at the tolerance its
mantissa allows (FP16 5e-4, BF16 4e-3 on u, relative to the peak speed).
"""
import numpy as np
import pytest

import cases as C

pytestmark = pytest.mark.gpu

TOL = 2e-5


def run_both(c, steps, storage=0, options=0):
    o = C.make_oracle(c)
    L = C.make_lattice(c, storage=storage, options=options)
    o.step(steps)
    L.step(steps)
    return o, L


def compare(o, L, tol=TOL, pops=True):
    ro, uo, _ = o.moments()
    rl, ul, _ = L.moments()
    dr = np.abs(rl - ro).max()
    du = np.abs(ul - uo).max()
    assert np.isfinite(rl).all() and np.isfinite(ul).all()
    assert dr <= tol, "rho max diff %g" % dr
    assert du <= tol, "u max diff %g" % du
    if pops:
        fo = o.populations()
        fl = L.populations()
        m = np.isfinite(fl)
        df = np.abs(fl[m] - fo[m]).max()
        assert df <= tol, "populations max diff %g" % df
        # the engine drops (NaN) only values that streamed out of the domain
        assert not (~m & ~lost_slots(L, o)).any()
    return dr, du


def lost_slots(L, o):
    """Slots whose post-collision value left a non-periodic domain in the last step."""
    ny, nx = L.ny, L.nx
    lost = np.zeros((9, ny, nx), bool)
    if L.t % 2 == 0:
        return lost
    per = L.params.periodic_x, L.params.periodic_y
    cx = [0, 1, 0, -1, 0, 1, -1, -1, 1]
    cy = [0, 0, 1, 0, -1, 1, 1, -1, -1]
    X, Y = np.meshgrid(np.arange(nx), np.arange(ny))
    for q in range(1, 9):
        out = np.zeros((ny, nx), bool)
        if not per[0]:
            out |= (X + cx[q] < 0) | (X + cx[q] >= nx)
        if not per[1]:
            out |= (Y + cy[q] < 0) | (Y + cy[q] >= ny)
        lost[q] = out
    return lost


@pytest.mark.parametrize("op", [C.BGK, C.MRT, C.CM])
@pytest.mark.parametrize("quirks", [0, C.QUIRKS_REFERENCE])
def test_taylor_green(op, quirks):
    c = C.taylor_green(64, 48, op=op, quirks=quirks)
    o, L = run_both(c, 101)
    compare(o, L)


def test_taylor_green_cm_optimal():
    c = C.taylor_green(64, 48, op=C.CM_OPT, quirks=C.QUIRKS_REFERENCE)
    o, L = run_both(c, 30)
    compare(o, L, tol=5e-5)
    ao = o.averages()
    aL = L.averages()
    assert np.allclose(aL, ao, rtol=1e-5)


def test_cm_optimal_lagged_close_to_strict():
    c = C.taylor_green(64, 48, op=C.CM_OPT)
    Ls = C.make_lattice(c)
    Ll = C.make_lattice(c, options=1)
    Ls.step(20)
    Ll.step(20)
    _, us, _ = Ls.moments()
    _, ul, _ = Ll.moments()
    assert np.abs(us - ul).max() < 1e-4


@pytest.mark.parametrize("op", [C.BGK, C.MRT, C.CM])
def test_cavity_regularized(op):
    c = C.cavity_regularized(48, 40, op=op, quirks=C.QUIRKS_REFERENCE)
    o, L = run_both(c, 150)
    compare(o, L)


@pytest.mark.parametrize("steps", [1, 2, 77])
def test_cavity_moving_wall(steps):
    c = C.random_state(C.cavity_moving_wall(48, 40, op=C.MRT), seed=3)
    o, L = run_both(c, steps)
    compare(o, L)


def test_cavity_zouhe_top():
    c = C.cavity_zouhe(40, 32, op=C.BGK)
    o, L = run_both(c, 120)
    compare(o, L)


@pytest.mark.parametrize("op", [C.BGK, C.MRT, C.CM])
@pytest.mark.parametrize("quirks", [0, C.QUIRKS_REFERENCE])
def test_poiseuille_body_force(op, quirks):
    c = C.poiseuille(64, 32, op=op, quirks=quirks)
    o, L = run_both(c, 200)
    compare(o, L)


def test_poiseuille_cm_optimal():
    # with the shipped regression the adapter sets the higher-order rates
    # near 2; single-precision rounding then grows by ~x1e4 over 40 steps in
    # the oracle's own FP32 build as well, so parity is checked on 20 steps
    c = C.poiseuille(64, 32, op=C.CM_OPT, nu=0.02, quirks=C.QUIRKS_REFERENCE)
    o, L = run_both(c, 20)
    compare(o, L, tol=1e-5)


@pytest.mark.parametrize("quirks", [0, C.QUIRKS_REFERENCE])
@pytest.mark.parametrize("outlet", ["zg", "pressure"])
def test_channel_zouhe_inlet(quirks, outlet):
    c = C.channel(96, 48, quirks=quirks, outlet=outlet)
    o, L = run_both(c, 150)
    compare(o, L)


def test_channel_parabolic_zouhe_pressure():
    c = C.channel(96, 48, inlet="parabolic", outlet="zouhe_p", op=C.BGK)
    o, L = run_both(c, 150)
    compare(o, L)


@pytest.mark.parametrize("op", [C.BGK, C.MRT])
def test_channel_reference_corner_boundaries(op):
    # CornerBoundary (cornerBoundaries.cuh:38-82) at the inlet's two corners:
    # a uniform Zou-He inlet at the corners' fixed ux = 0.03; own-node rules
    # on populations that partly come from the edge store
    c = C.random_state(C.channel(96, 48, op=op, u_in=0.03), seed=13)
    c["flags"][0, 0] = C.CORNER_BOTTOM_LEFT
    c["flags"][-1, 0] = C.CORNER_TOP_LEFT
    o, L = run_both(c, 151)
    compare(o, L)


@pytest.mark.parametrize("quirks", [0, C.QUIRKS_REFERENCE])
def test_channel_ibm_cylinder(quirks):
    mk = C.cylinder_markers(32.3, 24.1, 6.0, 32)
    c = C.channel(96, 48, quirks=quirks, markers=mk, u_in=0.05)
    o, L = run_both(c, 120)
    compare(o, L, tol=5e-5)
    uo, ro, Fo = o.markers()
    FL, dl = L.marker_forces()
    assert np.abs(FL - Fo).max() <= 5e-5 * max(1.0, np.abs(Fo).max())
    assert np.allclose(dl, -Fo.sum(axis=1), atol=1e-4)


@pytest.mark.parametrize("storage", [0, 1])
@pytest.mark.parametrize("stencil_quirks", [0, C.QUIRKS_REFERENCE])
def test_ibm_is_bitwise_reproducible(storage, stencil_quirks):
    """The spread adds each node's stencil contributions in a fixed order, so
    two runs of the same IBM channel agree bit for bit: populations, marker
    forces and drag/lift."""
    mk = C.cylinder_markers(32.3, 24.1, 6.0, 32)
    c = C.channel(96, 48, quirks=stencil_quirks, markers=mk, u_in=0.05)
    runs = []
    for _ in range(2):
        L = C.make_lattice(c, storage=storage)
        L.step(200)
        F, dl = L.marker_forces()
        runs.append((np.nan_to_num(L.populations()), F, np.asarray(dl)))
    (pa, Fa, da), (pb, Fb, db) = runs
    assert np.array_equal(pa, pb)
    assert np.array_equal(Fa, Fb) and np.array_equal(da, db)


def test_step_forces_series():
    """lbmx_step_forces records every step's drag and lift inside the IBM
    kernel; each entry equals what lbmx_ibm_forces reports after that step,
    and pageable, pinned and device series are the same bit for bit."""
    import torch

    mk = C.cylinder_markers(32.3, 24.1, 6.0, 32)
    c = C.channel(96, 48, markers=mk, u_in=0.05, inlet="parabolic", outlet="zouhe_p")
    L = C.make_lattice(c)
    want = []
    for _ in range(12):
        L.step(1)
        want.append(L.marker_forces()[1])
    want = np.array(want)
    L2 = C.make_lattice(c)
    got = L2.step_forces(12)
    assert np.allclose(got, want, rtol=1e-12, atol=1e-15)
    L3 = C.make_lattice(c)
    pinned = torch.zeros(24, dtype=torch.float64).pin_memory()
    L3.step_forces(12, out=pinned)
    L3.synchronize()
    L4 = C.make_lattice(c)
    dev = torch.zeros(24, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()  # the fill runs on torch's stream, the steps on the lattice's
    L4.step_forces(12, out=dev)
    L4.synchronize()
    assert np.array_equal(pinned.numpy().reshape(12, 2), got)
    assert np.array_equal(dev.cpu().numpy().reshape(12, 2), got)


def test_poiseuille_ibm_reference_scenario():
    # PoiseuilleScenario::add_bodies: cylinder of D=16 at (48, NY/2), 16 markers
    mk = C.cylinder_markers(48.0, 50.0, 8.0, 16)
    c = C.poiseuille(150, 100, op=C.BGK, quirks=C.QUIRKS_REFERENCE, markers=mk)
    o, L = run_both(c, 100)
    compare(o, L, tol=5e-5)


def test_solid_cylinder_flag():
    c = C.channel(80, 40, quirks=C.QUIRKS_REFERENCE)
    X, Y = np.meshgrid(np.arange(80), np.arange(40))
    c["flags"][(X - 25) ** 2 + (Y - 20) ** 2 <= 36] = C.CYLINDER
    o, L = run_both(c, 100)
    compare(o, L)


@pytest.mark.parametrize("nx,ny", [(5, 4), (37, 29), (130, 3)])
def test_ragged_sizes(nx, ny):
    c = C.random_state(C.taylor_green(nx, ny, op=C.MRT), seed=nx)
    o, L = run_both(c, 9)
    compare(o, L)
    c = C.random_state(C.cavity_regularized(max(nx, 4), max(ny, 4), op=C.BGK), seed=ny)
    o, L = run_both(c, 9)
    compare(o, L)


@pytest.mark.parametrize("case", ["cavity", "taylor_green"])
@pytest.mark.parametrize("steps", [20, 21])
def test_staged_tiles_many_per_cta(case, steps):
    # 1024 x 514: 8 x 128 staged interior tiles, several per persistent CTA,
    # so every stage of the shared-memory ring is refilled more than once
    if case == "cavity":
        c = C.random_state(C.cavity_moving_wall(1024, 514, op=C.MRT, nu=0.05), seed=11)
    else:
        c = C.random_state(C.taylor_green(1024, 514, op=C.BGK), seed=12)
    o, L = run_both(c, steps)
    compare(o, L)


@pytest.mark.parametrize("op", [C.BGK, C.MRT, C.CM, C.CM_OPT])
def test_brinkman_drag(op):
    # per-node Brinkman field (no reference counterpart) against the oracle's
    # restatement of the same term; CM_OPT over a short horizon (its clamped
    # rate amplifies rounding once the drag has slowed the flow)
    c = C.channel_brinkman(96, 40, op=op, sigma=3.0, gamma_scale=0.3 if op != C.CM_OPT else 0.02)
    c["u"] = c["u"] + 0.02 * np.random.default_rng(3).standard_normal(c["u"].shape)
    o = C.make_oracle(c)
    o.set_gamma(c["gamma"])
    L = C.make_lattice(c)
    L.set_brinkman(c["gamma"])
    steps = 20 if op == C.CM_OPT else 60
    o.step(steps)
    L.step(steps)
    compare(o, L)
    # and gamma = 0 is the plain step, bit for bit
    L0 = C.make_lattice(c)
    L0.set_brinkman(np.zeros_like(c["gamma"]))
    L1 = C.make_lattice(c)
    L0.step(7)
    L1.step(7)
    np.testing.assert_array_equal(L0.moments()[1], L1.moments()[1])


@pytest.mark.parametrize("storage,tol", [(1, 5e-4), (2, 4e-3)])
def test_offset_storage_against_fp32(storage, tol):
    c = C.cavity_moving_wall(96, 96, op=C.MRT, nu=0.05)
    L32 = C.make_lattice(c)
    L16 = C.make_lattice(c, storage=storage)
    L32.step(300)
    L16.step(300)
    _, u32, s32 = L32.moments()
    _, u16, s16 = L16.moments()
    err = np.abs(u16 - u32).max() / 0.1
    assert err <= tol * 10, "relative u error %g" % err
    # FP64 sums: 16-bit storage keeps total mass within its rounding
    assert abs(s16[0] - s32[0]) / s32[0] < 1e-3


def test_mass_conservation_and_determinism_full_size():
    # 1024^2 lid-driven cavity, MRT, moving-wall lid: bounce-back conserves mass
    c = C.cavity_moving_wall(1024, 1024, op=C.MRT, nu=0.1024)
    L = C.make_lattice(c)
    _, _, s0 = (None, None, None)
    L.step(1)
    _, _, s1 = L.moments()
    L.step(199)
    r, u, s2 = L.moments()
    assert abs(s2[0] - s1[0]) / s1[0] < 1e-6
    L2 = C.make_lattice(c)
    L2.step(200)
    r2, u2, _ = L2.moments()
    assert np.array_equal(u, u2) and np.array_equal(r, r2)


def test_flag_validation():
    import lbmx
    c = C.taylor_green(16, 16)
    L = C.make_lattice(c)
    bad = np.zeros((16, 16), np.uint8)
    bad[3, 3] = 4
    with pytest.raises(lbmx.LbmxError) as e:
        L.set_flags(bad)
    assert e.value.code == 4
    bad[3, 3] = 200
    with pytest.raises(lbmx.LbmxError):
        L.set_flags(bad)
    bad[3, 3] = C.CORNER_BOTTOM_LEFT + 1  # one past the last flag
    with pytest.raises(lbmx.LbmxError):
        L.set_flags(bad)
    bad[:] = 0
    bad[5, 0] = C.PRESSURE_OUTLET
    with pytest.raises(lbmx.LbmxError):
        L.set_flags(bad)
    with pytest.raises(lbmx.LbmxError) as e:
        lbmx.Lattice(2, 16)
    assert e.value.code == 1


def test_nonfinite_detection():
    import lbmx
    c = C.taylor_green(32, 32)
    c["rho"] = c["rho"].copy()
    c["rho"][4, 4] = np.nan
    L = C.make_lattice(c)
    with pytest.raises(lbmx.LbmxError) as e:
        L.step(2, flags=lbmx.STEP_STORE_MOMENTS | lbmx.STEP_CHECK_FINITE)
    assert e.value.code == 7


@pytest.mark.parametrize("nx,ny", [(64, 17), (130, 33), (66, 3)])
def test_averages_take_each_density_at_full_precision(nx, ny):
    """CM_OPT: the pre-pass' mass sum is the sum of every node's density,
    each rounded to 2^-30 by itself, to the last unit."""
    c = C.random_state(C.taylor_green(nx, ny, op=C.CM_OPT, nu=0.05), seed=3)
    L = C.make_lattice(c)
    f = L.populations()
    cx, cy = [0, 1, 0, -1, 0, 1, -1, -1, 1], [0, 0, 1, 0, -1, 1, 1, -1, -1]
    f = [np.roll(f[q], (cy[q], cx[q]), axis=(0, 1)) for q in range(9)]
    rho = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7])) + f[8]
    # the perimeter's units of two nodes take the general path, which adds in order
    edge = np.ones((ny, nx), bool)
    edge[1:-1, 2:-2] = False
    seq = f[0]
    for q in range(1, 9):
        seq = seq + f[q]
    rho = np.where(edge, seq, rho)
    assert rho.dtype == np.float32
    want = int(np.rint(rho.astype(np.float64) * 2.0 ** 30).astype(np.int64).sum())
    assert int(L.opt_partials()[0]) == want
