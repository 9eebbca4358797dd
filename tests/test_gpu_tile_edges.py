"""The simplified flux path (paired values, faces summed in registers, shuffles and shared exchange rows) and the one-launch
ghost fill at the sizes where they can go wrong: one cell below, at and above the 32 x 8 tiles, axes of one to three cells,
every limiter, the three solvers with their own unit, walls, inlet, outflow, symmetry and connections. (The launch that
also carries the records and the clock is in test_gpu_surface.py.)

Tolerances: the FP64 production form against the oracle at the north-star gate of one step (1e-12, max-norm relative to
the field, momentum against its vector); the parity form bit for bit. The mixed form: every face flux carries a few FP32
roundings of the state's own size (p and rho u H), so a step moves the conserved variables by at most about
3 faces x 8 roundings x 2^-24 x the CFL-limited share of a cell (<= 1), 1.5e-6; bound 3e-6."""
import numpy as np
import pytest

import helpers as H
from mosegpu import abi

pytestmark = pytest.mark.gpu

SIZES = [(31, 7, 3), (32, 8, 4), (33, 9, 5), (34, 15, 2), (63, 16, 3), (65, 17, 1), (5, 41, 3)]


@pytest.fixture(scope="module")
def engine():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mosegpu.engine import Engine
    return Engine


def _steps(engine, case, precision, tol, exact=False, n=2):
    import oracle
    orc = oracle.Oracle(case)
    P = case.P0.copy()
    assert orc.step(P, n) == 0
    eng = engine(case, precision=precision)
    eng.step(n, graph=True)
    m = case.interior_mask()
    if exact:
        assert np.array_equal(eng.state()[:, m], P[:, m])
    e = H.rel_err(H.conserved(case, eng.state()), H.conserved(case, P))
    assert np.all(e <= tol), e
    assert eng.status().code == 0
    eng.close()


@pytest.mark.parametrize("riemann,limiter", [(abi.RS_HLLC, abi.LIM_MINMOD), (abi.RS_AUSMP, abi.LIM_VANLEER),
                                             (abi.RS_LMROE, abi.LIM_VANALBADA), (abi.RS_LMROE, abi.LIM_MC),
                                             (abi.RS_HLLC, abi.LIM_SUPERBEE), (abi.RS_AUSMP, abi.LIM_FIRST)])
@pytest.mark.parametrize("n", SIZES)
def test_duct_at_tile_edges(engine, n, riemann, limiter):
    from mosegpu import case as cs
    case = cs.duct_3d(widths=(n[0],), heights=(n[1],), depths=(n[2],), mach=1.5, amp=0.02, cfl=0.2, riemann=riemann,
                      limiter=limiter, bc={2: abi.BC_EXTRAPOLATION, 3: abi.BC_WALL, 4: abi.BC_SYMMETRY,
                                           5: abi.BC_EXTRAPOLATION, 6: abi.BC_EXTRAPOLATION})
    _steps(engine, case, abi.PREC_FP64_FAST, 1e-12)
    _steps(engine, case, abi.PREC_MIXED, 3e-6)


@pytest.mark.parametrize("n", [(2, 2, 2), (3, 2, 4), (33, 9, 2), (4, 33, 3)])
@pytest.mark.parametrize("mco", [1.0, 0.2])
def test_two_cell_periodic_blocks(engine, n, mco):
    """Connections whose donors are two cells deep (the one-launch fill copies both of their layers)."""
    from mosegpu import case as cs
    th = cs.ideal_gas_tables(mu=2e-2)
    h = [1.0 / q for q in n]

    def nodes(iu, iv, iw):
        return np.stack([iu * h[0], iv * h[1], iw * h[2]], axis=-1)

    def prim(c):
        x, y, z = (2 * np.pi * c[..., q] for q in range(3))
        return np.stack([1.0 + 0.1 * np.sin(x) * np.cos(y), 30 * np.sin(y) * np.cos(z), 20 * np.cos(x + z), 10 * np.sin(x),
                         8.0e4 + 2e3 * np.cos(y + z)])
    sch = dict(limiter=abi.LIM_VANALBADA, riemann=abi.RS_LMROE, visc=1, n_rk=3, ndir=3, cfl=0.4, prandtl=0.71, mco=mco,
               dt_additive=1)
    case = cs.layout_case("periodic", [[0, q] for q in n], nodes, (True,) * 3, {}, th, sch, prim)
    _steps(engine, case, abi.PREC_FP64, 1e-12, exact=True)
    _steps(engine, case, abi.PREC_FP64_FAST, 1e-12)


BCS = {"wall": abi.BC_WALL, "extrapolation": abi.BC_EXTRAPOLATION, "symmetry": abi.BC_SYMMETRY, "none": abi.BC_NONE}


@pytest.mark.parametrize("visc", [0, 1])
@pytest.mark.parametrize("n2", [1, 2, 3])
@pytest.mark.parametrize("low,high", [("wall", "wall"), ("wall", "extrapolation"), ("symmetry", "extrapolation"),
                                      ("extrapolation", "extrapolation"), ("symmetry", "none")])
def test_thin_axes_take_the_general_fill(engine, low, high, n2, visc):
    """The rules that merge the ghost passes, on a mesh with connections, against the sequential fill of the oracle: every
    pair of face types on an axis of one, two and three cells, bit for bit. (Viscous walls one or two cells apart are left
    out: their ghosts start from ghosts that are zero here, and the oracle's field leaves the tables.)"""
    from mosegpu import case as cs
    case = cs.multiblock_2d(cols=2, rows=1, widths=[6, 35], heights=[n2], visc=visc, mach=0.5, n_rk=3, cfl=0.2,
                            riemann=abi.RS_HLLC, limiter=abi.LIM_MINMOD,
                            bc={1: abi.BC_INFLOW, 2: abi.BC_EXTRAPOLATION, 3: BCS[low], 4: BCS[high],
                                5: abi.BC_EXTRAPOLATION, 6: abi.BC_EXTRAPOLATION})
    import oracle
    orc = oracle.Oracle(case)
    P = case.P0.copy()
    if orc.step(P, 2) != 0:
        pytest.skip("viscous faces one or two cells apart: the field leaves the tables in the oracle itself")
    eng = engine(case)
    eng.step(2, graph=True)
    m = case.interior_mask()
    assert np.array_equal(eng.state()[:, m], P[:, m])


@pytest.mark.parametrize("nb,riemann", [(1, abi.RS_LMROE), (2, abi.RS_HLLC)])
def test_autotuned_mixed_form_agrees(engine, nb, riemann):
    """Whatever mb_autotune picks of the mixed 3-D sweep (chunk, queue, staging, CTAs per SM) gives the untuned result to
    the rounding of the staged pressure (one FP32 ulp of p, 6e-8, in the faces of three stages and two steps; the bound
    of the staging test, 1e-6, max-norm of the conserved variables, momentum against its vector)."""
    from mosegpu import case as cs
    case = cs.taylor_green(n=64, blocks=nb, riemann=riemann, share_geometry=nb > 1)
    a, b = engine(case, precision=abi.PREC_MIXED), engine(case, precision=abi.PREC_MIXED)
    b.fill_ghosts()
    b.autotune()
    a.step(2, graph=True)
    b.step(2, graph=True)
    e = H.rel_err(H.conserved(case, a.state()), H.conserved(case, b.state()))
    assert np.all(e < 1e-6), e


def test_a_one_cell_axis_with_a_condition_on_one_side_only(engine):
    """A face without records keeps the ghosts its caller put there (a halo, say), and the cubic ghost of the opposite face
    of a one-cell axis reads them: the sequential fill of the oracle, bit for bit. The records of one side, of the other,
    and of half a side."""
    from mosegpu import case as cs
    import oracle
    g = np.random.default_rng(5)
    for keep in (lambda r: r["face"] != 4, lambda r: r["face"] != 3, lambda r: (r["face"] != 4) | (r["i"] > 17)):
        case = cs.multiblock_2d(cols=1, rows=1, widths=[35], heights=[1], visc=1, mach=0.5, n_rk=3,
                                riemann=abi.RS_HLLC, limiter=abi.LIM_MINMOD,
                                bc={1: abi.BC_INFLOW, 2: abi.BC_EXTRAPOLATION, 3: abi.BC_EXTRAPOLATION,
                                    4: abi.BC_EXTRAPOLATION, 5: abi.BC_EXTRAPOLATION, 6: abi.BC_EXTRAPOLATION})
        assert len(case.conn) == 0
        case.rec = case.rec[keep(case.rec)].copy()
        inside = case.P0[:, case.interior_mask()].mean(axis=1, keepdims=True)
        case.P0 = np.where(case.interior_mask()[None], case.P0, inside * (1.0 + 0.01 * g.standard_normal(case.P0.shape)))
        P = case.P0.copy()
        oracle.Oracle(case).fill_ghosts(P)
        eng = engine(case)
        eng.fill_ghosts()
        assert np.array_equal(eng.state(), P)
        eng.close()


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED])
@pytest.mark.parametrize("n", [(33, 4, 3), (32, 5, 2), (31, 6, 5), (40, 7, 3), (34, 13, 1)])
def test_run_time_solver_unit_at_its_tile_edges(engine, n, precision, monkeypatch, capfd):
    """The run-time solver unit cuts tiles of its own height: one row below, at and above it, and the SM holds as many of
    its CTAs as the registers are capped for (2 in the FP64 forms, 3 in the mixed one)."""
    from mosegpu import case as cs
    monkeypatch.setenv("MB_REPORT", "1")
    case = cs.duct_3d(widths=(n[0],), heights=(n[1],), depths=(n[2],), mach=1.5, amp=0.02, cfl=0.2, riemann=abi.RS_HLLE,
                      limiter=abi.LIM_MINMOD, bc={2: abi.BC_EXTRAPOLATION, 3: abi.BC_WALL, 4: abi.BC_SYMMETRY,
                                                  5: abi.BC_EXTRAPOLATION, 6: abi.BC_EXTRAPOLATION})
    engine(case, precision=precision).close()
    report = capfd.readouterr().err
    assert ", %d CTAs per SM (" % (3 if precision == abi.PREC_MIXED else 2) in report, report
    _steps(engine, case, precision, 3e-6 if precision == abi.PREC_MIXED else 1e-12, exact=precision == abi.PREC_FP64)


def test_hllc_star_flux_has_no_cancellation(engine):
    """2000 Riemann problems with states that FP32 holds exactly, first order: the mixed form's fluxes against the FP64
    form's, rms over the rms flux of each conserved variable. The contact speed carries a rounding or two of the sound
    speed, five times the rms velocity here: 2^-24 / sqrt(3) x 5 = 1.7e-7 in the mass and energy fluxes (measured 1.5e-7
    and 2.1e-7, bound 3e-7). Summed as F + S (U* - U), differences of large terms, the mass flux had 4.3e-7."""
    from mosegpu import case as cs
    n, w = 16000, 8
    case = cs.riemann_1d(n=n, riemann=abi.RS_HLLC, limiter=abi.LIM_FIRST)
    g = np.random.default_rng(3)
    s = np.stack([g.uniform(0.5, 2.0, n // w), g.uniform(-0.5, 0.5, n // w), np.zeros(n // w), np.zeros(n // w),
                  g.uniform(0.5, 4.0, n // w)]).astype(np.float32).astype(np.float64)
    case.interior(case.P0, 0)[:] = np.repeat(s, w, axis=1).reshape(case.interior(case.P0, 0).shape)
    out = []
    for p in (abi.PREC_FP64, abi.PREC_MIXED):
        eng = engine(case, precision=p)
        eng.fill_ghosts()
        out.append(eng.residual().cpu().numpy()[:, case.interior_mask()].reshape(5, n))
        eng.close()
    face = [q for q in range(w, n - w) if q % w in (0, w - 1)]  # the cells at a jump: one face of each is a Riemann problem
    ref, got = out[0][:, face], out[1][:, face]
    rho, u, pr = s[0], s[1], s[4]
    scale = {0: rho * u, 1: rho * u * u + pr, 4: u * (3.5 * pr + 0.5 * rho * u * u)}
    area = case.blocks[0]["fm1"].reshape(-1, 4)[0, 3]
    for v in (0, 1, 4):
        e = np.sqrt(np.mean((got[v] - ref[v]) ** 2)) / (area * np.sqrt(np.mean(scale[v] ** 2)))
        assert e <= 3e-7, (v, e)


def test_wall_friction_below_an_ulp_of_the_pressure_is_kept(engine):
    """A record's convective and viscous contributions are FP32 values added one after the other in FP64: the friction of an
    inclined wall shows in the mixed form's residual although it is below an FP32 rounding of the pressure on that wall. A
    uniform stream along the walls of a rotated channel has no other viscous flux, so the difference of two residuals with
    different viscosities is the friction's; to 1e-5 (a few FP32 roundings of the friction itself) it is the FP64 form's."""
    from mosegpu import case as cs
    co, si, n = np.cos(0.5), np.sin(0.5), (40, 9, 1)
    R = cs.ideal_gas_tables()["R"]
    diff = []
    for precision in (abi.PREC_FP64, abi.PREC_MIXED):
        res = []
        for mu in (2.5e-7, 5e-7):
            def nodes(i, j, k):
                x, y = i / 40.0, j / 40.0
                return np.stack([co * x - si * y, si * x + co * y, k / 40.0], axis=-1)

            def prim(c):
                return np.stack([np.full(c.shape[:-1], v) for v in (1e5 / (R * 300.0), 100.0 * co, 100.0 * si, 0.0, 1e5)])
            sch = dict(limiter=abi.LIM_MINMOD, riemann=abi.RS_HLLC, visc=1, n_rk=3, ndir=2, cfl=0.4, prandtl=0.71)
            case = cs.layout_case("rotated", [[0, q] for q in n], nodes, (False,) * 3,
                                  {1: abi.BC_EXTRAPOLATION, 2: abi.BC_EXTRAPOLATION, 3: abi.BC_WALL, 4: abi.BC_WALL,
                                   5: abi.BC_EXTRAPOLATION, 6: abi.BC_EXTRAPOLATION}, cs.ideal_gas_tables(mu=mu), sch, prim)
            eng = engine(case, precision=precision)
            eng.fill_ghosts()
            r = case.interior(eng.residual().cpu().numpy(), 0)
            res.append(np.concatenate([r[1:3, 2:-2, 0], r[1:3, 2:-2, -1]]))
            eng.close()
        diff.append(res[1] - res[0])
    scale = np.abs(diff[0]).max()
    assert 0 < scale < 1e5 / 40 ** 2 * 6e-8  # below an ulp of the pressure force
    assert np.abs(diff[1] - diff[0]).max() < 1e-5 * scale, (np.abs(diff[1]).max(), scale)


@pytest.mark.parametrize("riemann,limiter", [(abi.RS_LMROE, abi.LIM_VANALBADA), (abi.RS_HLLC, abi.LIM_VANALBADA),
                                             (abi.RS_AUSMP, abi.LIM_VANALBADA), (abi.RS_HLLC, abi.LIM_MC)])
@pytest.mark.parametrize("n,visc", [((24, 20, 1), 1), ((33, 9, 1), 0), ((20, 1, 24), 1), ((1, 24, 20), 1)])
def test_periodic_axis_one_cell_deep(engine, n, visc, riemann, limiter):
    """The second ghost layer of a periodic axis one cell deep comes from no interior cell but from the first one, which is
    copied before; until something fills it the faces beside it read no temperature from there."""
    import oracle
    from mosegpu import case as cs
    th = cs.ideal_gas_tables(mu=2e-2)
    h = [1.0 / q for q in n]

    def prim(c):
        x, y, z = (2 * np.pi * c[..., q] * (n[q] > 1) for q in range(3))
        return np.stack([1.0 + 0.1 * np.sin(x) * np.cos(y + z), 30 * np.sin(y) * np.cos(z), 20 * np.cos(x + z),
                         10 * np.sin(x + y), 8.0e4 + 2e3 * np.cos(y + z)])
    sch = dict(limiter=limiter, riemann=riemann, visc=visc, n_rk=3, ndir=3, cfl=0.3, prandtl=0.71, dt_additive=1)
    case = cs.layout_case("slab", [[0, q] for q in n], lambda i, j, k: np.stack([i * h[0], j * h[1], k * h[2]], axis=-1),
                          (True,) * 3, {}, th, sch, prim)
    P = case.P0.copy()
    oracle.Oracle(case).fill_ghosts(P)
    eng = engine(case)
    eng.fill_ghosts()
    assert np.array_equal(eng.state(), P)
    eng.close()
    _steps(engine, case, abi.PREC_FP64, 1e-12)
    _steps(engine, case, abi.PREC_FP64_FAST, 1e-12)
    _steps(engine, case, abi.PREC_MIXED, 3e-6)


@pytest.mark.parametrize("riemann", [abi.RS_LMROE, abi.RS_HLLC, abi.RS_AUSMP])
def test_a_face_without_records_beside_empty_ghosts(engine, riemann):
    """No record, no flux and no ghosts: the faces next to such a boundary reach cells of zero density, whose temperature is
    not a number, and keep finite fluxes as in the parity form."""
    from mosegpu import case as cs
    case = cs.multiblock_2d(cols=1, rows=1, widths=[35], heights=[9], visc=0, mach=0.5, n_rk=3, cfl=0.2, riemann=riemann,
                            limiter=abi.LIM_VANALBADA, bc={1: abi.BC_INFLOW, 2: abi.BC_EXTRAPOLATION, 3: abi.BC_WALL,
                                                           4: abi.BC_EXTRAPOLATION, 5: abi.BC_EXTRAPOLATION,
                                                           6: abi.BC_EXTRAPOLATION})
    case.rec = case.rec[case.rec["face"] != 4].copy()
    case.P0 = np.where(case.interior_mask()[None], case.P0, 0.0)
    _steps(engine, case, abi.PREC_FP64, 1e-12, exact=True)
    _steps(engine, case, abi.PREC_FP64_FAST, 1e-12)
