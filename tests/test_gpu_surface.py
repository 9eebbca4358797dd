"""The merged launches of a stage: where no boundary record reads a ghost the records, the ghost fill and (in mb_step) the
case clock share one launch; elsewhere the fill is a launch of its own, or several where one ghost is computed from another.
Which of them a mesh takes shows in the number of launches of a step; the results are the oracle's sequential fill and
record loop, bit for bit in the parity form, within the one-step gates in the production forms (1e-12, and 3e-6 for the
mixed form: its bound in test_gpu_tile_edges.py)."""
import numpy as np
import pytest

import helpers as H
from mosegpu import abi

pytestmark = pytest.mark.gpu

E, W, S, I = abi.BC_EXTRAPOLATION, abi.BC_WALL, abi.BC_SYMMETRY, abi.BC_INFLOW
OUT = (abi.BC_OUTLET, (0.95e5, 0.5))
ISO = (abi.BC_WALL_T, (310.0,))


@pytest.fixture(scope="module")
def engine():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mosegpu.engine import Engine
    return Engine


def _channel(n1, n2, faces, visc, **kw):
    """One block, i faces 1 / 2 and j faces as given, extrapolated k faces; in the viscous cases the ghosts start as the
    uniform state."""
    from mosegpu import case as cs
    scheme = {q: kw.pop(q) for q in ("irs", "local_dt") if q in kw}
    a = dict(mach=0.5, n_rk=3, cfl=0.2, riemann=abi.RS_HLLC, limiter=abi.LIM_MINMOD)
    a.update(kw)
    case = cs.multiblock_2d(cols=1, rows=1, widths=[n1], heights=[n2], visc=visc,
                            bc={1: faces[0], 2: faces[1], 3: faces[2], 4: faces[3], 5: E, 6: E}, **a)
    case.scheme.update(scheme)
    if visc:
        m = case.interior_mask()
        case.P0 = np.where(m[None], case.P0, case.P0[:, m][:, :1])
    assert len(case.conn) == 0
    return case


def _run(engine, case, precision, n=2):
    import oracle
    orc = oracle.Oracle(case)
    P = case.P0.copy()
    assert orc.step(P, n) == 0
    m = case.interior_mask()
    eng = engine(case, precision=precision)
    eng.step(n, graph=True)
    assert eng.status().code == 0
    if precision == abi.PREC_FP64 and OUT[0] not in case.rec["type"]:  # an outlet's pow is not the host library's
        assert np.array_equal(eng.state()[:, m], P[:, m])
    e = H.rel_err(H.conserved(case, eng.state()), H.conserved(case, P))
    assert np.all(e <= (3e-6 if precision == abi.PREC_MIXED else 1e-12)), e
    before = eng.launches
    eng.step(1, graph=False)
    launches = eng.launches - before
    eng.close()
    return launches


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED])
@pytest.mark.parametrize("n,faces,visc,merged", [
    ((33, 9), (I, E, W, W), 1, True),
    ((33, 9), (I, OUT, ISO, W), 1, True),
    ((32, 8), (I, OUT, S, W), 0, True),
    ((32, 8), (I, OUT, S, W), 1, False),    # a viscous symmetry face reads the transverse ghosts
    ((31, 3), (I, E, W, E), 1, True),
    ((3, 33), (I, E, W, W), 1, True),
    ((33, 2), (I, OUT, S, S), 0, True),     # the cell behind the boundary cell is the opposite one
    ((33, 1), (I, OUT, S, S), 0, False),    # and here a ghost
    ((2, 33), (I, OUT, W, W), 1, True),
    ((33, 1), (E, E, E, E), 0, True),
    ((1, 33), (E, E, E, E), 1, True),
])
def test_one_launch_for_records_ghosts_and_clock(engine, n, faces, visc, merged, precision):
    case = _channel(n[0], n[1], faces, visc)
    launches = _run(engine, case, precision)
    assert (launches == 2 * 3) == merged, launches  # per stage: the merged launch and the sweep


def test_walls_two_cells_apart_keep_their_order(engine):
    """A wall's ghost reads the opposite wall's: launches of their own."""
    assert _run(engine, _channel(33, 2, (I, E, W, W), 0), abi.PREC_FP64) > 2 * 3


@pytest.mark.parametrize("kw", [dict(n_rk=1), dict(n_rk=2), dict(n_rk=4), dict(irs=2), dict(local_dt=1),
                                dict(riemann=abi.RS_HLLE), dict(riemann=abi.RS_LMROE, limiter=abi.LIM_VANALBADA)])
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_MIXED])
def test_other_steps_with_merged_launches(engine, kw, precision):
    """RK1, RK2, RK4, residual smoothing, local time steps and the run-time solver unit on a mesh of the merged form."""
    _run(engine, _channel(33, 9, (I, E, W, W), 1, **kw), precision, n=3)


@pytest.mark.parametrize("low,high,n2", [(E, E, 1), (S, abi.BC_NONE, 1), (E, E, 2), (S, E, 2), (S, abi.BC_NONE, 2)])
def test_thin_viscous_axes(engine, low, high, n2):
    """Viscous faces one or two cells apart."""
    _run(engine, _channel(35, n2, (I, E, low, high), 1, mach=0.1, cfl=0.05), abi.PREC_FP64)


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("at", [(31, 7), (32, 8), (0, 15), (69, 19)])
def test_a_value_that_is_not_finite_stays_within_its_stencil(engine, at, bad, precision):
    """A pressure that is not finite at a tile's corner, in its neighbour or at a boundary: the residuals of cells that no
    face reading it touches (two cells along each axis) keep their bits, whatever the shuffles, the exchange rows and the
    reciprocals carry."""
    case = _channel(70, 20, (E, E, E, E), 0)
    P = case.P0.copy()
    case.interior(P, 0)[4, at[0], at[1], 0] = bad
    res = []
    for state in (case.P0, P):
        eng = engine(case, precision=precision)
        eng.set_state(state)
        eng.fill_ghosts()
        res.append(case.interior(eng.residual().cpu().numpy(), 0)[:, :, :, 0])
        eng.close()
    i, j = np.meshgrid(np.arange(70), np.arange(20), indexing="ij")
    di, dj = abs(i - at[0]), abs(j - at[1])
    far = ~(((di <= 2) & (dj == 0)) | ((dj <= 2) & (di == 0)))
    assert np.array_equal(res[0][:, far], res[1][:, far])
    assert not np.isfinite(res[1][:, at[0], at[1]]).all()


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED])
def test_a_supersonic_hllc_face_takes_nothing_from_downstream(engine, precision):
    """At Mach 2 the flux of a face is its left state's. A cell that is not a number spoils the right state of the face two
    cells upstream and the states of the next one: the residual two cells upstream keeps its bits."""
    case = _channel(70, 20, (E, E, E, E), 0, mach=2.0)
    P = case.P0.copy()
    case.interior(P, 0)[4, 33, 9, 0] = np.nan
    res = []
    for state in (case.P0, P):
        eng = engine(case, precision=precision)
        eng.set_state(state)
        eng.fill_ghosts()
        res.append(case.interior(eng.residual().cpu().numpy(), 0)[:, :, 9, 0])
        eng.close()
    assert np.array_equal(res[0][:, :32], res[1][:, :32])
    assert not np.isfinite(res[1][:, 32]).all()
