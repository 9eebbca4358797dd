"""The k-chunk of the sweep's tiles does not change a bit of the result, whatever stages the tile: a chunk's first plane
computes the k-face below itself from the four planes it staged, and must be done with them before the next plane lands
in the first one's slot. Odd row counts (no tensor map: the mixed form stages by plain loads), every chunk short enough
that most planes start a chunk."""
import numpy as np
import pytest

from mosegpu import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED])
@pytest.mark.parametrize("n", [33, 53])
def test_short_chunks_are_bit_identical(precision, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mosegpu import case as cs
    from mosegpu.engine import Engine
    case = cs.taylor_green(n=n)
    assert case.ncell % 2 == 1
    m = case.interior_mask()
    ref = None
    for kc in (64, 1, 2, 3):
        eng = Engine(case, precision=precision)
        eng.set_tuning(kc, False)
        eng.step(3, graph=True)
        s = eng.state()[:, m]
        ref = s if ref is None else ref
        assert np.array_equal(s, ref), kc
        eng.close()


def _step_us(torch, eng, n=40):
    """median time of a step of five runs of n"""
    eng.step(n)
    t = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        eng.step(n)
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b) / n * 1e3)
    return sorted(t)[2]


def test_the_tuner_does_not_lose_to_the_untuned_chunk():
    """53^3 fills the device with tiles of a few planes, fewer than the tuner's fixed candidates: what it keeps is no slower
    than what ran before it (15 % for the noise of its three timed launches; tiles of 8 planes take 1.4 times as long)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mosegpu import case as cs
    from mosegpu.engine import Engine
    eng = Engine(cs.taylor_green(n=53), precision=abi.PREC_MIXED)
    assert eng.tuning()[0] < 8  # the chunk the sweeps take, not a default
    before = _step_us(torch, eng)
    eng.fill_ghosts()
    eng.autotune()
    after = _step_us(torch, eng)
    assert after <= 1.15 * before, (before, after, eng.tuning())
    eng.close()


def test_depth_classes_nobody_timed_follow_the_mesh():
    """mb_autotune fixes a chunk for the depth classes it timed only: another mesh in the same context gets its own for the
    others. mb_set_tuning fixes all."""
    import ctypes as C
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mosegpu import case as cs
    from mosegpu.engine import Engine

    def box(n):
        th = cs.ideal_gas_tables(mu=2e-2)
        h = [1.0 / q for q in n]
        sch = dict(limiter=abi.LIM_VANALBADA, riemann=abi.RS_LMROE, visc=1, n_rk=3, ndir=3, cfl=0.4, prandtl=0.71,
                   mco=1.0, dt_additive=1)
        return cs.layout_case("box", [[0, q] for q in n], lambda i, j, k: np.stack([i * h[0], j * h[1], k * h[2]], axis=-1),
                              (True,) * 3, {}, th, sch, lambda c: np.stack([np.full(c.shape[:-1], v) for v in (1., 10., 5., 2., 8e4)]))

    def mesh_of(eng, case):
        m = abi.MBMesh()
        m.nblk, m.nrec, m.nconn, m.ncell_total = len(case.blocks), len(eng._rec), len(eng._conn), case.ncell
        m.blk, m.rec, m.conn = eng._blk, eng._rec.ctypes.data, eng._conn.ctypes.data
        return m
    deep, flat = box((53, 53, 53)), box((40, 40, 12))
    want = Engine(deep, precision=abi.PREC_MIXED)
    ref = Engine(flat, precision=abi.PREC_MIXED)
    flat.P0 = np.concatenate([flat.P0, np.ones((5, deep.ncell - flat.ncell))], axis=1)
    flat.ncell = deep.ncell
    eng = Engine(flat, precision=abi.PREC_MIXED)
    assert eng.tuning()[0] == ref.tuning()[0]
    eng.fill_ghosts()
    eng.autotune()
    assert eng.lib.mb_reconfigure(eng.ctx, C.byref(mesh_of(want, deep))) == abi.MB_OK
    assert eng.tuning()[0] == want.tuning()[0]
    eng.set_tuning(5, False)
    assert eng.lib.mb_reconfigure(eng.ctx, C.byref(mesh_of(eng, flat))) == abi.MB_OK
    assert eng.tuning()[0] == 5
    for e in (eng, want, ref):
        e.close()
    one = Engine(cs.riemann_1d(n=64))
    assert one.tuning()[:2] == (16, 0)
    one.close()


def test_a_step_of_few_long_tiles_takes_no_longer_than_its_parts():
    """64^3 in 64 tiles of 16 planes, fewer than the SMs: a step's launches one after another take what its ghost fills and
    sweeps take by themselves. Chained, their tiles shared SMs and the step took 1.37 times that."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mosegpu import case as cs
    from mosegpu.engine import Engine
    eng = Engine(cs.taylor_green(n=64), precision=abi.PREC_MIXED)
    eng.set_tuning(16, False)
    step = _step_us(torch, eng)
    parts = sum(sum(eng.profile_stage(q, 20)) for q in (1, 2, 3)) * 1e3
    assert step <= 1.15 * parts, (step, parts)
    eng.close()


@pytest.mark.parametrize("irs", [0, 2])
def test_the_staging_is_the_one_measured_for_the_sweeps_that_run(irs, monkeypatch, capfd):
    """The 4-CTA form of the 3-D sweep stages by plain loads. Where it does not run, with residual smoothing (whose sweeps
    write residuals) or after mb_set_tuning, the staging is the faster of the two timed without it."""
    import re
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mosegpu import case as cs
    from mosegpu.engine import Engine
    case = cs.taylor_green(n=128, blocks=4, riemann=abi.RS_HLLC, share_geometry=True)
    case.scheme["irs"] = irs
    eng = Engine(case, precision=abi.PREC_MIXED)
    eng.fill_ghosts()
    monkeypatch.setenv("MB_REPORT", "1")
    eng.autotune()
    six, five = re.search(r"main list:.*?\(6-value ([\d.]+) ms, 5-value ([\d.]+) ms\)", capfd.readouterr().err).groups()
    if not irs:
        eng.set_tuning(8, False)
    if six != five:
        assert eng.staging_mode() == (float(five) < float(six)), (six, five)
    eng.close()
