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
