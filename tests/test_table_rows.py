"""Every row of the gas tables is held to the table before it is read, whatever the temperature: a state off the table, or
one that is not a number, is reported by the state check and the thermo guard, and must not read outside an array."""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

from mosegpu import abi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mose-gpu_b200", "csrc")

STATE = """
import sys
sys.path[:0] = [%r, %r]
import numpy as np, oracle
from mosegpu import abi, case as cs
case = cs.multiblock_2d(cols=2, rows=1, widths=[6, 7], heights=[5], riemann=%d, n_rk=3)
P = case.P0.copy()
case.interior(P, 0)[4, -1, 2, 0] = np.nan   # beside the connection
case.interior(P, 1)[4, 3, 0, 0] = 1e12      # on a wall
o = oracle.Oracle(case)
o.fill_ghosts(P)
o.residual(P)
"""


def sources():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cuh", ".cu")):
            with open(os.path.join(CSRC, f)) as h:
                yield f, re.sub(r"//[^\n]*", "", h.read())


def test_no_table_row_is_a_bare_conversion():
    """A row comes from tidx or trow; the two other conversions of a temperature clamp the rows they make."""
    for f, s in sources():
        for m in re.finditer(r"int (\w+) = \(int\)(T\w*)[^;]*;", s):
            after = s[m.end():m.end() + 200]
            held = re.search(r"max\(p\.tmin, min\(%s, p\.tmax\)\)" % m.group(1), after)
            assert held, (f, m.group(0))


@pytest.mark.parametrize("riemann", [abi.RS_SLAU, abi.RS_SLAU2, abi.RS_HLLE, abi.RS_EXACT, abi.RS_HLLC, abi.RS_LMROE,
                                     abi.RS_AUSMP, abi.RS_MICZEKROE])
def test_oracle_reads_inside_its_tables(riemann):
    """In a process of its own: a read outside the table ends it."""
    code = STATE % (os.path.join(ROOT, "mose-gpu_b200"), os.path.join(ROOT, "oracle"), riemann)
    assert subprocess.run([sys.executable, "-c", code]).returncode == 0


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [abi.PREC_FP64, abi.PREC_FP64_FAST, abi.PREC_MIXED])
@pytest.mark.parametrize("riemann", [abi.RS_SLAU, abi.RS_SLAU2, abi.RS_HLLE])
def test_engine_stays_usable_after_a_state_off_the_table(riemann, precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from mosegpu import case as cs
    from mosegpu.engine import Engine
    case = cs.multiblock_2d(cols=2, rows=1, widths=[6, 7], heights=[5], riemann=riemann, n_rk=3)
    eng = Engine(case, precision=precision)
    eng.fill_ghosts()
    good = eng.residual().cpu().numpy()
    P = case.P0.copy()
    case.interior(P, 0)[4, -1, 2, 0] = np.nan
    case.interior(P, 1)[4, 3, 0, 0] = 1e12
    eng.set_state(P)
    eng.fill_ghosts()
    bad = eng.residual().cpu().numpy()
    assert not np.isfinite(case.interior(bad, 0)[:, -1, 2, 0]).all()
    eng.set_state(case.P0)
    eng.fill_ghosts()
    m = case.interior_mask()
    assert np.array_equal(eng.residual().cpu().numpy()[:, m], good[:, m])
    eng.close()
