"""Kernels of a chained stage start before the kernels that write their input have ended, so what they read of arrays that
kernels write must be ordinary loads: the read-only path (ld, __ldg, const __restrict__ kernel parameters) is defined only
for data that no one writes during the kernel's whole life. A wrong load of this kind shows no wrong value on most runs, so
the sources are looked through instead: the headers of every chained kernel and of all that those kernels call."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mose-gpu_b200", "csrc")
HEADERS = ["mb_engine.cuh", "mb_face_fast.cuh"]
# the names the sources give to arenas and work arrays: stage input and output, old state, Ur, local steps, RK4
# accumulator, record contributions; pp is the pressure column of an arena
WRITTEN = r"(?:P|Pin|Pold|Pout|pp|q0|sf\.P|p\.ur|p\.dtl|p\.acc4|p\.recflux)"


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", HEADERS)
def test_arrays_that_kernels_write_are_read_by_ordinary_loads(name):
    s = source(name)
    bad = re.findall(r"\b(?:ld|ldg_|__ldg)\(\s*(?:&\s*)?%s\b[^;]*" % WRITTEN, s)
    assert not bad, bad
    bad = re.findall(r"const double\s*\*\s*__restrict__\s+(?:P|Pin|Pold|PO)\b", s)
    assert not bad, bad


def test_the_looked_for_names_are_the_ones_in_use():
    """The pattern above covers the parameters of the chained kernels and of the record functions."""
    s = source("mb_engine.cuh")
    args = re.search(r"k_sweep\((.*?)\)\s*\{", s, re.S).group(1)
    assert set(re.findall(r"double\s*\*\s*(\w+)", args)) <= {"Pin", "Pold", "Pout", "Rout"}
    args = re.search(r"k_records\((.*?)\)\s*\{", s, re.S).group(1)
    assert set(re.findall(r"double\s*\*\s*(\w+)", args)) == {"P"}


def test_the_records_do_not_read_what_the_clock_of_their_launch_writes():
    """k_records may carry the case clocks in a block of its own: clock_groups writes the DevState of every case there, so
    no other block of that launch reads one (the done flag only where the launch has no clock)."""
    s = source("mb_engine.cuh")
    body = s[s.index("k_records("):]
    body = body[:body.index("\n}\n")]
    reads = re.findall(r"[^;{}\n]*\bp\.st\b[^;\n]*", body)
    assert reads and all("!sf.clock &&" in r for r in reads), reads
    # the functions it calls for a record take nothing from the clocks
    for name in HEADERS:
        h = source(name)
        for f in re.findall(r"MB_HD void (?:bc_\w+|conn_fast|ghost_record)\([^{]*\{.*?\n\}\n", h, re.S):
            assert not re.search(r"\bp\.st\b|->time\b|->dt\b|rampf", f), f[:80]
