"""CPU test of a rule on the sources: a kernel started by launch_after
(ffg_internal.h) may be resident before the kernel that writes its operands has
finished, so the read-only path (__ldg, or a const __restrict__ kernel parameter)
is for the constant tables and the host's job records alone; operands, residues
and digits are read with plain loads behind after_previous()."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "fastfib_b200" / "csrc"
# twiddle tables, and the prefix sums uploaded with a batch's CRT records
TABLES = {"tw", "itwA", "itwB", "r3f", "r3i", "P.r3f", "P.r3i", "P.twl", "P.twh", "first"}
RECORDS = {"CrtJob", "SchoolJob", "ShiftJob", "CombJob", "KhatJob", "LeafJob"}


def _sources():
    for f in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        yield f.name, re.sub(r"//[^\n]*", "", f.read_text())


def test_read_only_loads_of_tables_only():
    seen = 0
    for name, text in _sources():
        for m in re.finditer(r"__ldg\(", text):
            arg = re.match(r"&([\w.]+)\[", text[m.end():])
            assert arg and arg.group(1) in TABLES, f"{name}: __ldg({text[m.end(): m.end() + 50]!r}"
            seen += 1
        assert "ld.global.nc" not in text, name
    assert seen >= 10


def test_restrict_parameters_are_job_records():
    """Of every kernel that waits for the one before it."""
    kernels = 0
    for name, text in _sources():
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(([^{;]*)\)\s*\{\s*after_previous\(\);", text):
            kernels += 1
            for p in m.group(2).split(","):
                if "__restrict__" in p:
                    kind, var = re.match(r"\s*const (\w+) \*__restrict__ (\w+)", p).groups()
                    assert kind in RECORDS or (kind, var) == ("uint32_t", "first"), (name, m.group(1), p)
    assert kernels >= 20
