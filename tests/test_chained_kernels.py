"""Kernels launched while their predecessor still runs (programmatic dependent
launch) wait for it before anything else and promise nothing about memory that
it writes: checked on the source, since a broken promise seldom shows."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "subway_gb300" / "csrc"


def _chained():
    names = set()
    for f in CSRC.glob("*.cu"):
        names |= set(re.findall(r"\bchain\(\s*(k_\w+)", f.read_text()))
    return names


def _kernels():
    """name -> (parameters, body) of every kernel in the sources."""
    out = {}
    for f in [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]:
        txt = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(k_\w+)\s*\(([^)]*)\)\s*\{", txt):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(txt[i], 0)
                i += 1
            out[m.group(1)] = (m.group(2), txt[m.end():i - 1])
    return out


def test_every_chained_kernel_waits_first():
    kernels, chained = _kernels(), _chained()
    assert len(chained) >= 10 and chained <= set(kernels)
    for k in sorted(chained):
        assert kernels[k][1].strip().startswith("chain_wait();"), k


def test_chained_kernels_take_no_restrict_pointers():
    kernels = _kernels()
    for k in sorted(_chained()):
        assert "__restrict__" not in kernels[k][0], k


def test_read_only_loads_are_of_arrays_that_no_kernel_writes():
    txt = (CSRC / "sgw_kernels.cuh").read_text()
    args = re.findall(r"__ldg\(([^;]*?)\)", txt)
    assert args
    for a in args:
        assert re.search(r"\boff\b|\bh\.base\b", a), a
