"""The rules of the chained launches (programmatic dependent launch), checked on the sources: a race
that breaking them makes shows only by chance on a GPU."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "solprop_b200" / "csrc"
CHAINED = sorted(p for p in CSRC.glob("*.cu") if "await_previous_kernel();" in p.read_text())


def _kernels(text):
    """(name, parameters, body's first statement) of every __global__ function with a body."""
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(([^{;]*?)\)\s*\{\s*([^;]*;)", text):
        yield m.groups()


def test_chained_kernels_wait_first():
    launched, waiting = set(), set()
    for path in CHAINED:
        text = path.read_text()
        launched |= set(re.findall(r"launch_chained\((k_\w+)", text))
        # the cluster transforms' width picks the kernel launched
        launched |= set(re.findall(r"case \d+: return (k_\w+)<R, \d>;", text))
        waiting |= {name for name, _, first in _kernels(text) if first == "await_previous_kernel();"}
    assert len(launched) >= 15 and launched <= waiting, launched - waiting


def test_chained_kernels_read_the_chain_coherently():
    """Non-coherent loads (__ldg, const __restrict__ parameters of a kernel) are for constant tables."""
    sources = [*CHAINED, CSRC / "fft.cuh", CSRC / "fft_regs.cuh", CSRC / "stage_output.cuh"]
    loads = {(p.name, a) for p in sources for a in re.findall(r"__ldg\(\s*([\w.]+)", p.read_text())}
    assert loads and {a for _, a in loads} <= {"table", "tw", "a.twiddles"}, loads
    for path in CHAINED:
        for name, parameters, first in _kernels(path.read_text()):
            assert first != "await_previous_kernel();" or "__restrict__" not in parameters, name


def test_no_kernel_lets_the_next_in_before_it_ends():
    """A trigger ahead of a kernel's work makes the whole chain resident, waiting on SMs that other
    kernels and streams need: runs of rows of 4 096 were up to a tenth slower than unchained."""
    assert not [p.name for p in CSRC.glob("*.cu*") if re.search(r'"griddepcontrol.launch_dependents', p.read_text())]
