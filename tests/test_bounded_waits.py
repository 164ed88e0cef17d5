"""The tensor-core kernels' give-up paths, checked on the sources (no wait runs out on a healthy GPU).

A wait that runs out, or another role's failure flag, must take a whole warp out of its role: the
tensor-memory instructions that follow are warp-wide, and lanes that left while others went on
would leave the warp waiting for itself."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "solprop_b200" / "csrc"


def _kernels(name):
    """Each kernel's text, cut at the barrier that ends its roles: (roles, ending)."""
    text = (CSRC / name).read_text()
    for m in re.finditer(r"__global__.*?\n}\n", text, re.S):
        if "mbar_wait(" in m.group():
            roles, ending = re.split(r"\n  __syncwarp\(\);[^\n]*\n  __syncthreads\(\);\n", m.group(), maxsplit=1)
            yield roles, ending


@pytest.mark.parametrize("name, count", [("modal_gemm.cu", 2), ("mlp_tcgen05.cu", 1)])
def test_whole_warp_roles_leave_as_one(name, count):
    kernels = list(_kernels(name))
    assert len(kernels) == count
    for roles, ending in kernels:
        role = roles[re.search(r"else if \(warp >= \d\)", roles).end():]
        waits = [line for line in role.splitlines() if "mbar_wait(" in line]
        assert waits and all("warp_agrees(" in line and "!failed" in line for line in waits)
        # no lane leaves, or goes round again, on a flag it read by itself
        assert not re.search(r"if \((?!!warp_agrees)[^\n]*failed[^\n]*\)", role)
        assert not re.search(r"for \([^\n]*failed[^\n]*\)", role)
        # once every role has ended, the loads asked for and not taken land before the CTA leaves
        assert re.search(r"for \(\w+ h = consumed; h < loads; \+\+h\) mbar_wait", ending)


def test_column_hand_over_waits_long_enough():
    """A tile gives an earlier one at least 2^26 ns: polls times the sleep between them."""
    text = (CSRC / "column_kernels.cu").read_text()
    limit = int(re.search(r"kSpinLimit = 1L << (\d+);", text).group(1))
    assert (1 << limit) * int(re.search(r"__nanosleep\((\d+)\)", text).group(1)) >= 1 << 26
