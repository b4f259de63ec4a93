"""Which global memory the kernels read through the read-only path, checked in their source on
the CPU.  A kernel that is launched while the one ahead of it still runs may use that path
(`__ldg`, ld.global.nc) only for data that nothing writes as long as the kernel lives: weights,
scales, biases, rotary tables.  Activations and query rows are what the launch ahead writes, and
the compiler may move such a read in front of the wait for that launch."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "whetstone_b200" / "csrc"

CONSTANT = {
    "ct", "st",                 # rotary tables
    "g.bias", "a.bias",
    "a.qw", "a.si", "at",       # packed words, scale bytes
    "g.sb", "a.sb",             # (d, dmin) of a row
}


def test_the_read_only_path_is_taken_for_constants_alone():
    seen = set()
    for path in sorted(CSRC.glob("*.cu*")):
        for arg in re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()?([\w.]+)", path.read_text()):
            assert arg in CONSTANT, f"{path.name}: __ldg({arg} ...)"
            seen.add(arg)
    assert seen, "no read found: the pattern no longer matches the sources"
