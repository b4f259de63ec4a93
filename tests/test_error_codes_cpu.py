"""The code that a wait leaves behind when it runs out (wst_b200_device_error) names the kernel
by its high byte, checked in the sources on the CPU."""

import re
from collections import defaultdict
from pathlib import Path

# the wait for another rank's rows, which two kernels make in the same way
SHARED = {"4": {"attention_api.cu", "attn_rows.cu"}}

CSRC = Path(__file__).resolve().parent.parent / "whetstone_b200" / "csrc"


def test_a_code_belongs_to_one_kernel_file():
    files = defaultdict(set)
    for path in sorted(CSRC.glob("*.cu")):
        for code in re.findall(r"\b0x([0-9A-F]{3})u\b", path.read_text()):
            files[code[0]].add(path.name)
    assert len(files) >= 8
    shared = {f"0x{k}..": sorted(v) for k, v in files.items() if len(v) > 1 and v != SHARED.get(k)}
    assert not shared, shared
