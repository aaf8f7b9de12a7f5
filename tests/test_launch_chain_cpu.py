"""The rule that orders the kernels of a pass (csrc/omni_pdl.cuh), checked in the sources: a kernel lets its
dependents start only behind a wait for the kernel in front that every one of its threads runs."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "cleffa_b200" / "csrc"


def test_dependents_are_released_behind_an_unconditional_wait():
    found = 0
    for path in sorted(CSRC.glob("*.cu")):
        lines = [re.sub(r"//.*", "", line).strip() for line in path.read_text().splitlines()]
        for i, line in enumerate(lines):
            if "dep_launch();" in line:
                found += 1
                assert lines[i - 1] == "dep_wait();", f"{path.name}:{i + 1}: {lines[i - 1]!r} in front of dep_launch"
            elif "dep_wait" in line:
                assert line == "dep_wait();" and "dep_launch();" in lines[i + 1], f"{path.name}:{i + 1}: {line!r}"
    assert found >= 12
