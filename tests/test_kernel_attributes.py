"""Kernel attributes belong to the device that is current when they are set: the
library looks at the return code of every such call and keeps no process-wide
note of having made it."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "getm_gb300" / "csrc"


def test_attributes_are_set_per_device():
    found = 0
    for path in sorted(CSRC.glob("*.cu*")):
        text = path.read_text()
        assert not re.search(r"static\s+bool\s+\w+\s*=", text), path.name
        for m in re.finditer(r"cudaFuncSetAttribute\(", text):
            found += 1
            assert re.search(r"[!=]=\s*cudaSuccess", text[m.end():m.end() + 200]), (path.name, m.start())
    assert found
