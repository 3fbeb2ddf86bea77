"""The bound of a kernel's dynamic shared memory belongs to the function, and
the library is called without Python's lock: a call that set it to its own
launch's size could lower it between another thread's setting and launch."""

import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "redbirdpy_b200" / "csrc"


def test_shared_memory_bounds_are_constants():
    found = 0
    for path in sorted(CSRC.glob("*.cu*")):
        text = path.read_text()
        for m in re.finditer(r"cudaFuncAttributeMaxDynamicSharedMemorySize,[\s\\]*([^;]*?)\)+\s*(?:!=|;)", text):
            found += 1
            value = re.sub(r"\(int\)", "", m.group(1)).strip()
            assert re.fullmatch(r"k[A-Z]\w*", value) or re.search(rf"\bconstexpr [\w ]+ {value} =", text), \
                (path.name, value)
    assert found >= 10
