"""Shared-memory arrays of bytes or half words in the kernels say their alignment: the
type alone promises less than the word accesses that such arrays are there for."""
import os
import re

from conftest import PKG


def test_narrow_shared_arrays_are_aligned():
    found, csrc = [], os.path.join(PKG, "csrc")
    for name in sorted(os.listdir(csrc)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(csrc, name)) as f:
            text = f.read()
        for m in re.finditer(r"__shared__\s+([^;]*?)\b(u?int8_t|u?int16_t|unsigned char|char)\s+\w+\[",
                             text):
            if "__align__" not in m.group(1):
                found.append(f"{name}:{text.count(chr(10), 0, m.start()) + 1}")
    assert not found
