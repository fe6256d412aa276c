"""The line lengths of the built-in passes: the list that the dispatch is made
from and the one that the build compiles, each length a translation unit (and
so a module that is loaded) of its own."""
import os
import re

from crava_b200 import build


def test_every_length_is_compiled_on_its_own():
    with open(os.path.join(build.CSRC, "fft_lengths.cuh")) as f:
        text = f.read()
    listed = [int(n) for n in re.findall(r"X\((\d+)\)", text)]
    assert listed == build.LENGTHS and len(set(listed)) == len(listed)
    units = build.units()
    assert len({obj for _, obj, _ in units}) == len(units)
    per_length = [(obj, flags) for src, obj, flags in units if src == "fft_len.cu"]
    assert per_length == [(f"fft_len{n}.o", [f"-DCRAVA_LENGTH={n}"]) for n in listed]
