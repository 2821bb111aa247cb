"""The sources that are compiled in parts, a module each: build.py's counts are the headers'."""
import os
import re

from pfsoftlib_b200 import build


def _constants(header):
    text = open(os.path.join(build.CSRC, header)).read()
    out = {}
    for line in re.findall(r"constexpr int ([^;]+);", text):
        for name, value in re.findall(r"(\w+) = ([^,{]+)", line):
            out[name] = value.strip()
    return out


def test_counts_are_the_headers():
    dwt, fft = _constants("dwt.cuh"), _constants("fft_two.cuh")
    first, last, span = (int(dwt[k]) for k in ("kFixedFirst", "kFixedLast", "kFixedSpan"))
    assert build.PARTS["dwt_fixed.cu"] == ("DWT_PART", (last - first) // span + 1)
    assert build.PARTS["fft_two_kind.cu"] == ("FFT_KIND", int(fft["kKinds"]))
    names = [name for _, name, _ in build.units()]
    assert len(set(names)) == len(names) == len(build.sources()) - 2 + 13 + 7
