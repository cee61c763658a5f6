"""Fixed-point coordinate differences of the pair histogram (csrc/wrap32.h), compiled with a trap on
signed overflow, against the minimum image in exact integers; the kernel forms them by this function
alone."""
import os
import re
import subprocess

import numpy as np

from tests.helpers import ROOT

CSRC = os.path.join(ROOT, "mdff20_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include "wrap32.h"
int main() {
    int a, b;
    while (scanf("%d %d", &a, &b) == 2) printf("%d\\n", mdffgpu::wrap_diff(a, b));
}
"""


def test_differences_wrap_without_signed_overflow(tmp_path):
    src, exe = tmp_path / "w.cpp", tmp_path / "w"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-fsanitize=signed-integer-overflow", "-fsanitize-undefined-trap-on-error",
                    f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    edge = [-2 ** 31, -2 ** 31 + 1, -2 ** 30, -1, 0, 1, 2 ** 30, 2 ** 31 - 1]
    rnd = np.random.default_rng(1).integers(-2 ** 31, 2 ** 31, size=(500, 2)).tolist()
    pairs = [(a, b) for a in edge for b in edge] + rnd
    out = subprocess.run([str(exe)], input="\n".join(f"{a} {b}" for a, b in pairs), text=True, check=True,
                         capture_output=True).stdout.split()
    assert [int(x) for x in out] == [(a - b + 2 ** 31) % 2 ** 32 - 2 ** 31 for a, b in pairs]


def test_the_kernel_uses_it():
    text = open(os.path.join(CSRC, "rdf.cu")).read()
    assert len(re.findall(r"wrap_diff\(me\[m\]\.[xyz], o\.[xyz]\)", text)) == 3
    assert not re.search(r"me\[m\]\.[xyz] - o\.", text)
