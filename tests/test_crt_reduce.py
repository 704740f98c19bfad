"""The CRT pre-pass's reduction as the library compiles it, built by the host compiler with signed overflow, shifts and
conversions trapped: its products exceed 32 bits by design, so they have to be unsigned.  Every modulus of the largest
context, extreme and random residues."""
import os
import subprocess

import numpy as np

import oracle as O
from conftest import ROOT

CSRC = os.path.join(ROOT, "sdpvibe_b200", "csrc")
MAIN = r"""
#include "crt_reduce.h"
#include <cmath>
#include <cstdio>
#include <cstring>
int main() {
  unsigned m, inv, a, y;
  while (scanf("%u %u %u", &m, &inv, &a) == 3) {
    const float q = fmaf((float)a, (float)((double)inv / m), 12582912.0f);
    unsigned qb;
    memcpy(&qb, &q, 4);
    y = sdpv::crt_reduce(a, inv, m, 0x4B400000u * m, qb);
    if (y != (unsigned long long)a * inv % m) return printf("%u %u %u: %u\n", m, inv, a, y), 1;
  }
  return 0;
}
"""


def test_reduction_has_no_signed_overflow(tmp_path):
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=undefined", "-fsanitize-undefined-trap-on-error", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    T = O.tables(58)
    rng = np.random.default_rng(0)
    rows = []
    for m, inv in zip(T.mods, T.inv):
        for a in (0, 1, 2, m // 2, m - 2, m - 1, *rng.integers(0, m, 20)):
            rows.append(f"{m} {inv} {a}")
    r = subprocess.run([str(exe)], input="\n".join(rows), text=True, capture_output=True)
    assert r.returncode == 0, r.stdout + r.stderr
    with open(os.path.join(CSRC, "crt.cu")) as f:
        assert "crt_reduce(" in f.read()
