"""Arithmetic of the CRT kernels as the library compiles it, built by the host compiler with signed overflow, shifts and
conversions trapped.  The pre-pass's reduction (its products exceed 32 bits by design, so they have to be unsigned): every
modulus of the largest context, extreme and random residues.  The barrier phases that a kernel whose wait gave up lets its
last table copies complete: against the copies of every schedule, counted one by one."""
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


def _build(tmp_path, main):
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(main)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=undefined", "-fsanitize-undefined-trap-on-error", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    return str(exe)


def test_reduction_has_no_signed_overflow(tmp_path):
    exe = _build(tmp_path, MAIN)
    T = O.tables(58)
    rng = np.random.default_rng(0)
    rows = []
    for m, inv in zip(T.mods, T.inv):
        for a in (0, 1, 2, m // 2, m - 2, m - 1, *rng.integers(0, m, 20)):
            rows.append(f"{m} {inv} {a}")
    r = subprocess.run([exe], input="\n".join(rows), text=True, capture_output=True)
    assert r.returncode == 0, r.stdout + r.stderr
    with open(os.path.join(CSRC, "crt.cu")) as f:
        assert "crt_reduce(" in f.read()


PARITY = r"""
#include "crt_reduce.h"
#include <cstdio>
int main() {
  unsigned loads, nslot, s;
  while (scanf("%u %u %u", &loads, &nslot, &s) == 3) printf("%d\n", sdpv::last_load_parity(loads, nslot, s));
  return 0;
}
"""


def test_last_copies_are_waited_for(tmp_path):
    rows, want = [], []
    for nslot in range(1, 5):
        for nchunk in range(nslot, 5):                                  # resident (nslot = nchunk) and streamed tables
            for tiles in range(1, 4):
                copies = [0] * nslot                                    # completed phases of each slot's barrier
                for loads in range(nslot * tiles + nchunk * (tiles - 1) + 1):
                    for s in range(nslot):
                        rows.append(f"{loads} {nslot} {s}")
                        want.append(copies[s] - 1 & 1 if copies[s] else -1)
                    copies[loads % nslot] += 1
    r = subprocess.run([_build(tmp_path, PARITY)], input="\n".join(rows), text=True, capture_output=True, check=True)
    assert [int(v) for v in r.stdout.split()] == want
    with open(os.path.join(CSRC, "crt.cu")) as f:
        src = f.read()
    # a product's phase is flipped after its wait: the one to drain is the flipped parity's other
    assert "mbar_wait(&H.done, phase ^ 1u, err)" in src and "last_load_parity(loads, nslot, s)" in src
