"""The mat-vec's own choice of K chunks (csrc/matvec_rules.h) over the shapes
its entry points accept: every choice meets the launch's conditions, and
tiles that do not pair up are not split for pairs."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "inspire-gpu_b200", "csrc")

SWEEP = r"""
#include <cstdio>
#include <initializer_list>
#include "matvec_rules.h"
using namespace ipb;
int main() {
    int bad = 0;
    for (size_t r = 1; r <= 34; ++r) {  // 1024 .. 32768, then 65536 and 98304
        const size_t rows = r <= 32 ? 1024 * r : 32768 * (r - 31);
        for (size_t cols = 128; cols <= 128 * 600; cols += 128)
            for (int nq = 1; nq <= 32; ++nq)
                for (int sms : {1, 132, 148}) {
                    const int kc = matvec_tc_kchunk_rows(rows, cols, sms, nq);
                    if (CHECK) continue;
                    if (bad++ < 5) std::printf("rows %zu cols %zu queries %d SMs %d: %d\n", rows, cols, nq, sms, kc);
                }
    }
    return bad != 0;
}
"""


def _sweep(tmp_path, check):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "sweep.cpp", tmp_path / "sweep"
    src.write_text(SWEEP.replace("CHECK", check))
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_every_default_chunk_is_accepted_by_the_launch(tmp_path):
    _sweep(tmp_path, "mv_kchunk_ok(rows, kc)")


def test_odd_tile_counts_split_for_the_last_wave_only(tmp_path):
    """An odd number of 128-column tiles runs one tile per item.  A chunk whose
    double already gives two items per SM is there only because the items'
    last wave is fuller."""
    _sweep(tmp_path, "cols / 128 % 2 == 0 || 2 * kc > kKChunk || rows % (2 * (size_t)kc) || "
                     "cols / 128 * (rows / (2 * kc)) < 2 * (size_t)sms || "
                     "2 * ((cols / 128 * (rows / (2 * kc)) + sms - 1) / sms) > (cols / 128 * (rows / kc) + sms - 1) / sms")
