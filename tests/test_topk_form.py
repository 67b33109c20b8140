"""Which kernel a top-k call takes, from the rule compiled for the host: the clusters only where they were measured to be
faster than a block a row, every list and every slice within its shared memory."""

import ctypes as C
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hyquant_b200", "csrc")
PROGRAM = r"""
#include "hq_topk_form.h"
extern "C" void form(int rows, int n, int k, int sms, long long* out) {
  const hq::TopkForm f = hq::topk_form(rows, n, k, sms);
  out[0] = f.blocks; out[1] = f.seg; out[2] = f.list; out[3] = f.kept; out[4] = (long long)f.smem;
}
"""
SMS, LIMIT = 148, 224 * 1024


@pytest.fixture(scope="module")
def form(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("topk")
    (d / "form.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "form.so"), str(d / "form.cpp")],
                   check=True)
    lib = C.CDLL(str(d / "form.so"))

    def call(rows, n, k, sms=SMS):
        out = (C.c_longlong * 5)()
        lib.form(rows, n, k, sms, out)
        return tuple(out)
    return call


# rows, n, k where the clusters were slower than a block a row (up to 2.6 times): many rows, or half the row selected
@pytest.mark.parametrize("rows,n,k", [(75, 12288, 614), (96, 16384, 819), (148, 32768, 1638), (148, 65536, 3276), (75, 32768, 8192),
                                      (74, 16384, 819), (74, 131072, 6553), (37, 32768, 8192), (36, 65536, 16384), (64, 65536, 16384),
                                      (64, 16384, 4096), (32, 8192, 409), (1, 12287, 614)])
def test_a_block_a_row_where_it_is_faster(form, rows, n, k):
    assert form(rows, n, k)[0] == 1


@pytest.mark.parametrize("rows,n,k,blocks", [(1, 12288, 614, 4), (8, 32768, 1638, 8), (32, 32768, 1638, 8), (32, 16384, 819, 4), (64, 32768, 1638, 4),
                                             (32, 131072, 6553, 4), (14, 131072, 6553, 8), (16, 131072, 6553, 4), (32, 65536, 16384, 4)])
def test_a_cluster_where_it_is_faster(form, rows, n, k, blocks):
    assert form(rows, n, k)[0] == blocks


def test_every_form_fits(form):
    sizes = sorted({x + d for x in (64, 2048, 8192, 12288, 16384, 20480, 32768, 53000, 57000, 100003, 262144, 440001, 1 << 20) for d in (-1, 0, 1, 31)})
    for rows in (1, 2, 13, 14, 15, 28, 29, 32, 33, 37, 38, 64, 65, 148, 149, 1000):
        for n in sizes:
            for k in {1, min(n, 64), min(n, 65), min(max(1, n // 20), 16384), min(n // 8, 16384), min(n // 8 + 1, 16384), min(n, 16384)}:
                for sms in (SMS, 132, 16):
                    blocks, seg, room, kept, smem = form(rows, n, k, sms)
                    assert blocks in (1, 4, 8) and (blocks == 1 or rows * blocks <= 2 * sms)
                    assert blocks * seg >= n and (blocks == 1 or (seg % 32 == 0 and (blocks - 1) * seg < n))
                    assert room & (room - 1) == 0 and room >= min(k, seg) and room >= 64
                    need = 8 * room + 8192 * (2 if blocks > 1 else 1)
                    assert smem == need + (4 * seg if kept else 0) <= LIMIT and kept == (need + 4 * seg <= LIMIT)
