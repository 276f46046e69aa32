"""Which kernel a plain GEMM runs on (gemm_choice.hpp, compiled for the host): shapes whose kernels were measured to be 8 % or more apart,
either side of each line."""
import ctypes
import subprocess

import pytest

from cute_mma_b200 import build

HARNESS = r"""
#include "gemm_choice.hpp"
extern "C" int small(int m, int n, int steps, int whole_k) { return b200::small_wins(m, n, steps, whole_k != 0, 148); }
extern "C" int wide(int m, int n, int steps, int nt, int whole_lines) { return b200::wide_wins(m, n, steps, nt != 0, whole_lines != 0, 148); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("choice")
    (d / "rules.cpp").write_text(HARNESS)
    subprocess.run([build.nvcc_path(), "-std=c++17", "-shared", "-Xcompiler", "-fPIC", f"-I{build.CSRC}", str(d / "rules.cpp"), "-o", str(d / "rules.so")], check=True)
    return ctypes.CDLL(str(d / "rules.so"))


# m, n, K steps, us on small_kernel / on pair tiles; narrow tiles of many steps, whose 128 rows cost as much as their columns,
# among others
@pytest.mark.parametrize("m,n,steps,small,pair", [(7016, 272, 40, 29.5, 21.0), (12601, 169, 40, 34.4, 23.3), (33475, 147, 46, 67.8, 47.9), (11929, 175, 90, 47.2, 35.2),
                                                  (15189, 145, 82, 57.1, 45.0), (32930, 143, 107, 150.3, 114.2), (58201, 230, 15, 63.4, 42.5), (5936, 776, 91, 118, 68),
                                                  (12242, 297, 6, 7.6, 13.3), (11904, 276, 9, 9.9, 15.7), (6176, 720, 6, 7.4, 11.5), (640, 1280, 32, 10, 29), (65536, 120, 64, 100, 128)])
def test_small_or_pair(rules, m, n, steps, small, pair):
    assert rules.small(m, n, steps, 0) == (small < pair)


# m, n, K steps, NT, rows on whole 128-byte lines, us on tiles of 256 x 256 / of 256 x 512
@pytest.mark.parametrize("m,n,steps,nt,lines,pair,wide", [(12544, 1792, 64, 0, 1, 126, 142), (12544, 768, 64, 0, 1, 55, 62), (49664, 768, 73, 1, 1, 247, 264),
                                                          (48000, 768, 12, 0, 1, 47, 52), (4096, 2048, 64, 0, 1, 77.0, 75.6), (1152, 6144, 86, 0, 1, 87, 92), (20480, 331, 106, 0, 1, 115, 105), (21888, 424, 98, 0, 1, 121, 111), (49664, 704, 73, 0, 1, 240, 266), (3583, 5376, 14, 0, 1, 39, 42),
                                                          (13171, 10088, 4, 0, 1, 98, 138), (8192, 8192, 128, 0, 1, 864, 831), (1600, 12608, 120, 0, 1, 327, 313),
                                                          (11008, 3001, 64, 0, 1, 252, 219), (4096, 4096, 256, 1, 1, 471, 436), (4096, 4096, 128, 1, 1, 221, 209),
                                                          (49664, 1024, 73, 1, 1, 343, 337), (5952, 6336, 17, 0, 0, 102, 83), (15713, 1302, 12, 0, 0, 55, 47),
                                                          (4690, 9804, 151, 1, 0, 906, 782)])
def test_256_or_512_columns(rules, m, n, steps, nt, lines, pair, wide):
    assert rules.wide(m, n, steps, nt, lines) == (wide < pair)


def test_512_columns_need_a_second_round_and_a_second_half(rules):
    for nt in (0, 1):
        for lines in (0, 1):
            assert rules.wide(1000, 2000, 400, nt, lines) == 0 and rules.wide(100000, 256, 400, nt, lines) == 0


def test_sizes_that_round_up_beyond_an_int(rules):
    top = 2**31 - 1
    assert rules.small(top, 100, 4, 0) == 1 and rules.small(top, 1000, 4, 0) == 0
    assert rules.wide(top, 512, 64, 1, 1) == 1 and rules.wide(top, top, 64, 0, 0) == 1
