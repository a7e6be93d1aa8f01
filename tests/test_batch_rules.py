"""The batch's rules on sizes and memory (infoli_lane.h), compiled for the host: two lanes per receiver only in clusters
that the device runs, entry lists only where they and the bitmasks they are packed from fit."""
import ctypes
import subprocess

import pytest

from infoli_gb300 import build as B

SOURCE = r"""
#include "infoli_lane.h"
extern "C" int lanes(int n, double edges, double all, int block, int sms, const unsigned char* r) {
  bool runs[infoli::kListMaxCtas + 1];
  for (int i = 0; i <= infoli::kListMaxCtas; ++i) runs[i] = r[i] != 0;
  return infoli::list_lanes(n, edges, all, block, sms, runs);
}
extern "C" int fit(long long rows, long long words, double mem) { return infoli::lists_fit(rows, words, mem); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    where = tmp_path_factory.mktemp("rules")
    (where / "rules.cpp").write_text(SOURCE)
    cuda = B._nvcc().rsplit("/bin/", 1)[0] + "/include"
    subprocess.run(["g++", "-std=c++17", "-I", B.SRC, "-I", B.INC, "-I", cuda, "-shared", "-fPIC", "-o",
                    str(where / "rules.so"), str(where / "rules.cpp")], check=True)
    lib = ctypes.CDLL(str(where / "rules.so"))
    lib.lanes.argtypes = [ctypes.c_int, ctypes.c_double, ctypes.c_double, ctypes.c_int, ctypes.c_int, ctypes.c_char_p]
    lib.fit.argtypes = [ctypes.c_longlong, ctypes.c_longlong, ctypes.c_double]
    return lib


@pytest.mark.parametrize("block", [512, 1024])
@pytest.mark.parametrize("largest", [0, 1, 8, 16])  # the largest cluster that runs
def test_two_lanes_only_in_clusters_that_run(rules, block, largest):
    runs = bytes([0] + [int(k <= largest) for k in range(1, 17)])
    for n in (1, block // 2, block // 2 + 1, block, 4 * block, 4 * block + 1, 8192 if block == 1024 else 4096, 8192):
        for share in (0.01, 0.9):  # a small part of the batch's edges, and nearly all
            got = rules.lanes(n, share * 1e8, 1e8, block, 152, runs)
            one, two = -(-n // block), -(-2 * n // block)
            assert got in (1, 2)
            if got == 2:
                assert two <= min(largest, 16)
            elif two <= min(largest, 16):
                assert two > one and share / one <= 0.75 / 152


def test_lists_and_their_bitmasks_fit(rules):
    gib = 2.0 ** 30
    assert rules.fit(0, 0, gib) and rules.fit(1 << 20, 0, gib)  # half of the memory
    assert not rules.fit((1 << 20) + 1, 0, gib)
    assert rules.fit(1 << 18, 1 << 27, gib)                      # 1/8 and 1/2
    assert not rules.fit(1 << 10, 1 << 28, gib)                  # the bitmasks alone are all of it
    assert not rules.fit(2 ** 31, 0, 1e13)                       # pair rows are counted in 32 bits
