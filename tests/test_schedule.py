"""Which build of the chain kernel a batch of small lattices runs on
(csrc/z2_schedule.h, compiled for the host), on 148 SMs: never the slower one
by more than a few percent in the batches timed on the GPU (ms per bin with the
256-thread kernel and with 1 to 4 blocks of the 128-thread kernel per SM)."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "z2_gauge_zfy_b200", "csrc")
SRC = """
#include "z2_schedule.h"
extern "C" int blocks(int n, const int *N, const int *L, int nsm, int occ) {
  std::vector<Z2ChainLoad> c;
  for (int i = 0; i < n; ++i) c.push_back({N[i], z2_chain_cost(N[i], L[i], true)});
  return z2_small_blocks_per_sm(c, nsm, occ);
}
"""
# (sites, slices) x chains, blocks that fit, times (256 threads, 1 ... 4 blocks)
TIMED = [
    ([(16, 40, 149)], 4, (2.52, 2.48, 1.46, 1.45, 1.45)),
    ([(16, 40, 300)], 4, (3.93, 3.84, 2.77, 2.24, 2.26)),
    ([(16, 40, 1000)], 4, (9.91, 9.66, 7.57, 7.07, 6.39)),
    ([(36, 40, 160)], 4, (4.65, 5.12, 3.10, 3.07, 3.09)),
    ([(36, 40, 450)], 4, (9.28, 10.33, 6.59, 6.41, 5.85)),
    ([(64, 40, 149)], 3, (6.90, 8.28, 5.04, 5.07)),
    ([(64, 40, 300)], 3, (10.63, 12.80, 9.91, 6.41)),
    ([(64, 40, 1000)], 3, (26.05, 30.95, 21.27, 20.74)),
    ([(16, 40, 128), (16, 80, 128), (36, 40, 128), (36, 80, 128)], 4, (10.51, 10.95, 8.21, 9.44, 10.70)),
    # two blocks fit (delay rank 32), one (64)
    ([(64, 40, 300)], 2, (11.45, 13.58, 10.20)),
    ([(64, 40, 160)], 1, (7.83, 8.90)),
    ([(64, 40, 300)], 1, (11.61, 13.34)),
    ([(64, 40, 600)], 1, (19.37, 22.04)),
    # few long chains
    ([(16, 40, 200), (64, 320, 1)], 3, (25.41, 30.90, 30.87, 30.88)),
    ([(16, 40, 500), (64, 160, 4)], 3, (14.28, 17.11, 18.40, 17.97)),
    ([(16, 80, 128), (64, 80, 128)], 3, (9.98, 11.23, 11.04, 10.95)),
]


@pytest.fixture(scope="module")
def blocks(tmp_path_factory):
    d = tmp_path_factory.mktemp("schedule")
    (d / "s.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-std=c++17", "-I", CSRC, "-o", str(d / "s.so"),
                    str(d / "s.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "s.so"))

    def call(batch, occ, nsm=148):
        N = [n for n, _, k in batch for _ in range(k)]
        L = [t for _, t, k in batch for _ in range(k)]
        arr = ctypes.c_int * len(N)
        return lib.blocks(len(N), arr(*N), arr(*L), nsm, occ)

    return call


@pytest.mark.parametrize("batch,occ,ms", TIMED)
def test_picks_no_slower_kernel(blocks, batch, occ, ms):
    b = blocks(batch, occ)
    assert 0 <= b <= occ
    assert ms[b] <= 1.05 * ms[0]          # never behind one 256-thread block per SM
    if min(ms[1:]) < 0.9 * ms[0]:         # and not left there where the other build gains
        assert b > 0


def test_without_room_the_256_thread_kernel_runs(blocks):
    assert blocks([(64, 40, 300)], 0) == 0
