"""Shared memory of the split scan, over the whole range of shapes an index can have (host
code of the library, no GPU): whatever layout is chosen, every part of the block stays within
it, the sampled keys and their histogram included.
"""
import ctypes
import os
import subprocess

import pytest

from puck_gb300 import build, native

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "pgpu_internal.h"
using namespace pgpu;
extern "C" void split_of(uint32_t nsq, uint32_t d, uint32_t F, uint32_t P, uint32_t T, uint32_t* out) {
    DeviceIndex ix;
    ix.nsq = nsq;
    ix.d = d;
    ix.lsq = d / nsq;
    ix.F = F;
    ix.C = 8192;
    const SplitLayout y = split_choice(ix, P, T);
    out[0] = y.keys;
    out[1] = y.cap;
    out[2] = y.bytes;
}
// The most keys' room that a query takes while its bound is sampled, over record counts N > cap.
extern "C" uint32_t sampled_keys(uint32_t cap, uint32_t T) {
    uint32_t most = 0;
    for (uint64_t N = cap + 1ull; N < (1ull << 32); N += N / 3 + 1) {
        const uint32_t S = sample_count(cap, T, (uint32_t)N);
        if (S + kSplitHistKeys > most) most = S + kSplitHistKeys;
    }
    return most;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("host")
    src, so = d / "host.cpp", d / "host.so"
    src.write_text(SOURCE)
    lib = build.build()
    native.load()
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", str(src), "-o", str(so), lib,
                    "-I" + os.path.join(REPO, "puck_gb300", "csrc"),
                    "-I" + os.path.join(build._cuda_home(), "include"), "-Wl,-rpath," + os.path.dirname(lib)],
                   check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("nsq", [4, 8, 12, 16, 20, 24, 28, 32])
def test_split_layout_holds_the_sampled_keys(host, nsq):
    out = (ctypes.c_uint32 * 3)()
    fine = sorted(set([1, 3, 20, 500, 1023, 1024, 1025, 2048, 4095, 4096, 4097, 5000, 8191, 8192] +
                      list(range(5000, 8192, 97))))
    need, chosen = {}, 0
    for lsq in (1, 4, 16, 64):
        d = nsq * lsq
        if d > 1024:
            continue
        for F in fine:
            for P in (1, 8, 128, 300, 512, 8192):
                for T in (1, 10, 100, 200, 340, 500, 1100, 2048):
                    host.split_of(nsq, d, F, P, T, out)
                    keys, cap, size = out
                    if size == 0:
                        continue
                    chosen += 1
                    at = (nsq, d, F, P, T, cap)
                    assert size <= 220 * 1024 and keys + 8 * cap <= size, at
                    assert cap > T, at
                    if (cap, T) not in need:
                        need[cap, T] = host.sampled_keys(cap, T)
                    assert need[cap, T] <= cap, at
    assert chosen > 0
