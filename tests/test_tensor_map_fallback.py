"""The selecting contraction is only chosen where its operands' tensor maps can be encoded
(host code of the library, no GPU): elsewhere nearest_center and knn keep the forms that
need none.
"""
import ctypes
import os
import subprocess

import pytest
import torch

from puck_gb300 import build, native

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cuda.h>
#include "pgpu_internal.h"
namespace pgpu {
bool encode_bf16_rows(CUtensorMap* map, const uint16_t* p, uint64_t rows, uint64_t rs, uint32_t K,
                      uint32_t box_rows);
}
extern "C" int applies(uint32_t d) { return pgpu::tc_filter_applies(d); }
extern "C" int encodes(uint32_t d, uint64_t rows, uint32_t box) {
    CUtensorMap map;
    return pgpu::encode_bf16_rows(&map, reinterpret_cast<const uint16_t*>(1 << 20), rows, (d + 7u) & ~7u, d,
                                  box);
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("host")
    src, so = d / "host.cpp", d / "host.so"
    src.write_text(SOURCE)
    lib = build.build()
    native.load()
    if torch.cuda.is_available():
        torch.empty(1, device="cuda")  # the driver encodes once it is initialised
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", str(src), "-o", str(so), lib,
                    "-I" + os.path.join(REPO, "puck_gb300", "csrc"),
                    "-I" + os.path.join(build._cuda_home(), "include"), "-Wl,-rpath," + os.path.dirname(lib)],
                   check=True)
    return ctypes.CDLL(str(so))


def test_applies_only_where_maps_encode(host):
    host.encodes.argtypes = [ctypes.c_uint32, ctypes.c_uint64, ctypes.c_uint32]
    for d in (1, 4, 7, 8, 30, 96, 128, 255, 256):
        for rows, box in ((1, 128), (1, 256), (129, 128), (2 ** 24 - 1, 256)):
            assert bool(host.applies(d)) == bool(host.encodes(d, rows, box)), (d, rows)
    assert not host.applies(257)
