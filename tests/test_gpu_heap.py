"""The warp's replay of Puck's bounded heap against the one-thread heap, step for step: values
in any order, equal ones, infinities and values that are not numbers.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from puck_gb300 import build

pytestmark = pytest.mark.gpu
REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "pgpu_internal.h"
#include "device_common.cuh"
using namespace pgpu;
__global__ void k_replay(const float* v, uint32_t n, uint32_t K, int warp, float* ov, uint32_t* ot,
                         uint32_t* filled) {
    extern __shared__ __align__(16) unsigned char smem[];
    if (warp) {
        uint2* heap = reinterpret_cast<uint2*>(smem);  // [K + 2]
        const uint32_t f = warp_heap_replay(heap, v, nullptr, n, K);
        for (uint32_t i = threadIdx.x; i < K; i += 32) {
            ov[i] = __uint_as_float(heap[i + 1].x);
            ot[i] = heap[i + 1].y;
        }
        if (threadIdx.x == 0) *filled = f;
    } else if (threadIdx.x == 0) {
        float* hv = reinterpret_cast<float*>(smem);  // [K + 1]
        uint32_t* ht = reinterpret_cast<uint32_t*>(hv + K + 1);
        for (uint32_t i = 0; i <= K; ++i) {
            hv[i] = sentinel_f();
            ht[i] = 0;
        }
        uint32_t dpc = K;
        for (uint32_t i = 0; i < n; ++i) heap_update(hv, ht, K, dpc, v[i], i);
        heap_reorder(hv, ht, K);
        for (uint32_t i = 0; i < K; ++i) {
            ov[i] = hv[i + 1];
            ot[i] = ht[i + 1];
        }
        *filled = K - dpc;
    }
}
extern "C" int replay(const float* v, uint32_t n, uint32_t K, int warp, float* ov, uint32_t* ot,
                      uint32_t* filled) {
    k_replay<<<1, 32, 8 * (K + 2)>>>(v, n, K, warp, ov, ot, filled);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    d = tmp_path_factory.mktemp("heap")
    src, so = d / "heap.cu", d / "heap.so"
    src.write_text(SOURCE)
    subprocess.run([os.path.join(build._cuda_home(), "bin", "nvcc"), *build.ARCH, "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", "-I" + os.path.join(REPO, "puck_gb300", "csrc"), str(src), "-o",
                    str(so)], check=True)
    so = ctypes.CDLL(str(so))
    so.replay.argtypes = [ctypes.c_void_p, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_int] + [ctypes.c_void_p] * 3
    return so


@pytest.mark.parametrize("special", ["none", "nan", "inf", "both"])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 31, 32, 33, 64, 100, 1100])
def test_warp_replay_is_the_heap(lib, K, special):
    import torch
    rng = np.random.default_rng(K)
    for n in (1, K - 1, K, K + 1, 3 * K + 7, 2000):
        if n < 1:
            continue
        v = rng.integers(-40, 40, n).astype(np.float32) / 8  # many equal ones
        at = rng.random(n) < 0.05
        if special in ("nan", "both"):
            v[at] = np.nan
        if special in ("inf", "both"):
            v[rng.random(n) < 0.05] = np.inf
            v[rng.random(n) < 0.01] = -np.inf
        dv = torch.from_numpy(v).cuda()
        got = []
        for warp in (0, 1):
            ov = torch.empty(K, device="cuda")
            ot = torch.empty(K, dtype=torch.int32, device="cuda")
            f = torch.zeros(1, dtype=torch.int32, device="cuda")
            assert lib.replay(dv.data_ptr(), n, K, warp, ov.data_ptr(), ot.data_ptr(), f.data_ptr()) == 0
            got.append((ov.cpu().numpy().view(np.uint32), ot.cpu().numpy(), f.item()))
        assert got[0][2] == got[1][2], n
        assert np.array_equal(got[0][0], got[1][0]), n
        used = got[0][0] != 0x7F7F7F7F  # the tag of a slot not filled is not defined
        assert np.array_equal(got[0][1][used], got[1][1][used]), n
