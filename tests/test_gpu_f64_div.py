"""The device branch of the affine search's integer double division (uavs3e_gb300/csrc/f64div.cuh) against
IEEE division: the operands of test_f64_div.py, in a kernel built for this test."""
import ctypes as C
import importlib
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "uavs3e_gb300", "csrc")
KERNEL = """
#include "f64div.cuh"
__global__ void k_div(const uint64_t *a, const uint64_t *b, uint64_t *r, unsigned char *done, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { uint64_t v = 0; done[i] = uc::f64_div_bits(a[i], b[i], &v); r[i] = v; }
}
extern "C" int run(const uint64_t *a, const uint64_t *b, uint64_t *r, unsigned char *done, int n)
{
    k_div<<<(n + 255) / 256, 256>>>(a, b, r, done, n);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def divide(gpu, tmp_path_factory):
    import torch
    build = importlib.import_module("uavs3e_gb300.build")
    d = tmp_path_factory.mktemp("f64div")
    (d / "k.cu").write_text(KERNEL)
    subprocess.run([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, "-o",
                                                  str(d / "k.so"), str(d / "k.cu")], check=True)
    f = C.CDLL(str(d / "k.so")).run
    f.argtypes = [C.c_void_p] * 4 + [C.c_int]

    def call(a, b):
        t = [torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b)]
        r, done = torch.zeros_like(t[0]), torch.zeros(len(a), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        assert f(t[0].data_ptr(), t[1].data_ptr(), r.data_ptr(), done.data_ptr(), len(a)) == 0
        return r.cpu().numpy().view(np.float64), done.cpu().numpy().astype(bool)
    return call


@pytest.mark.parametrize("kind", ["bits", "integers", "ends", "near", "unit"])
def test_device_division_is_correctly_rounded(divide, kind):
    n, one, mant = 1 << 20, np.uint64(1023 << 52), np.uint64((1 << 52) - 1)
    rng = np.random.default_rng(len(kind))
    a, b = (rng.integers(0, 1 << 64, n, dtype=np.uint64) for _ in range(2))
    if kind == "integers":
        a, b = ((x.view(np.int64) >> rng.integers(0, 41, n)).astype(np.float64).view(np.uint64) for x in (a, b))
    elif kind == "ends":
        a, b = (one | np.where(rng.random(n) < 0.5, x % np.uint64(8), mant - x % np.uint64(8)) for x in (a, b))
    elif kind == "near":
        b = a ^ (b & np.uint64(15))
    elif kind == "unit":
        a, b = (one | (x & mant) for x in (a, b))
    got, done = divide(a, b)
    with np.errstate(all="ignore"):
        want = a.view(np.float64) / b.view(np.float64)
    assert done.sum() > n // 4
    assert np.array_equal(got[done].view(np.uint64), want[done].view(np.uint64))
