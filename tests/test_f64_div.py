"""The affine search's integer double division (uavs3e_gb300/csrc/f64div.cuh) against the host's IEEE
division: random bit patterns, integer-valued operands as the normal equations give, mantissas at the
ends of their range, nearly equal operands."""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "uavs3e_gb300", "csrc")
HARNESS = """
#include "f64div.cuh"
#include <string.h>
static uint64_t st;
static uint64_t rnd() { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return st; }
extern "C" long check(int kind, long n, uint64_t seed, long *done)
{
    const uint64_t M = 0xFFFFFFFFFFFFFull, E1 = 1023ull << 52;
    long bad = 0;
    st = seed;
    *done = 0;
    for (long i = 0; i < n; i++) {
        uint64_t a = rnd(), b = rnd(), r, w;
        if (kind == 1) {
            double x = (double)(int64_t)(a >> (rnd() & 40)), y = (double)(int64_t)(b >> (rnd() & 40));
            memcpy(&a, &x, 8);
            memcpy(&b, &y, 8);
        } else if (kind == 2) {
            a = E1 | (rnd() & 1 ? rnd() % 8 : M - rnd() % 8);
            b = E1 | (rnd() & 1 ? rnd() % 8 : M - rnd() % 8);
        } else if (kind == 3) {
            b = a ^ (rnd() & 15);
        } else if (kind == 4) {
            a = E1 | (a & M);
            b = E1 | (b & M);
        }
        if (!uc::f64_div_bits(a, b, &r)) continue;
        ++*done;
        double x, y, z;
        memcpy(&x, &a, 8);
        memcpy(&y, &b, 8);
        z = x / y;
        memcpy(&w, &z, 8);
        bad += w != r;
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("f64div")
    (d / "h.cpp").write_text(HARNESS)
    so = d / "h.so"
    subprocess.run([os.environ.get("CXX", "g++"), "-x", "c++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    "-o", str(so), str(d / "h.cpp")], check=True)
    f = C.CDLL(str(so)).check
    f.restype = C.c_long
    f.argtypes = [C.c_int, C.c_long, C.c_uint64, C.POINTER(C.c_long)]
    return f


@pytest.mark.parametrize("kind", range(5), ids=["bits", "integers", "ends", "near", "unit"])
def test_division_is_correctly_rounded(harness, kind):
    done = C.c_long()
    assert harness(kind, 2000000, 88172645463325252 + kind, C.byref(done)) == 0
    assert done.value > 500000
