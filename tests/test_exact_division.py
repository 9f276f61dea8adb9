"""div_by (gr_internal.h), the raster's branch-free division by a known
reciprocal, equals the correctly rounded quotient bit for bit over the range
that narrow_fast admits: edge values over their sum (whole numbers of up to 31
bits), and barycentrics over W's of magnitudes in [2^-60, 2^61).  The header's
own function is compiled for the host; its operations are the same there."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstring>
#include "gr_internal.h"
typedef unsigned long long u64;
static u64 st;
static u64 rnd() { u64 z = (st += 0x9E3779B97F4A7C15ull); z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull; return z ^ (z >> 31); }
static unsigned bits(float f) { unsigned u; memcpy(&u, &f, 4); return u; }
static float from(unsigned u) { float f; memcpy(&f, &u, 4); return f; }
static unsigned sig() {  // significands: random, and near the ends where roundings are hardest
  switch (rnd() & 3) { case 0: return 0x7FFFFF - (rnd() & 3); case 1: return rnd() & 3; default: return rnd() & 0x7FFFFF; } }
static long bad(float a, float b) { return bits(gr::div_by(a, b, 1.0f / b)) != bits(a / b); }
extern "C" long check(long n, u64 seed) {
  st = seed;
  long wrong = 0;
  for (long i = 0; i < n; ++i) {
    const int s = (int)(rnd() % 31);
    const long sum = 1 + (long)(rnd() & ((2ull << s) - 1));
    const long e12 = 1 + (long)(rnd() % sum), e20 = 1 + (long)(rnd() % sum);
    const float sf = (float)-sum, a = (float)-e12, b = (float)-e20;
    wrong += bad(a, sf) + bad(b, sf);
    const float al = a / sf, be = b / sf, ga = (1.0f - al) - be;
    const float w = from(((67 + (unsigned)(rnd() % 121)) << 23) | sig() | ((unsigned)(rnd() & 1) << 31));
    wrong += bad(al, w) + bad(be, w) + bad(ga, w);
    wrong += bad(from((127u - 31u + (unsigned)(rnd() % 32)) << 23 | sig()), w);
  }
  wrong += bad(0.0f, -3.0f) + bad(0.0f, 3.0f) + bad(1.0f, -1.0f);
  return wrong;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("division")
    (d / "t.cpp").write_text(SRC)
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-D__host__=", "-D__device__=",
                           "-I" + os.path.join(ROOT, "gorender_gb300", "csrc"), "-I" + cuda, "-o", str(d / "t.so"), str(d / "t.cpp")])
    f = C.CDLL(str(d / "t.so")).check
    f.argtypes, f.restype = [C.c_long, C.c_uint64], C.c_long
    return f


@pytest.mark.parametrize("seed", [1, 2])
def test_div_by_is_the_rounded_quotient(check, seed):
    assert check(1_000_000, seed) == 0
