"""Plan-time rules of the FP32 split (csrc/f32_split_rule.h), compiled for the
CPU as they stand."""
import ctypes
import os
import shutil
import subprocess

import pytest

from tccg_b200 import build

WRAP = """
#include "f32_split_rule.h"
extern "C" int fits(long long m, long long n, long long k) { return tccg::f32_split_fits(m, n, k); }
extern "C" int memory(long long m, long long n, long long k) { return tccg::f32_split_memory(m, n, k); }
extern "C" int chunk(long long chain, long long splits) { return tccg::f32_split_chunk(chain, splits); }
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("rule")
    src, out = os.path.join(d, "wrap.cpp"), os.path.join(d, "librule.so")
    with open(src, "w") as f:
        f.write(WRAP)
    subprocess.run([gxx, "-std=c++17", "-shared", "-fPIC", "-I" + build.CSRC, src, "-o", out], check=True)
    lib = ctypes.CDLL(out)
    lib.fits.argtypes = [ctypes.c_longlong] * 3
    lib.memory.argtypes = [ctypes.c_longlong] * 3
    lib.chunk.argtypes = [ctypes.c_longlong] * 2
    return lib


@pytest.mark.parametrize("k", [1, 32, 4096, 1 << 29, 700_000_000, 715_827_872, 715_827_873, 715_827_900,
                               800_000_000, (1 << 30) - 1])
def test_last_packed_column_is_a_tma_coordinate(rule, k):
    """The last k-block's lo part starts at column 96 (kb - 1) + 64 and ends at
    96 kb: inside signed 32 bits wherever the rule admits K, and the rule turns
    nothing down that would fit."""
    end = 96 * -(-k // 32)
    assert bool(rule.fits(8, 8, k)) == (end <= 2 ** 31 - 1)


def test_rows(rule):
    assert rule.fits((1 << 30) - 1, 8, 64) and not rule.fits(1 << 30, 8, 64) and not rule.fits(8, 1 << 30, 64)


def test_chunk_follows_the_chain(rule):
    """No split below a chain of 256 adds; a chunk's truncations (2 per k-block)
    at most a 48th of the chain's roundings plus 3 up to the longest chunk."""
    assert rule.chunk(255, 1) == 0 and rule.chunk(256, 1) == 1
    assert rule.chunk(128, 2) == 1 and rule.chunk(400, 28) == 1 and rule.chunk(2 * 768, 2) == 3
    chunks = [rule.chunk(c, 1) for c in range(0, 5000)]
    assert chunks == sorted(chunks) and max(chunks) == 4
    assert all(2 * k <= c / 48 + 3 for c, k in enumerate(chunks))


@pytest.mark.parametrize("m,n,k,fits", [(4096, 4096, 1024, 1), (32768, 32768, 65536, 1), (65536, 65536, 65536, 0),
                                        (100_000_000, 256, 256, 0), (8, 8, 500_000_000, 1)])
def test_footprint(rule, m, n, k, fits):
    assert rule.memory(m, n, k) == fits
    assert fits == (10 * (m + n) * -(-k // 32) * 32 + 4 * m * n <= 90e9)
