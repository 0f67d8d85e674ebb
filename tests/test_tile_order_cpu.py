"""The tile order of the GEMMs divides by multiplying: FastDiv, compiled for the host from csrc/gemm.cu as it stands there,
against integer division.  The order itself is restated here: it shows that the formula takes every tile once, not that the
kernel follows it (the products of every other test do)."""
import ctypes
import os
import random
import re
import subprocess

import pytest

GEMM = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "triton_int8_b200", "csrc", "gemm.cu")


@pytest.fixture(scope="module")
def fast_div(tmp_path_factory):
    struct = re.search(r"^struct FastDiv \{.*?^\};", open(GEMM).read(), re.S | re.M).group(0)
    tmp = tmp_path_factory.mktemp("fastdiv")
    src, lib = tmp / "fastdiv.cpp", tmp / "fastdiv.so"
    src.write_text("#include <stdint.h>\n#define __device__\n#define __forceinline__ inline\n" + struct +
                   '\nextern "C" int fast_div(int n, int d) { FastDiv f; f.set(d); return f.div(n); }\n')
    subprocess.run([os.environ.get("CXX") or "g++", "-O1", "-fPIC", "-shared", "-o", str(lib), str(src)], check=True)
    fn = ctypes.CDLL(str(lib)).fast_div
    return lambda d: lambda n: fn(n, d)


def test_division(fast_div):
    rng = random.Random(1)
    for d in [*range(1, 300), *(rng.randrange(1, 1 << 31) for _ in range(300)), (1 << 31) - 1, 1 << 30, (1 << 30) + 1]:
        div = fast_div(d)
        ns = [0, d - 1, d, d + 1, (1 << 31) - 1, (1 << 31) // d * d - 1, *(rng.randrange(1 << 31) for _ in range(50))]
        assert all(div(n) == n // d for n in ns if 0 <= n < 1 << 31)


def test_every_tile_once(fast_div):
    for m_units in (1, 3, 16, 31, 32, 33, 80, 97):
        for n_tiles in (1, 2, 7, 43):
            for raster in (8, 16, 32):
                per_group, full = fast_div(raster * n_tiles), fast_div(raster)
                last_size = m_units % raster or raster
                last = fast_div(last_size)
                seen = set()
                for t in range(m_units * n_tiles):
                    g = per_group(t)
                    local, first = t - g * raster * n_tiles, g * raster
                    div, size = (full, raster) if first + raster <= m_units else (last, last_size)
                    n = div(local)
                    m = first + local - n * size
                    assert 0 <= m < m_units and 0 <= n < n_tiles
                    seen.add((m, n))
                assert len(seen) == m_units * n_tiles
