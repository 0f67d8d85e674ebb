"""CPU-only checks of the boundary: the shared library loads, exports every symbol the header
declares, and argument validation fails with the documented codes before any device work."""
import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    from triton_int8_b200 import build, _lib
    build.build()
    return _lib.load()


def test_every_declared_symbol_is_exported(lib):
    hdr = open(os.path.join(ROOT, "include", "i8linear.h")).read()
    declared = set(re.findall(r"I8L_API\s+[\w\s\*]+?\b(i8l_\w+)\s*\(", hdr))
    assert len(declared) >= 8
    for name in declared:
        assert hasattr(lib, name), name
    from triton_int8_b200 import _lib
    assert declared == set(_lib.SIGNATURES) | {"i8l_last_error"}


def test_argument_validation_without_a_gpu(lib):
    buf = ctypes.create_string_buffer(1 << 16)
    p = ctypes.addressof(buf)
    p += (16 - p % 16) % 16
    rc = lib.i8l_quant_tile(p, 1, 100, 128, 0, 0, 0, p, p, None, None, None)
    assert rc == -1 and b"multiples of 128" in lib.i8l_last_error()
    rc = lib.i8l_quant_tile(p + 1, 1, 128, 128, 0, 0, 0, p, p, None, None, None)
    assert rc == -2
    rc = lib.i8l_quant_tile(p, 1, 128, 128, 0, 0, 64, p, p, None, None, None)
    assert rc == -6
    rc = lib.i8l_gemm_block(p, p, p, p, 0, 0, 0, None, 1.0, p, 1, 128, 128, 100, 0, None, None)
    assert rc == -1
    rc = lib.i8l_gemm_block(p, p, None, p, 0, 0, 0, None, 1.0, p, 1, 128, 128, 128, 0, None, None)
    assert rc == -6
    rc = lib.i8l_quant_row(p, 128, 3000, 0, -1, p, p, None)
    assert rc == -1


@pytest.mark.skipif(torch.cuda.is_available(), reason="checks the no-GPU behaviour")
def test_no_cpu_fallback(lib):
    from triton_int8_b200 import I8LError, block_channel
    with pytest.raises(ValueError):
        block_channel.triton_per_block_quant(torch.zeros(1, 128, 128, dtype=torch.bfloat16))
    buf = ctypes.create_string_buffer(1 << 16)
    p = ctypes.addressof(buf); p += (16 - p % 16) % 16
    rc = lib.i8l_quant_tile(p, 1, 128, 128, 0, 0, 0, p, p, None, None, None)
    assert rc in (-3, -4)   # no device / wrong architecture: an error, never a CPU result


def test_product_calls_validate_before_any_launch(lib):
    """i8l_quant_gemm and i8l_linear_backward check extents, the combination of groupings and the workspace first."""
    buf = ctypes.create_string_buffer(1 << 16)
    p = ctypes.addressof(buf); p += (256 - p % 256) % 256

    def product(M=128, a_gran=0, b_gran=2, ws_bytes=1 << 15, a_qt=None, batch=1):
        return lib.i8l_quant_gemm(p, p, None, p, a_qt, a_qt, batch, M, 128, 128, 0, a_gran, b_gran, 0, 0, 1.0, 0, p, ws_bytes,
                                  None, None)
    assert product(M=100) == -1 and product(M=0) == -1
    assert product(a_gran=2, b_gran=0) == -6 and product(b_gran=5) == -6 and product(a_qt=p, batch=2) == -6
    assert product(ws_bytes=1 << 15) == -6 and b"too small" in lib.i8l_last_error()

    def backward(gran=0, ws_bytes=1 << 15, x_qt=p):
        return lib.i8l_linear_backward(p, p, x_qt, p, p, p, 128, 128, 128, gran, 0, 0, 1.0, 1.0, 0, p, ws_bytes, None, None)
    assert backward() == -6 and b"too small" in lib.i8l_last_error()
    assert backward(gran=5, ws_bytes=1 << 20) == -6 and backward(x_qt=None, ws_bytes=1 << 20) == -6


@pytest.mark.parametrize("off", [1, 4, 8])
def test_product_calls_refuse_a_workspace_off_its_alignment(lib, off):
    """... before any launch, whichever kernels would write to it: small operands share a launch, long columns have their
    maxima cleared first, the bias gradient comes first.  No device here: what passes the checks ends in another error."""
    buf = ctypes.create_string_buffer(1 << 12)
    p = ctypes.addressof(buf); p += (256 - p % 256) % 256
    for gran, b_gran, qmode in ((0, 2, 0), (1, 2, 1), (2, 2, 3), (0, 0, 0), (5, 2, 0)):
        for M in (128, 65536):
            for a_qt in (None, p) if b_gran == 2 and gran != 5 else (None,):
                assert lib.i8l_quant_gemm(p, p, None, p, a_qt, a_qt, 1, M, 256, 256, 0, gran, b_gran, qmode, 0, 1.0, 0, p + off,
                                          1 << 40, None, None) == -2
    for gran, qmode in ((0, 0), (1, 1), (2, 3)):
        for N in (128, 8192):
            for dx, dw, db in ((p, p, p), (p, None, None), (None, p, None), (p, p, None)):
                assert lib.i8l_linear_backward_bias(p, p, p, p, dx, dw, db, 128, N, 128, gran, qmode, 0, 1.0, 1.0, 0, p + off,
                                                    1 << 40, None, None) == -2


@pytest.mark.parametrize("batch,M,N", [(65535, 128, 128), (70000, 128, 128), (131071, 128, 256), ((1 << 24) - 1, 128, 128)])
def test_product_call_takes_the_batches_of_its_steps(lib, batch, M, N):
    """Per-row scales have no limit on the batch of their own: the quantizer and the GEMM take batch * M below 2^31.  The
    128x128-tile quantizer takes 65535.  No device here: what passes the checks ends in an architecture or CUDA error."""
    buf = ctypes.create_string_buffer(1 << 12)
    p = ctypes.addressof(buf); p += (256 - p % 256) % 256

    def product(gran, b_batched=0, batch=batch, M=M, N=N, K=128):
        return lib.i8l_quant_gemm(p, p, None, p, None, None, batch, M, N, K, b_batched, gran, 2, 3 if gran == 2 else 0, 0, 1.0, 0,
                                  p, 1 << 50, None, None)
    fits = batch * max(M, N) < 1 << 31
    for b_batched in (0, 1):
        assert product(2, b_batched) in ((-3, -4) if fits else (-1,)), lib.i8l_last_error()
    assert product(0) in ((-3, -4) if batch <= 65535 else (-1,))
    # extents whose products would not fit 64 bits are refused before they are multiplied
    assert product(2, batch=1 << 30, M=1 << 30, K=1 << 30) == -1 and product(2, batch=1 << 62) == -1


def test_wrappers_check_what_their_pointers_describe():
    """A bias is read as N consecutive bf16 values and saved scales in the layout of the grouping: what is shorter, of another
    type or of another grouping is refused, a strided bias is made contiguous."""
    from triton_int8_b200 import _lib as L, kernels as K
    b = torch.arange(256, dtype=torch.float32)
    assert K._check_bias(None, 128) is None
    with pytest.raises(TypeError):
        K._check_bias(b, 256)
    with pytest.raises(ValueError):
        K._check_bias(b.to(torch.bfloat16)[:100], 128)
    strided = b.to(torch.bfloat16)[::2]
    got = K._check_bias(strided, 128)
    assert got.is_contiguous() and torch.equal(got, strided)

    M, Kd = 256, 384
    q = torch.zeros(1, Kd, M, dtype=torch.int8)
    scales = {L.GRAN_TILE128: torch.zeros(1, Kd // 128, M // 128), L.GRAN_GROUP128: torch.zeros(1, Kd, M // 128),
              L.GRAN_ROW: torch.zeros(1, Kd)}
    for gran in scales:
        for made_with, st in scales.items():
            if made_with == gran:
                assert K._check_saved(q, st, M, Kd, gran)[1] is st
            else:
                with pytest.raises(ValueError):
                    K._check_saved(q, st, M, Kd, gran)
        with pytest.raises(ValueError):
            K._check_saved(q, scales[gran].double(), M, Kd, gran)
        with pytest.raises(ValueError):
            K._check_saved(q[:, :, :128], scales[gran], M, Kd, gran)
