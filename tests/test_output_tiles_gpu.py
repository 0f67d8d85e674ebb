"""bf16 outputs of every GEMM kind leave through shared memory and TMA stores, fp32 outputs straight from registers: for
the same operands the bf16 result is the fp32 result rounded once (twice with a bias in the row x column kind), bit for bit, at
tiles that the output ends in, and nothing around the output is written."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from triton_int8_b200 import _lib as L
    from triton_int8_b200 import kernels as K

DEV = "cuda"
GUARD = 1024   # bf16 elements kept around the output
# kind: a_scale_kind, b_scale_kind, flags (None: row x column)
KINDS = {"rowcol": None, "fast": (0, 0, 0), "fast_tile": (0, 1, 0), "row_channel": (1, 0, 0), "row_tile": (1, 1, 0),
         "column": (0, 2, 2), "outer": (1, 2, 0), "tile_divisors": (0, 1, 2), "exact": (0, 0, 1)}


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("B,M,N,Kd,bias", [
    (1, 128, 128, 128, False),      # one tile, its second half outside the output
    (1, 256, 384, 256, True),       # CTA pair; the last tile is half outside
    (3, 384, 640, 384, True),       # batches, an odd number of row blocks
    (1, 4992, 1664, 640, False),    # 39 x 7 tiles: a second and a third tile per CTA
    (1, 10240, 1152, 256, False),   # 40 x 5 pair tiles, 80 x 5 single ones
    (1, 12544, 384, 384, True),     # narrow tiles, 98 x 3: a second one on most CTAs
])
def test_bf16_output_is_the_fp32_output_rounded(kind, B, M, N, Kd, bias):
    g = torch.Generator().manual_seed(M + N)
    a = torch.randint(-127, 128, (B, M, Kd), generator=g, dtype=torch.int8).to(DEV)
    b = torch.randint(-127, 128, (N, Kd), generator=g, dtype=torch.int8).to(DEV)
    a_s = (torch.rand(B * M * (Kd // 128), generator=g) * 0.1 + 0.01).to(DEV)
    b_s = (torch.rand(N * (Kd // 128), generator=g) * 0.1 + 0.01).to(DEV)
    bv = (torch.randn(N, generator=g) * 30).to(torch.bfloat16).to(DEV) if bias else None
    status = torch.zeros(1, dtype=torch.int32, device=DEV)

    def call(out, flags, bv=bv):
        stream = torch.cuda.current_stream().cuda_stream
        if KINDS[kind] is None:
            L.call("i8l_gemm_rowcol", a.data_ptr(), b.data_ptr(), a_s.data_ptr(), b_s.data_ptr(), 0,
                   None if bv is None else bv.data_ptr(), 1.0, out, B, M, N, Kd, flags, status.data_ptr(), stream)
        else:
            ak, bk, fl = KINDS[kind]
            L.call("i8l_gemm_block", a.data_ptr(), b.data_ptr(), a_s.data_ptr(), b_s.data_ptr(), ak, bk, 0,
                   None if bv is None else bv.data_ptr(), 0.25, out, B, M, N, Kd, fl | flags, status.data_ptr(), stream)

    f32 = torch.empty(B * M, N, device=DEV)
    call(f32.data_ptr(), L.GEMM_OUT_F32)
    want = f32.to(torch.bfloat16)
    if kind == "rowcol" and bias:   # bf16 outputs are rounded ahead of the bias too, as the reference stores them there
        plain = torch.empty_like(f32)
        call(plain.data_ptr(), L.GEMM_OUT_F32, None)
        assert torch.equal(f32, plain + bv.float())
        want = (plain.to(torch.bfloat16).float() + bv.float()).to(torch.bfloat16)
    for shift in (0, 8):   # 32-byte aligned, 16-byte aligned
        buf = torch.full((2 * GUARD + B * M * N,), 7.0, dtype=torch.bfloat16, device=DEV)
        call(buf[GUARD + shift:].data_ptr(), 0)
        torch.cuda.synchronize()
        got = buf[GUARD + shift:GUARD + shift + B * M * N].view(B * M, N)
        assert torch.equal(got, want)
        assert (buf[:GUARD + shift] == 7).all() and (buf[GUARD + shift + B * M * N:] == 7).all()
    assert status.item() == 0


def _takes_narrow_tiles(kind, m_blocks, N, ctas):
    """The rule of narrow_tiles in csrc/gemm.cu."""
    percent = {"rowcol": 80, "outer": 67}.get(kind, 62)
    waves = lambda tiles: -(-tiles // ctas)
    return waves(m_blocks * (N // 128)) * percent < waves(m_blocks * -(-N // 256)) * 100


@pytest.mark.parametrize("kind", [k for k in KINDS if k not in ("rowcol", "exact")] + ["rowcol"])
@pytest.mark.parametrize("B,M,N,Kd", [(1, 128, 256, 128), (2, 128, 640, 1152), (1, 256, 256, 24960)])   # 195 K blocks: a second chunk of factors
def test_narrow_tiles_equal_wide_ones(kind, B, M, N, Kd):
    """Few tiles are 128 columns wide; on a single CTA (cta_limit) the same product takes wide ones, the last of them half
    empty at N = 640.  Same bits."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _takes_narrow_tiles(kind, B * M // 128, N, sms) and not _takes_narrow_tiles(kind, B * M // 128, N, 1)
    g = torch.Generator().manual_seed(N + Kd)
    a = torch.randint(-127, 128, (B, M, Kd), generator=g, dtype=torch.int8).to(DEV)
    b = torch.randint(-127, 128, (N, Kd), generator=g, dtype=torch.int8).to(DEV)
    kb = Kd // 128
    if kind == "rowcol":
        a_s, b_s = torch.rand(B, M, generator=g).to(DEV), torch.rand(N, generator=g).to(DEV)
        call = lambda: K.gemm_rowcol(a, b, a_s, b_s)
    else:
        ak, bk, fl = KINDS[kind]
        a_s = (torch.rand(B, M // 128 if ak == 0 else M, kb, generator=g) * 0.1 + 0.01).to(DEV)
        b_s = (torch.rand({0: (N,), 1: (N // 128, kb), 2: (N, kb)}[bk], generator=g) * 0.1 + 0.01).to(DEV)
        call = lambda: K.gemm_block(a, b, a_s, b_s, ak, bk, None, 0.25, fl)
    narrow = call()
    with K.cta_limit(1):
        wide = call()
    torch.cuda.synchronize()
    assert torch.equal(narrow, wide)
    K.check_status(DEV)


@pytest.mark.parametrize("b_kind", ["tile", "group"])
@pytest.mark.parametrize("B,M,N,Kd", [(1, 128, 128, 128), (2, 256, 640, 384), (1, 4992, 1664, 256)])   # grids of any other kind's narrow tiles, then of wide ones
def test_divisors_per_row_of_a_take_wide_tiles_at_any_size(b_kind, B, M, N, Kd):
    """Divisors with a scale per row and K block of A have no kernel of their own: the generic kind takes them, which has
    wide tiles only.  Each K block costs three fp32 roundings (product of the scales, division, sum), the end one more."""
    g = torch.Generator().manual_seed(M + N + Kd)
    kb = Kd // 128
    a = torch.randint(-127, 128, (B, M, Kd), generator=g, dtype=torch.int8)
    b = torch.randint(-127, 128, (N, Kd), generator=g, dtype=torch.int8)
    a_s = torch.rand(B, M, kb, generator=g) + 0.5
    b_s = torch.rand(*{"tile": (N // 128, kb), "group": (N, kb)}[b_kind], generator=g) + 0.5
    fb = (b_s.repeat_interleave(128, 0) if b_kind == "tile" else b_s).double().to(DEV)
    ref, mag = torch.zeros(B, M, N, dtype=torch.double, device=DEV), torch.zeros(B, M, N, dtype=torch.double, device=DEV)
    for k in range(kb):
        cut = slice(k * 128, (k + 1) * 128)
        term = a[:, :, cut].to(DEV).double() @ b[:, cut].to(DEV).double().t() / (a_s[:, :, k, None].to(DEV).double() * fb[:, k])
        ref += term
        mag += term.abs()
    out = K.gemm_block(a.to(DEV), b.to(DEV), a_s.to(DEV), b_s.to(DEV), L.ASCALE_GROUP,
                       {"tile": L.BSCALE_TILE, "group": L.BSCALE_GROUP}[b_kind], flags=L.GEMM_DIVIDE | L.GEMM_OUT_F32)
    K.check_status(DEV)
    assert ((out.double() - ref).abs() <= (3 * kb + 1) * 2.0 ** -24 * mag).all()
