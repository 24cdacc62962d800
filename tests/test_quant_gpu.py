"""GPU parity of the quantization entry points against the CPU oracle, through the C ABI: bit-exact nibbles, scale bytes
(linear and swizzled, padding untouched), globals and the amax statistic.  Recipes and shapes follow the reference's
own quantizer test (tests/test_nvfp4effma.cu:498-524 there)."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from nvfp4effma_b200 import _lib as L
from util import dev, host, ptr, quant_input, stream, tensor

pytestmark = pytest.mark.gpu

SW, UE, AM, PR = L.SCALES_SWIZZLED, L.SCALES_UE5M3, L.GLOBAL_AMAX, L.GLOBAL_PER_ROW
SPECS = [  # name, tile, fos, flags, smax, compute, col
    ("1x16 given g", 1, 0, 0, 0, False, False),
    ("1x16 amax given, swizzled", 1, 0, AM | SW, 0, False, True),
    ("1x16 amax computed, swizzled", 1, 0, AM | SW, 0, True, False),
    ("16x16 amax computed", 16, 0, AM, 0, True, True),
    ("16x16 amax given, swizzled", 16, 0, AM | SW, 0, False, True),
    ("1x16 per-row amax computed", 1, 0, AM | PR, 0, True, True),
    ("1x16 4over6 MAE, 256", 1, 1, AM, 256, True, True),
    ("1x16 4over6 MSE, 448", 1, 2, AM | SW, 448, True, True),
    ("16x16 4over6 MAE, 256", 16, 1, AM | SW, 256, True, True),
    ("16x16 4over6 MSE, 256", 16, 2, AM, 256, False, True),
    ("1x16 per-row 4over6 MAE", 1, 1, AM | PR, 256, True, False),
    ("1x16 UE5M3 amax, swizzled", 1, 0, UE | AM | SW, 0, True, True),
    ("16x16 UE5M3 given g", 16, 0, UE, 0, False, True),
]


def test_hardware_conversions_equal_software_encoders_on_every_fp32():
    bad = torch.zeros(4, dtype=torch.int64, device="cuda")
    L.check(L.lib.nvfp4a_b200_codec_selftest(0, 1 << 32, ptr(bad), stream()))
    torch.cuda.synchronize()
    assert bad.tolist() == [0, 0, 0, 0]   # E2M1 low / high nibble, E4M3, packed BF16 rounding of the GEMM epilogues


def run_quant(dtype, rows, cols, spec, seed):
    name, tile, fos, flags, smax, compute, col = spec
    rng = np.random.default_rng(seed)
    lds = cols + 16
    x, raw = quant_input(rng, rows, cols, lds, dtype)
    amax_mode, per_row = bool(flags & AM), bool(flags & PR)
    rows16 = (rows + 15) // 16 * 16
    tam = float(np.abs(x[:, :cols]).max())
    ram = np.abs(x[:, :cols]).max(1).astype(np.float32)
    n_g = rows if per_row else 1
    g_given = (2000.0 + 37.0 * np.arange(n_g)).astype(np.float32) if amax_mode else np.full(n_g, 0.0625, np.float32)
    g_row0 = np.zeros(n_g, np.float32) if compute else g_given
    g_col0 = np.zeros(1, np.float32) if compute else g_given[:1].copy()
    # destinations with padded leading dimensions and 0xEE everywhere (padding must stay untouched)
    hr = O.Fp4(rows, cols, ld=cols + 32, ld_scale=cols // 16 + 3, flags=flags, scale_max=smax, glob=g_row0.copy(), fill=0xEE)
    hc = O.Fp4(cols, rows16, ld=rows16 + 32, ld_scale=rows16 // 16 + 1, flags=flags & ~PR, scale_max=smax, glob=g_col0.copy(), fill=0xEE)
    d_x = dev(raw)
    dr_d, dr_s, dr_g, dr_a = dev(hr.data), dev(hr.scales), dev(g_row0), dev(np.zeros(1, np.float32))
    dc_d, dc_s, dc_g, dc_a = dev(hc.data), dev(hc.scales), dev(g_col0), dev(np.zeros(1, np.float32))
    S = tensor(d_x, dtype)
    R = tensor(dr_d, L.NVFP4, dr_s, hr.ld_scale, dr_g, dr_a, flags, smax)
    Cc = tensor(dc_d, L.NVFP4, dc_s, hc.ld_scale, dc_g, dc_a, flags & ~PR, smax)
    cfg = L.QuantConfig(tile, fos, int(compute))
    st = L.lib.nvfp4a_quantize_ex(ctypes.byref(S), lds, rows, cols, ctypes.byref(R), hr.ld, ctypes.byref(Cc) if col else None, hc.ld,
                                  ctypes.byref(cfg), stream())
    L.check(st)
    torch.cuda.synchronize()
    # oracle
    O.quantize(x, hr, cols=cols, tile=tile, fos=fos, compute_amax=compute)
    assert np.array_equal(host(dr_g), hr.glob), f"{name}: rowwise global"
    assert np.array_equal(host(dr_d), hr.data), f"{name}: rowwise nibbles"
    assert np.array_equal(host(dr_s), hr.scales), f"{name}: rowwise scales"
    assert float(host(dr_a)[0]) == tam, f"{name}: amax statistic"
    if compute:
        assert np.array_equal(hr.glob, ram if per_row else np.array([tam], np.float32))
    if col:
        O.quantize(x, hc, cols=cols, transposed=True, tile=tile, fos=fos, compute_amax=compute)
        assert np.array_equal(host(dc_g), hc.glob), f"{name}: columnwise global"
        assert np.array_equal(host(dc_d), hc.data), f"{name}: columnwise nibbles"
        assert np.array_equal(host(dc_s), hc.scales), f"{name}: columnwise scales"
        assert float(host(dc_a)[0]) == tam
    return hr, dr_d, dr_s, dr_g


@pytest.mark.parametrize("spec", SPECS, ids=[s[0] for s in SPECS])
@pytest.mark.parametrize("dtype", [L.BF16, L.FP32])
def test_quantize_ex_recipes(spec, dtype):
    run_quant(dtype, 517, 1056, spec, 11)
    run_quant(dtype, 256, 320, spec, 12)


@pytest.mark.parametrize("spec", [SPECS[1], SPECS[11]], ids=["e4m3", "ue5m3"])
@pytest.mark.parametrize("dtype,rows,cols", [(L.BF16, 2064, 2128), (L.FP32, 2064, 2128), (L.FP32, 2177, 2112), (L.FP32, 17, 18944)])
def test_both_halves_of_many_tiles(spec, dtype, rows, cols):
    """The sizes from which a CTA takes a tall tile of rows (128 of FP32, 256 of 16-bit values): a last tile of a few rows, of part of a block, and nothing else."""
    run_quant(dtype, rows, cols, spec, 17)


def test_quantize_ex_small_and_fp16():
    run_quant(L.FP16, 40, 48, SPECS[8], 13)
    for dtype in (L.BF16, L.FP16, L.FP32):
        run_quant(dtype, 3, 16, SPECS[0], 14)
        run_quant(dtype, 517, 1056, SPECS[0], 15)
        run_quant(dtype, 130, 80, SPECS[2], 16)  # cols/16 = 5: swizzled rows with a ragged last group of 4


@pytest.mark.parametrize("dtype", [L.BF16, L.FP16, L.FP32])
def test_quantize_int8(dtype):
    rng = np.random.default_rng(21)
    rows, cols = 517, 1056
    lds, ld8, lsc = cols + 16, cols + 16, cols // 16 + 4
    u = ((rng.integers(0, 1 << 24, (rows, lds)) / float(1 << 24)) * 2 - 1) * np.ldexp(1.0, rng.integers(-10, 10, (rows, lds)))
    raw = O.from_f32(u.astype(np.float32), dtype)
    x = O.to_f32(raw, dtype).reshape(rows, lds)
    x[5, :32] = 0  # zero blocks: scale 0, codes 0
    raw = O.from_f32(x, dtype)
    h = O.Q8(rows, cols, ld=ld8, ld_scale=lsc)
    h.data[:] = 0x55
    h.scales[:] = np.frombuffer(b"\x55" * 4, np.float32)[0]
    d_q, d_s, d_a = dev(h.data), dev(h.scales), dev(np.zeros(1, np.float32))
    S = tensor(dev(raw), dtype)
    Q = tensor(d_q, L.INT8, d_s, lsc, None, d_a)
    L.check(L.lib.nvfp4a_quantize(ctypes.byref(S), lds, ctypes.byref(Q), ld8, rows, cols, stream()))
    torch.cuda.synchronize()
    amax = O.quantize_int8(x, h)
    assert np.array_equal(host(d_q), h.data)
    assert np.array_equal(host(d_s).view(np.uint32), h.scales.view(np.uint32))
    assert float(host(d_a)[0]) == amax


@pytest.mark.parametrize("flags,smax", [(0, 0), (AM | SW, 0), (AM, 256), (UE | AM | SW, 0), (AM | PR, 0)])
@pytest.mark.parametrize("dtype", [L.BF16, L.FP16, L.FP32])
def test_dequantize(flags, smax, dtype):
    from util import rand_fp4, DevFp4
    rng = np.random.default_rng(31)
    rows, cols = 517, 1056
    h = rand_fp4(rng, rows, cols, ld=cols + 32, ld_scale=cols // 16 + 3, flags=flags, scale_max=smax, glob=37.5 if flags & AM else 0.375)
    d = DevFp4(h)
    ldy = cols + 48
    esz = 4 if dtype == L.FP32 else 2
    y = torch.full((rows * ldy * esz,), 0xEE, dtype=torch.uint8, device="cuda")
    am = dev(np.zeros(1, np.float32))
    src, dst = d.tensor(), tensor(y, dtype, amax=am)
    L.check(L.lib.nvfp4a_dequantize(ctypes.byref(src), h.ld, ctypes.byref(dst), ldy, rows, cols, stream()))
    torch.cuda.synchronize()
    want, wamax = O.dequantize(h, dtype)
    got_raw = host(y).view(np.float32 if dtype == L.FP32 else np.uint16).reshape(rows, ldy)
    got = O.to_f32(got_raw[:, :cols], dtype)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    pad = host(y).reshape(rows, ldy * esz)[:, cols * esz:]
    assert np.all(pad == 0xEE)
    assert float(host(am)[0]) == wamax


@pytest.mark.parametrize("rows,cols", [(517, 1056), (3, 16), (128, 64)])
def test_swizzle_scales_both_ways(rows, cols):
    rng = np.random.default_rng(41)
    ld = cols // 16 + 5
    lin = rng.integers(0, 256, rows * ld, dtype=np.uint8)
    d_lin = dev(lin)
    d_swz = torch.full((O.scale_bytes(True, 0, rows, cols),), 0xEE, dtype=torch.uint8, device="cuda")
    d_back = torch.full((rows * ld,), 0xEE, dtype=torch.uint8, device="cuda")
    L.check(L.lib.nvfp4a_swizzle_scales(ptr(d_lin), ptr(d_swz), ld, rows, cols, 1, stream()))
    L.check(L.lib.nvfp4a_swizzle_scales(ptr(d_swz), ptr(d_back), ld, rows, cols, 0, stream()))
    torch.cuda.synchronize()
    assert np.array_equal(host(d_swz), O.swizzle_scales(lin, ld, rows, cols, True))
    b = host(d_back).reshape(rows, ld)
    assert np.array_equal(b[:, : cols // 16], lin.reshape(rows, ld)[:, : cols // 16]) and np.all(b[:, cols // 16:] == 0xEE)


def test_transpose_of_16x16_tiles_is_the_columnwise_quantization():
    spec = ("16x16 amax given", 16, 0, AM, 0, False, True)
    rows, cols = 256, 320
    rng = np.random.default_rng(51)
    x, raw = quant_input(rng, rows, cols, cols, L.BF16)
    g = np.array([2000.0], np.float32)
    hr = O.Fp4(rows, cols, flags=AM, glob=g)
    hc = O.Fp4(cols, rows, flags=AM, glob=g)
    O.quantize(x, hr, tile=16)
    O.quantize(x, hc, transposed=True, tile=16)
    from util import DevFp4
    dr = DevFp4(hr)
    ht = O.Fp4(cols, rows, flags=AM, glob=g, fill=0xEE)
    dt = DevFp4(ht)
    s, d = dr.tensor(), dt.tensor()
    L.check(L.lib.nvfp4a_transpose(ctypes.byref(s), cols, ctypes.byref(d), rows, rows, cols, stream()))
    torch.cuda.synchronize()
    assert np.array_equal(host(dt.data), hc.data) and np.array_equal(host(dt.scales), hc.scales)


def test_full_size_8192_square_bf16_swizzled_amax_computed():
    """Quantization of 8192 x 8192 at full size: N(0,1) with 1 % of entries x 50, swizzled scales, amax computed; bit-exact."""
    rng = np.random.default_rng(1)
    rows = cols = 8192
    x = rng.standard_normal((rows, cols), dtype=np.float32)
    x[rng.random((rows, cols)) < 0.01] *= 50.0
    raw = O.from_f32(x, L.BF16)
    x = O.to_f32(raw, L.BF16).reshape(rows, cols)
    flags = AM | SW
    h = O.Fp4(rows, cols, flags=flags, glob=np.zeros(1, np.float32))
    d_d = torch.zeros(h.data.size, dtype=torch.uint8, device="cuda")
    d_s = torch.zeros(h.scales.size, dtype=torch.uint8, device="cuda")
    d_g, d_a = dev(np.zeros(1, np.float32)), dev(np.zeros(1, np.float32))
    S = tensor(dev(raw), L.BF16)
    R = tensor(d_d, L.NVFP4, d_s, 0, d_g, d_a, flags, 0)
    cfg = L.QuantConfig(1, 0, 1)
    L.check(L.lib.nvfp4a_quantize_ex(ctypes.byref(S), cols, rows, cols, ctypes.byref(R), cols, None, 0, ctypes.byref(cfg), stream()))
    torch.cuda.synchronize()
    amax = O.quantize(x, h, compute_amax=True)
    assert float(host(d_g)[0]) == amax == float(host(d_a)[0])
    assert np.array_equal(host(d_d), h.data)
    assert np.array_equal(host(d_s), h.scales)


@pytest.mark.parametrize("dtype,flags,lds_pad,rows,cols", [(L.BF16, AM | SW, 0, 3001, 4160), (L.FP16, AM, 64, 2100, 4096), (L.BF16, AM | UE, 0, 8190, 1088)])
def test_one_read_kernel_equals_the_two_launch_path(dtype, flags, lds_pad, rows, cols):
    """Large matrices with the common recipe run as one cooperative kernel that keeps part of the matrix on the chip between the
    amax visit and the encode visit; nvfp4a_b200_set_quant_fused(0) pins the amax kernel + encode kernel pair instead.  Both must
    write the same bytes (rows that do not divide over the SMs, a ragged last 64-block unit per row, padded source pitch, FP16,
    UE5M3 scales) -- and repeated calls must agree (the grid barrier's counter carries over from launch to launch)."""
    rng = np.random.default_rng(rows + cols)
    lds = cols + lds_pad
    x = rng.standard_normal((rows, lds), dtype=np.float32) * 3.0
    x[rng.random((rows, lds)) < 0.002] *= 100.0
    d_x = dev(O.from_f32(x, dtype))
    sbytes = O.scale_bytes(bool(flags & SW), 0 if flags & SW else cols // 16, rows, cols)
    outs = []
    try:
        for fused in (1, 0, 1):
            assert L.lib.nvfp4a_b200_set_quant_fused(fused) == 0
            d_d = torch.full((rows * cols // 2,), 0xEE, dtype=torch.uint8, device="cuda")
            d_s = torch.full((sbytes,), 0xEE, dtype=torch.uint8, device="cuda")
            d_g, d_a = dev(np.zeros(1, np.float32)), dev(np.zeros(1, np.float32))
            S, R = tensor(d_x, dtype), tensor(d_d, L.NVFP4, d_s, 0, d_g, d_a, flags, 0)
            cfg = L.QuantConfig(1, 0, 1)
            L.check(L.lib.nvfp4a_quantize_ex(ctypes.byref(S), lds, rows, cols, ctypes.byref(R), cols, None, 0, ctypes.byref(cfg), stream()))
            torch.cuda.synchronize()
            outs.append((host(d_d), host(d_s), float(host(d_g)[0]), float(host(d_a)[0])))
    finally:
        L.lib.nvfp4a_b200_set_quant_fused(1)
    st = ctypes.c_uint(0)
    L.check(L.lib.nvfp4a_b200_kernel_status(ctypes.byref(st), 1))
    assert st.value == 0
    for other in outs[1:]:
        assert np.array_equal(outs[0][0], other[0]) and np.array_equal(outs[0][1], other[1]) and outs[0][2:] == other[2:]
    xr = O.to_f32(O.from_f32(x, dtype), dtype).reshape(rows, lds)[:, :cols]
    assert outs[0][2] == float(np.abs(xr).max()) == outs[0][3]


@pytest.mark.parametrize("flags,compute", [(0, False), (AM | SW, True), (UE | AM, True)])
@pytest.mark.parametrize("dtype", [L.BF16, L.FP16, L.FP32])
def test_both_directions_from_one_read_at_the_edges_of_its_tiles(dtype, flags, compute):
    """Rowwise and columnwise 1 x 16 blocks without 4over6 take the one-read kernel: 64-row and (the last shape) 256-row tiles of 64
    columns, with every kind of remainder, against the oracle byte for byte."""
    for i, (rows, cols) in enumerate([(1, 16), (16, 48), (63, 64), (65, 80), (80, 1040), (257, 128), (2064 + 5, 2320)]):
        if i == 6 and dtype != L.BF16 and flags:
            continue
        run_quant(dtype, rows, cols, ("one read", 1, 0, flags, 0, compute, True), 700 + i)


@pytest.mark.parametrize("flags", [0, AM | SW, UE | AM, PR])
@pytest.mark.parametrize("dtype", [L.BF16, L.FP16])
def test_dequantize_by_table_equals_dequantize_value_by_value(dtype, flags):
    """A 16-bit destination without amax takes the table kernel; with amax the value-by-value one.  Same bytes for every nibble under every
    scale code (negative E4M3 codes, 0x7F and 0xFF = +-480 included) and globals from 0 over subnormal to Inf and NaN, at the edges of the 4-row,
    32-block units; the finite case also against the oracle."""
    rng = np.random.default_rng(77)
    from util import rand_fp4, DevFp4
    for rows, cols, pad in ((1, 16, 0), (4, 512, 16), (5, 528, 0), (130, 1056, 48)):
        for gv in (0.375, 0.0, 1e-40, 3e38, float("inf"), float("nan"), -2.5):
            h = rand_fp4(rng, rows, cols, ld=cols + 32, ld_scale=cols // 16 + 3, flags=flags, glob=0.375)
            if not flags & UE:
                h.scales[:] = rng.integers(0, 256, h.scales.size)
            h.glob[:] = gv
            d = DevFp4(h)
            out = []
            for with_amax in (False, True):
                y = torch.full((rows * (cols + pad),), 0x55, dtype=torch.int16, device="cuda")
                am = dev(np.zeros(1, np.float32))
                src, dst = d.tensor(), tensor(y, dtype, amax=am if with_amax else None)
                L.check(L.lib.nvfp4a_dequantize(ctypes.byref(src), h.ld, ctypes.byref(dst), cols + pad, rows, cols, stream()))
                torch.cuda.synchronize()
                out.append(host(y).view(np.uint16).reshape(rows, cols + pad))
            assert np.array_equal(out[0], out[1]), (rows, cols, gv)
            if gv == 0.375 and flags & UE:
                want, _ = O.dequantize(h, dtype)
                assert np.array_equal(O.to_f32(np.ascontiguousarray(out[0][:, :cols]).reshape(-1), dtype).reshape(rows, cols), want)


@pytest.mark.parametrize("lo,hi", [(-10, 10), (-61, -66), (62, 67), (-126, -100), (100, 127), (-149, 127)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_quantize_int8_without_divisions_equals_ieee_divisions(dtype, lo, hi):
    """q = clamp(rint(x / sb), +-127) by a reciprocal and two fused multiply-adds, or by IEEE divisions where a block's scale is too far from one or a value is a
    NaN: torch's IEEE division gives the same bytes.  Quotients at and beside every half integer, random significands, zeros, infinities, NaNs."""
    import nvfp4effma_b200.api as nf
    gen = torch.Generator(device="cuda").manual_seed(5)
    n = 1 << 20
    e = torch.randint(min(lo, hi), max(lo, hi) + 1, (n, 1), generator=gen, device="cuda").float()
    x = (torch.rand(n, 16, generator=gen, device="cuda") * 2 - 1).double()
    x[: n // 2, 0] = 1.0 - torch.rand(n // 2, generator=gen, device="cuda").double() / 4
    half = (torch.randint(0, 127, (n // 2, 15), generator=gen, device="cuda").double() + 0.5) / 127.0 * x[: n // 2, :1]   # quotients near k + 1/2
    x[: n // 2, 1:] = half * (1 + torch.randint(-2, 3, half.shape, generator=gen, device="cuda").double() * 2.0 ** -24)
    x = (x * torch.exp2(e.double())).to(dtype)
    x[7] = 0.0
    if hi - lo > 200:
        x[8:1000:9, 3] = float("nan")
        x[9:1000:9, 5] = float("inf")
    x = x.view(-1, 512)
    got = nf.quantize_int8(x)
    v = x.float().view(n, 16)
    bmax = torch.where(v.isnan(), torch.zeros_like(v), v.abs()).amax(-1, keepdim=True)
    sb = bmax / torch.tensor(127.0, device="cuda")
    q = (v / sb).round()
    q = torch.where(q.isnan(), torch.full_like(q, -127.0), q.clamp(-127, 127))   # (fmax(NaN, -127) = -127)
    q = torch.where(sb > 0, q, torch.zeros_like(q)).to(torch.int8)
    assert torch.equal(got.scales.view(n, 1).view(torch.int32), sb.view(torch.int32))
    assert torch.equal(got.data.view(n, 16), q)


@pytest.mark.parametrize("offset,pad", [(0, 0), (16, 0), (0, 16), (16, 48)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_blocks_of_32_bytes_at_every_alignment(dtype, offset, pad):
    """32-byte loads and stores where base and row pitch allow them, 16-byte ones elsewhere: the same bytes from the quantizer (amax computed, in one launch
    and in two, and given) and from the dequantizer (padding untouched)."""
    import nvfp4effma_b200.api as nf
    esz = torch.empty(0, dtype=dtype).element_size()
    for rows, cols in ((37, 1040), (1031, 8192)):
        ld = cols + pad
        gen = torch.Generator(device="cuda").manual_seed(rows)
        base = torch.randn(rows * ld + 64, generator=gen, device="cuda").to(dtype)
        x = base[offset // esz:][: rows * ld].view(rows, ld)
        xc = x[:, :cols].contiguous()
        want = nf.quantize(xc)
        for compute in (1, 0):
            data = torch.zeros(rows, cols // 2, dtype=torch.uint8, device="cuda")
            sc = torch.zeros(rows, cols // 16, dtype=torch.uint8, device="cuda")
            glob = want.amax.clone().float().reshape(1) if not compute else torch.zeros(1, device="cuda")
            S, Q = tensor(x, {torch.bfloat16: L.BF16, torch.float16: L.FP16, torch.float32: L.FP32}[dtype]), tensor(data, L.NVFP4, sc, cols // 16, glob, None, L.GLOBAL_AMAX)
            cfg = L.QuantConfig(1, 0, compute)
            L.check(L.lib.nvfp4a_quantize_ex(ctypes.byref(S), ld, rows, cols, ctypes.byref(Q), cols, None, 0, ctypes.byref(cfg), stream()))
            assert torch.equal(data, want.data.view(torch.uint8)) and torch.equal(sc, want.scales.view(torch.uint8).reshape(rows, -1)[:, : cols // 16])
        if dtype == torch.float32:
            continue
        back = torch.full((rows * ld + 64,), 7.0, dtype=dtype, device="cuda")
        out = back[offset // esz:][: rows * ld].view(rows, ld)
        Dt = tensor(out, L.BF16 if dtype == torch.bfloat16 else L.FP16)
        Q = tensor(want.data, L.NVFP4, want.scales, want.scales.shape[-1], want.amax, None, L.GLOBAL_AMAX)
        L.check(L.lib.nvfp4a_dequantize(ctypes.byref(Q), cols, ctypes.byref(Dt), ld, rows, cols, stream()))
        assert torch.equal(out[:, :cols], nf.dequantize(want, dtype))
        assert bool((back[: offset // esz] == 7).all()) and bool((out[:, cols:] == 7).all()) and bool((back[offset // esz + rows * ld:] == 7).all())


@pytest.mark.parametrize("offset,pad", [(0, 0), (16, 0), (0, 16), (16, 48)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_both_directions_at_every_alignment(dtype, offset, pad):
    """The one-read kernel of both directions takes a block's 32 bytes in one load where base and pitch allow it: the same bytes as from an aligned copy, with
    64-row and 256-row tiles and remainders of both."""
    import nvfp4effma_b200.api as nf
    esz, code = torch.empty(0, dtype=dtype).element_size(), {torch.bfloat16: L.BF16, torch.float16: L.FP16, torch.float32: L.FP32}[dtype]
    for rows, cols in ((80, 208), (2064, 2320)):
        ld = cols + pad
        gen = torch.Generator(device="cuda").manual_seed(rows + 1)
        base = torch.randn(rows * ld + 64, generator=gen, device="cuda").to(dtype)
        x = base[offset // esz:][: rows * ld].view(rows, ld)
        want = nf.quantize(x[:, :cols].contiguous(), columnwise=True)
        out = []
        for r, c in ((rows, cols), (cols, rows)):
            data, sc = torch.zeros(r, c // 2, dtype=torch.uint8, device="cuda"), torch.zeros(r, (c // 16 + 3) // 4 * 4, dtype=torch.uint8, device="cuda")
            out.append((data, sc, tensor(data, L.NVFP4, sc, sc.shape[1], torch.zeros(1, device="cuda"), None, L.GLOBAL_AMAX)))
        S, cfg = tensor(x, code), L.QuantConfig(1, 0, 1)
        L.check(L.lib.nvfp4a_quantize_ex(ctypes.byref(S), ld, rows, cols, ctypes.byref(out[0][2]), cols, ctypes.byref(out[1][2]), rows, ctypes.byref(cfg), stream()))
        for (data, sc, _), w, c in ((out[0], want, cols), (out[1], want.columnwise, rows)):
            assert torch.equal(data, w.data.view(torch.uint8)) and torch.equal(sc[:, : c // 16], w.scales.view(torch.uint8)[:, : c // 16])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_one_launch_equals_two_on_infinities_nans_and_zeros(dtype):
    """From 65536 values up the amax and the encoding are one launch: the bytes and the amax of the two-launch path for matrices of zeros, with a NaN of either sign, an
    infinity, both, nothing but NaNs, subnormals and the largest finite value; rows that end inside a unit; linear and swizzled scales, E4M3 and UE5M3."""
    import nvfp4effma_b200.api as nf
    gen = torch.Generator(device="cuda").manual_seed(31)
    top, tiny = torch.finfo(dtype).max, torch.finfo(dtype).smallest_normal / 4
    for rows, cols in ((64, 1024), (300, 576), (1031, 2048)):
        normal = torch.randn(rows, cols, generator=gen, device="cuda")
        at = torch.randint(0, rows * cols, (5,), generator=gen, device="cuda")
        cases = [torch.zeros(rows, cols, device="cuda"), torch.full((rows, cols), float("nan"), device="cuda"), normal * tiny, normal]
        for values in ([float("nan")], [-float("nan"), float("nan")], [float("inf")], [-float("inf"), float("nan"), top], [-top, tiny, -0.0]):
            x = normal.clone()
            x.view(-1)[at[: len(values)]] = torch.tensor(values, device="cuda")
            cases.append(x)
        for i, x in enumerate(cases):
            x = x.to(dtype)
            out = []
            try:
                for fused in (1, 0):
                    L.lib.nvfp4a_b200_set_quant_fused(fused)
                    q = nf.quantize(x, swizzled=i % 2 == 0, scale_dtype="ue5m3" if i % 3 == 2 else "e4m3")
                    out.append((q.data.view(torch.uint8), q.scales.view(torch.uint8), q.amax.view(torch.int32)))
            finally:
                L.lib.nvfp4a_b200_set_quant_fused(1)
            assert all(torch.equal(a, b) for a, b in zip(*out)), (rows, cols, i)


def test_small_matrices_quantize_in_one_launch_on_several_streams():
    """The cooperative kernel from 65536 values up, many launches on four streams at once (launches of it share a barrier counter and alternate between two
    arrays of maxima): every result has the bytes of the two-launch path."""
    import nvfp4effma_b200.api as nf
    gen = torch.Generator(device="cuda").manual_seed(9)
    xs = [(torch.randn(r, c, generator=gen, device="cuda") * 2.0 ** i).to(dt) for i, (r, c, dt) in
          enumerate([(64, 1024, torch.bfloat16), (131, 512, torch.float16), (300, 4096, torch.bfloat16), (1000, 2048, torch.float16), (2048, 4096, torch.bfloat16)])]
    L.lib.nvfp4a_b200_set_quant_fused(0)
    try:
        want = [nf.quantize(x, swizzled=True) for x in xs]
    finally:
        L.lib.nvfp4a_b200_set_quant_fused(1)
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    got = []
    for rep in range(40):
        for i in range(len(xs)):
            with torch.cuda.stream(streams[(rep + i) % 4]):
                got.append((i, nf.quantize(xs[i], swizzled=True)))
    torch.cuda.synchronize()
    for i, q in got:
        w = want[i]
        assert torch.equal(q.data.view(torch.uint8), w.data.view(torch.uint8)) and torch.equal(q.scales.view(torch.uint8), w.scales.view(torch.uint8))
        assert torch.equal(q.amax, w.amax)


@pytest.mark.parametrize("dtype,flags,rows,cols,pad,offset", [
    (torch.float16, AM | SW, 4100, 8256, 0, 0),      # 33.8 M values: units in shared memory, in tensor memory and read again; the last unit of a row is ragged
    (torch.bfloat16, AM | UE, 8190, 4160, 16, 0),
    (torch.float16, AM | UE, 6001, 8192, 16, 8),     # rows on 16-byte boundaries only: two loads for a block
    (torch.bfloat16, AM | SW, 4100, 4160, 0, 0),     # tensor memory, nothing read again
])
def test_quantizer_that_keeps_units_in_tensor_memory_equals_the_two_launch_path(dtype, flags, rows, cols, pad, offset):
    gen = torch.Generator(device="cuda").manual_seed(rows)
    lds = cols + pad
    base = torch.randn(rows * lds + offset, generator=gen, device="cuda").mul_(3.0)
    base[torch.randint(0, rows * lds, (1000,), generator=gen, device="cuda")] *= 100.0
    x = base.to(dtype)[offset:]
    code = L.FP16 if dtype == torch.float16 else L.BF16
    sbytes = O.scale_bytes(bool(flags & SW), 0 if flags & SW else cols // 16, rows, cols)
    outs = []
    try:
        for fused in (1, 0, 1):
            assert L.lib.nvfp4a_b200_set_quant_fused(fused) == 0
            d, s = torch.full((rows * cols // 2,), 0xEE, dtype=torch.uint8, device="cuda"), torch.full((sbytes,), 0xEE, dtype=torch.uint8, device="cuda")
            glob, amax = torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda")
            S, R = tensor(x, code), tensor(d, L.NVFP4, s, 0 if flags & SW else cols // 16, glob, amax, flags, 0)
            cfg = L.QuantConfig(1, 0, 1)
            L.check(L.lib.nvfp4a_quantize_ex(ctypes.byref(S), lds, rows, cols, ctypes.byref(R), cols, None, 0, ctypes.byref(cfg), stream()))
            outs.append((d, s, glob, amax))
    finally:
        L.lib.nvfp4a_b200_set_quant_fused(1)
    assert float(outs[0][2]) == float(x[: rows * lds].view(rows, lds)[:, :cols].abs().max())
    for other in outs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(outs[0], other))


def test_both_quantizers_of_one_launch_take_turns_on_several_streams():
    """The sixteen-warp kernel and the one with tensor memory share the barrier's counter and the arrays of maxima: matrices of both, with and without tensor memory and a
    second read, on four streams at once."""
    import nvfp4effma_b200.api as nf
    gen = torch.Generator(device="cuda").manual_seed(10)
    xs = [(torch.randn(r, c, generator=gen, device="cuda") * 2.0 ** i).to(dt) for i, (r, c, dt) in
          enumerate([(64, 1024, torch.bfloat16), (3000, 4096, torch.bfloat16), (300, 4096, torch.float16), (4100, 4096, torch.float16), (8200, 4160, torch.bfloat16)])]
    L.lib.nvfp4a_b200_set_quant_fused(0)
    try:
        want = [nf.quantize(x, swizzled=True) for x in xs]
    finally:
        L.lib.nvfp4a_b200_set_quant_fused(1)
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()
    got = []
    for rep in range(16):
        for i in range(len(xs)):
            with torch.cuda.stream(streams[(rep + i) % 4]):
                got.append((i, nf.quantize(xs[i], swizzled=True)))
    torch.cuda.synchronize()
    for i, q in got:
        w = want[i]
        assert torch.equal(q.data.view(torch.uint8), w.data.view(torch.uint8)) and torch.equal(q.scales.view(torch.uint8), w.scales.view(torch.uint8))
        assert torch.equal(q.amax, w.amax)
