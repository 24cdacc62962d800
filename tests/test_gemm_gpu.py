"""GPU parity of nvfp4a_gemm / nvfp4a_gemm_ex / the image entries against the CPU oracle, through the C ABI.

Two kinds of check, as the reference's own tests make them (tests/test_util.h:153-155, :292-321 there):
  * the CUDA-core route computes the documented tiled order, so D and amax are compared bit for bit;
  * the tcgen05 and GEMV routes sum in their own order, so they are compared with the float64 value within the
    FP32-accumulation bound (k + 2) 2^-24 sum|a b| |s| + 4 2^-24 (|r s| + |bias| + |beta C|) + out_rel |v| + out_abs,
    amax within 2^-7 relative; the share of outputs within 1 BF16 ulp of the exact block-sum oracle is reported too.
Shapes, leading-dimension padding and format combinations follow tests/test_gemm.cu:13-41 and tests/test_gemv.cu:13-42 there."""
import ctypes
import os

import numpy as np
import pytest
import torch

import oracle as O
from nvfp4effma_b200 import _lib as L
from util import DevFp4, dev, host, ptr, rand_dense, rand_fp4, rand_q8, stream, tensor

pytestmark = pytest.mark.gpu

OUTS = [L.BF16, L.FP32, L.FP16]
OPS = [L.NVFP4, L.INT8, L.BF16, L.FP16, L.FP32]
SW, UE, AM, PR = L.SCALES_SWIZZLED, L.SCALES_UE5M3, L.GLOBAL_AMAX, L.GLOBAL_PER_ROW


def esize(t):
    return 4 if t == L.FP32 else 2


class Case:
    def __init__(self, m, n, k, bt, dt, ct, bias, alpha, beta, fa=0, fb=0, ma=0, mb=0):
        self.m, self.n, self.k, self.bt, self.dt, self.ct, self.bias, self.alpha, self.beta = m, n, k, bt, dt, ct, bias, alpha, beta
        self.fa, self.fb, self.ma, self.mb = fa, fb, ma, mb

    def __repr__(self):
        return f"m{self.m}n{self.n}k{self.k}-B{self.bt}-D{self.dt}-C{self.ct}-b{self.bias}-fa{self.fa:x}/{self.ma}-fb{self.fb:x}/{self.mb}"


def build_case(c, seed):
    """Host operands of a case, padded as the reference's run_case pads them."""
    rng = np.random.default_rng(seed)
    fp4b, q8b = c.bt == L.NVFP4, c.bt == L.INT8
    lda, ldb = c.k + 64, c.k + (128 if fp4b else 64)
    ldd = c.m + 3
    ldc = c.m + 1 if c.ct >= 0 else ldd
    ct = c.ct if c.ct >= 0 else c.dt
    A = rand_fp4(rng, c.m, c.k, ld=lda, ld_scale=c.k // 16 + 4, flags=c.fa, scale_max=c.ma, glob=37.5 if c.fa & AM else 0.375)
    if fp4b:
        B = rand_fp4(rng, c.n, c.k, ld=ldb, ld_scale=c.k // 16 + 8, flags=c.fb, scale_max=c.mb, glob=175.0 if c.fb & AM else 1.75)
    elif q8b:
        B = rand_q8(rng, c.n, c.k, ld=ldb, ld_scale=c.k // 16 + 8, glob=1.75)
    else:
        B = O.Dense(c.bt, rand_dense(rng, c.bt, ldb * c.n, 2.0), ldb)
    Cbuf = rand_dense(rng, ct, ldc * c.n, 4.0)
    if c.ct < 0:
        Dinit = rand_dense(rng, c.dt, ldd * c.n, 4.0)
        Cbuf = None
    else:
        Dinit = np.frombuffer(b"\xA5" * (ldd * c.n * esize(c.dt)), dtype=np.float32 if c.dt == L.FP32 else np.uint16).copy()
    bias = rand_dense(rng, c.bias, c.m, 8.0) if c.bias >= 0 else None
    return dict(A=A, B=B, C=Cbuf, ct=ct, ldc=ldc, Dinit=Dinit, ldd=ldd, bias=bias, lda=lda, ldb=ldb)


def oracle_case(c, h, want_ref=False, order=0):
    return O.gemm(c.m, c.n, c.k, h["A"], h["B"], D_dtype=c.dt, alpha=c.alpha, beta=c.beta, C=h["C"], C_dtype=h["ct"], ldc=h["ldc"],
                  ldd=h["ldd"], bias=h["bias"], bias_dtype=c.bias if c.bias >= 0 else L.FP32, lda=h["lda"], ldb=h["ldb"],
                  D_init=h["Dinit"], want_ref=want_ref, order=order)


def device_b(c, h):
    B = h["B"]
    if c.bt == L.NVFP4:
        d = DevFp4(B)
        return d, d.tensor()
    if c.bt == L.INT8:
        keep = (dev(B.data), dev(B.scales), dev(B.glob))
        return keep, tensor(keep[0], L.INT8, keep[1], B.ld_scale, keep[2])
    keep = dev(B.raw)
    return keep, tensor(keep, c.bt)


def run_gemm(c, h, lib=None):
    """nvfp4a_gemm on the device (of this library, or of ``lib``); returns (raw D buffer, amax)."""
    lib = lib or L.lib
    dA = DevFp4(h["A"])
    keepB, tB = device_b(c, h)
    dD, damax = dev(h["Dinit"]), dev(np.zeros(1, np.float32))
    dC = dev(h["C"]) if h["C"] is not None else None
    dbias = dev(h["bias"]) if h["bias"] is not None else None
    tA = dA.tensor()
    tC = tensor(dC, h["ct"]) if dC is not None else None
    tD = tensor(dD, c.dt, amax=damax)
    tbias = tensor(dbias, c.bias) if dbias is not None else None
    st = lib.nvfp4a_gemm(c.m, c.n, c.k, c.alpha, ctypes.byref(tA), h["lda"], ctypes.byref(tB), h["ldb"], c.beta,
                           ctypes.byref(tC) if tC is not None else None, h["ldc"], ctypes.byref(tD), h["ldd"],
                           ctypes.byref(tbias) if tbias is not None else None, stream())
    assert st == 0, lib.nvfp4a_last_error()
    torch.cuda.synchronize()
    return host(dD).view(h["Dinit"].dtype), float(host(damax)[0])


def values(raw, c, h):
    return O.to_f32(raw.reshape(c.n, h["ldd"])[:, : c.m], c.dt).astype(np.float64)


def check_bound(c, h, got_raw, got_amax, exp):
    """Tolerance check of a kernel that sums in its own order (reference tests/test_util.h:292-320)."""
    got = values(got_raw, c, h)
    with np.errstate(invalid="ignore", over="ignore"):
        err = np.abs(got - exp["ref64"])
        # an output that overflowed its dtype (FP16 Inf) counts as equal when the float64 value rounds to the same bits
        same = got == values(O.from_f32(exp["ref64"].astype(np.float32).reshape(-1), c.dt).reshape(c.n, c.m), c, dict(h, ldd=c.m))
        ratio = np.where(same, 0.0, err / exp["bound"])
    worst = float(np.nanmax(ratio)) if ratio.size else 0.0
    assert not np.isnan(ratio).any() and worst <= 1.0, f"{c}: max |error| / bound = {worst:.3f}"
    # padding between columns untouched
    g2 = got_raw.reshape(c.n, h["ldd"])[:, c.m:]
    i2 = h["Dinit"].reshape(c.n, h["ldd"])[:, c.m:]
    assert np.array_equal(g2, i2), f"{c}: padding of D was written"
    assert abs(got_amax - exp["amax"]) <= 2.0 ** -7 * exp["amax"] + 1e-30, f"{c}: amax {got_amax} vs {exp['amax']}"
    return worst


def cases_tiled():
    out, idx = [], 0
    sizes = [(1, 9, 64), (37, 45, 128), (200, 300, 192), (257, 129, 256), (128, 128, 64), (200, 64, 128), (150, 192, 256)]
    for bt in OPS:
        for m, n, k in sizes:
            out.append(Case(m, n, k, bt, OUTS[idx % 3], -1 if idx % 4 == 1 else (OUTS[(idx + 1) % 3] if idx % 4 == 2 else OUTS[idx % 3]),
                            -1 if idx % 3 == 0 else (L.BF16 if idx % 3 == 1 else L.FP32), 1.25 if idx % 2 else 1.0,
                            1.0 if idx % 4 == 1 else (0.5 if idx % 4 == 3 else 0.0)))
            idx += 1
    for bt in OPS:
        out.append(Case(1100, 1300, 512, bt, L.BF16, -1, -1, 1.0, 0.0))
        out.append(Case(1029, 700, 1024, bt, L.FP32, -1, L.FP32, 0.5, 1.0))
    return out


def set_formats(c, f, v):
    """The reference's format matrix (tests/test_util.h:135-151): bits 0..3 scale layout / type of A and B, 16 amax, 32 / 64 per-row."""
    fp4b = c.bt == L.NVFP4
    c.fa = (SW if f & 1 else 0) | (UE if f & 2 else 0) | (PR if f & 32 else 0)
    c.fb = ((SW if f & 4 else 0) | (UE if f & 8 else 0) | (PR if f & 64 else 0)) if fp4b else 0
    if f & 16:
        on = v % 3 if fp4b else 0
        if on != 1:
            c.fa |= AM
        if on != 0:
            c.fb |= AM
    c.ma = 256 if (c.fa & AM) and not (f & 2) and v % 2 else 0
    c.mb = 256 if (c.fb & AM) and not (f & 8) and v % 4 >= 2 else 0
    return c


def cases_formats(sizes):
    out, v = [], 0
    for bt in OPS:
        nf = 128 if bt == L.NVFP4 else 16
        for i in range(nf):
            m, n, k = sizes[v % len(sizes)]
            c = Case(m, n, k, bt, OUTS[v % 3], -1 if v % 4 == 1 else OUTS[v % 3], L.BF16 if v % 3 else -1, 1.25 if v % 2 else 1.0,
                     1.0 if v % 4 == 1 else 0.0)
            f = i if bt == L.NVFP4 else ((i & 3) | (16 if i & 4 else 0) | (32 if i & 8 else 0))
            out.append(set_formats(c, f, v))
            v += 1
    return out


@pytest.fixture
def exact_route():
    """Pins the GEMM entries to the CUDA-core kernel (the documented tiled order) for one test."""
    old = L.lib.nvfp4a_b200_set_route(1)
    yield
    L.lib.nvfp4a_b200_set_route(old)


def test_cuda_core_route_is_bit_exact_in_the_tiled_order(exact_route):
    """Every B dtype, tails, padded leading dimensions, C / accumulate / alpha / beta / bias / amax, all 128 + 4 x 16 formats."""
    fmt_sizes = [(257, 129, 256), (200, 64, 128), (300, 300, 320), (150, 192, 256)]
    bad = []
    for i, c in enumerate(cases_tiled()[:35] + cases_formats(fmt_sizes)):
        h = build_case(c, 1000 + i)
        exp = oracle_case(c, h)
        got, amax = run_gemm(c, h)
        if not np.array_equal(got, exp["D"]) or amax != exp["amax"]:
            bad.append(repr(c))
    assert not bad, f"{len(bad)} cases differ: {bad[:5]}"


def test_cuda_core_route_decodes_signed_block_scales_like_the_reference(exact_route):
    """Block-scale codes with the sign bit set are legal E4M3 for the reference (src/nvfp4effma.cuh:56-60 there); the tensor cores
    read scales as unsigned, so such tensors belong on the CUDA-core route, which must decode them exactly: D and amax equal the
    oracle's bit for bit with negative scales on both operands, linear and swizzled."""
    for i, (fa, fb) in enumerate([(0, 0), (SW, SW), (SW | AM, PR)]):
        c = Case(200, 150, 256, L.NVFP4, OUTS[i % 3], -1, L.FP32, 1.25, 0.0, fa=fa, fb=fb)
        h = build_case(c, 1500 + i)
        rng = np.random.default_rng(1500 + i)
        for t in (h["A"], h["B"]):
            flip = rng.integers(0, 3, t.scales.size) == 0
            t.scales[flip & (t.scales != 0)] |= 0x80
        assert (h["A"].scales & 0x80).any() and (h["B"].scales & 0x80).any()
        exp = oracle_case(c, h)
        got, amax = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == 1
        assert np.array_equal(got, exp["D"]) and amax == exp["amax"], c


def test_default_routes_within_the_accumulation_bound():
    """nvfp4a_gemm as routed by default (tcgen05 / GEMV / CUDA cores) against the float64 reference within the bound."""
    fmt_sizes = [(257, 129, 256), (200, 64, 128), (300, 300, 320), (150, 192, 256)]
    gemv_sizes = [(300, 3, 1024), (1000, 8, 576), (130, 20, 4160), (77, 1, 128), (64, 5, 64)]
    worst_all = 0.0
    for i, c in enumerate(cases_tiled() + cases_formats(fmt_sizes) + cases_formats(gemv_sizes)):
        h = build_case(c, 5000 + i)
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_gemm(c, h)
        worst_all = max(worst_all, check_bound(c, h, got, amax, exp))
    print(f"max |error| / bound over all cases = {worst_all:.3f}")


def test_gemv_shapes_n_1_to_8_and_groups():
    idx = 0
    gs = [(1, 64), (33, 576), (300, 1024), (1000, 4160)]
    cases = []
    for bt in OPS:
        for n in range(1, 9):
            m, k = gs[(n + bt) % 4]
            cases.append(Case(m, n, k, bt, OUTS[idx % 3], -1 if n == 3 else OUTS[idx % 3], -1 if idx % 3 == 0 else L.BF16,
                              0.75 if idx % 2 else 1.0, 1.0 if n == 3 else (-1.5 if idx % 4 == 1 else 0.0)))
            idx += 1
        for n in (12, 17, 32, 33, 48, 49):
            cases.append(Case(300, n, 1024, bt, OUTS[idx % 3], -1 if n == 17 else OUTS[idx % 3], L.BF16 if idx % 2 else -1, 1.0,
                              1.0 if n == 17 else 0.0))
            idx += 1
    for i, c in enumerate(cases):
        h = build_case(c, 9000 + i)
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_gemm(c, h)
        check_bound(c, h, got, amax, exp)


def test_k_zero_and_empty():
    c = Case(50, 3, 0, L.BF16, L.FP32, L.FP32, L.FP32, 1.0, 0.5)
    h = build_case(Case(50, 3, 64, L.BF16, L.FP32, L.FP32, L.FP32, 1.0, 0.5), 77)
    exp = O.gemm(50, 3, 0, h["A"], h["B"], D_dtype=L.FP32, alpha=1.0, beta=0.5, C=h["C"], C_dtype=L.FP32, ldc=h["ldc"], ldd=h["ldd"],
                 bias=h["bias"], bias_dtype=L.FP32, lda=h["lda"], ldb=h["ldb"], D_init=h["Dinit"])
    got, amax = run_gemm(c, h)
    assert np.array_equal(got, exp["D"]) and amax == exp["amax"]


def kernel_status(reset=True):
    st = ctypes.c_uint(0)
    L.check(L.lib.nvfp4a_b200_kernel_status(ctypes.byref(st), int(reset)))
    return st.value


def frac_within_1ulp_bf16(got, exact):
    """Share of outputs within one BF16 ulp of the exact block-sum oracle (both as float64 arrays of BF16 values)."""
    from util import ulp_bf16
    return float(np.mean(np.abs(got - exact) <= ulp_bf16(exact)))


@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("fa,fb", [(0, 0), (SW, SW), (SW, 0), (0, SW), (AM, AM | PR), (SW | PR, SW | AM)])
def test_w4a4_tcgen05_kernel(bn, fa, fb):
    """NVFP4 x NVFP4 on the tcgen05 route: every scale layout pair, m / n / k tails, both tile widths."""
    assert L.lib.nvfp4a_b200_set_tile_n(bn) == 0
    try:
        for i, (m, n, k) in enumerate([(128, 128, 256), (257, 129, 320), (200, 300, 192), (1100, 1300, 512), (64, 40, 64), (384, 512, 1024)]):
            c = Case(m, n, k, L.NVFP4, OUTS[i % 3], -1 if i % 4 == 1 else OUTS[i % 3], L.BF16 if i % 2 else -1, 1.25 if i % 2 else 1.0,
                     1.0 if i % 4 == 1 else 0.0, fa=fa, fb=fb, ma=256 if fa & AM else 0)
            h = build_case(c, 700 + i)
            exp = oracle_case(c, h, want_ref=True)
            got, amax = run_gemm(c, h)
            assert kernel_status() == 0
            check_bound(c, h, got, amax, exp)
    finally:
        L.lib.nvfp4a_b200_set_tile_n(0)


def test_w4a4_cta_pair_kernel_matches_the_single_cta_kernel():
    """The CTA-pair form (tcgen05.mma.cta_group::2, 256 x 256 tiles) against the bound and, bit for bit, against the single-CTA
    kernel, which feeds the same block products to the tensor cores in the same k order: odd numbers of 128-row tiles, tails
    in m / n / k, several tiles per pair (the barrier phases wrap), every epilogue input."""
    sizes = [(256, 256, 256), (129, 130, 64), (384, 512, 1024), (1100, 1300, 512), (257, 129, 320), (2304, 2100, 1344), (4096, 4096, 2048)]
    try:
        for i, (m, n, k) in enumerate(sizes):
            c = Case(m, n, k, L.NVFP4, OUTS[i % 3], -1 if i % 4 == 1 else OUTS[i % 3], L.BF16 if i % 2 else -1, 1.25 if i % 2 else 1.0,
                     1.0 if i % 4 == 1 else 0.0, fa=SW, fb=SW | (PR if i % 3 == 2 else 0))
            h = build_case(c, 900 + i)
            if i in (2, 6):   # dense D (ldd = m): the epilogue stores by TMA
                h["ldd"] = m
                h["Dinit"] = np.frombuffer(b"\xA5" * (m * n * esize(c.dt)), dtype=np.float32 if c.dt == L.FP32 else np.uint16).copy()
            exp = oracle_case(c, h, want_ref=True) if m * n <= 1500 * 1500 else None
            res = []
            for mode in (1, 0):
                assert L.lib.nvfp4a_b200_set_pair(mode) == 0
                got, amax = run_gemm(c, h)
                assert L.lib.nvfp4a_b200_last_route() == 4 and kernel_status() == 0
                if exp is not None:
                    check_bound(c, h, got, amax, exp)
                res.append((got, amax))
            assert np.array_equal(res[0][0], res[1][0]) and res[0][1] == res[1][1], (m, n, k)
    finally:
        L.lib.nvfp4a_b200_set_pair(-1)


def test_w4a4_swapped_orientation_matches_the_bound_and_the_other_orientation():
    """D that TMA can store (16-bit, 16-byte aligned pitch) runs with the tokens on the MMA's M side; the same cases with the
    orientation pinned the other way must agree within the bound too: bias, beta * C, per-row globals on either operand, FP16
    and BF16, tails in m / n / k, padded pitch."""
    sizes = [(128, 128, 256), (136, 40, 64), (200, 300, 192), (1104, 1300, 512), (264, 129, 320), (2304, 520, 1344)]
    try:
        for i, (m, n, k) in enumerate(sizes):
            dt = L.BF16 if i % 2 == 0 else L.FP16
            c = Case(m, n, k, L.NVFP4, dt, -1 if i % 3 == 0 else dt, L.BF16 if i % 2 else -1, 1.25 if i % 2 else 1.0,
                     0.0 if i % 3 == 0 else 0.5, fa=(SW if i % 2 else 0) | (PR if i in (2, 5) else 0), fb=(SW if i < 4 else 0) | (PR if i in (3, 5) else 0))
            h = build_case(c, 950 + i)
            h["ldd"] = m + (8 if i % 2 else 0)
            fill = np.frombuffer(b"\xA5" * (h["ldd"] * n * 2), dtype=np.uint16).copy()
            h["Dinit"] = fill
            exp = oracle_case(c, h, want_ref=True)
            res = []
            for mode in (1, 0):
                assert L.lib.nvfp4a_b200_set_swap(mode) == 0
                got, amax = run_gemm(c, h)
                assert L.lib.nvfp4a_b200_last_route() == 4 and kernel_status() == 0
                check_bound(c, h, got, amax, exp)
                res.append(got)
            print(f"{c}: equal bits between orientations: {np.mean(res[0] == res[1]):.6f}")
    finally:
        L.lib.nvfp4a_b200_set_swap(-1)


def make_image(kind, dfp4, rows, k, ld):
    nbytes = L.lib.nvfp4a_tc_image_bytes(kind, L.NVFP4, rows, k)
    img = torch.full((nbytes + 16,), 0xEE, dtype=torch.uint8, device="cuda")
    t = dfp4.tensor()
    L.check(L.lib.nvfp4a_tc_image(kind, ctypes.byref(t), ld, rows, k, ptr(img), stream()))
    return img, nbytes


@pytest.mark.parametrize("flags", [0, SW, UE])
def test_image_round_trip_and_convert(flags):
    rng = np.random.default_rng(61)
    for rows, k in [(128, 256), (200, 320), (517, 1088), (1, 64)]:
        ld = k + 64
        h = rand_fp4(rng, rows, k, ld=ld, ld_scale=k // 16 + 4, flags=flags, glob=0.375)
        d = DevFp4(h)
        img, nbytes = make_image(L.TC_A16, d, rows, k, ld)
        assert nbytes == ((rows + 127) // 128) * ((k + 255) // 256) * 18432
        img8 = torch.zeros_like(img)
        L.check(L.lib.nvfp4a_tc_image_convert(L.TC_A16, L.TC_A8, ptr(img), rows, k, ptr(img8), stream()))
        built8, _ = make_image(L.TC_A8, d, rows, k, ld)
        torch.cuda.synchronize()
        assert torch.equal(img8[:nbytes], built8[:nbytes])
        assert int(img[nbytes]) == 0xEE  # nothing written past the image
        # back to the plain tensor with linear scales
        out = O.Fp4(rows, k, ld=ld, ld_scale=k // 16 + 4, fill=0xEE)
        dout = DevFp4(out)
        t = dout.tensor()
        L.check(L.lib.nvfp4a_tc_image_to_raw(L.TC_A8, ptr(img8), rows, k, ctypes.byref(t), ld, stream()))
        torch.cuda.synchronize()
        gd, gs = host(dout.data).reshape(rows, ld // 2), host(dout.scales).reshape(rows, k // 16 + 4)
        assert np.array_equal(gd[:, : k // 2], h.data.reshape(rows, ld // 2)[:, : k // 2]) and np.all(gd[:, k // 2:] == 0xEE)
        lin = np.array([[h.scales[O.scale_pos(h.swz, h.ld_scale, k, r, c)] for c in range(k // 16)] for r in range(rows)], np.uint8)
        assert np.array_equal(gs[:, : k // 16], lin) and np.all(gs[:, k // 16:] == 0xEE)


def run_tc(c, h, gemv):
    """nvfp4a_gemm_tc (images of A and B) or nvfp4a_gemv_tc (image of A, B as it is)."""
    dA = DevFp4(h["A"])
    kindA = L.TC_A16 if c.bt == L.BF16 else L.TC_A8
    imgA, _ = make_image(kindA, dA, c.m, c.k, h["lda"])
    keepB, tB = device_b(c, h)
    dD, damax = dev(h["Dinit"]), dev(np.zeros(1, np.float32))
    dC = dev(h["C"]) if h["C"] is not None else None
    dbias = dev(h["bias"]) if h["bias"] is not None else None
    tA = dA.tensor()
    tA.data = imgA.data_ptr()
    tC = tensor(dC, h["ct"]) if dC is not None else None
    tD = tensor(dD, c.dt, amax=damax)
    tbias = tensor(dbias, c.bias) if dbias is not None else None
    cC, cb = (ctypes.byref(tC) if tC is not None else None), (ctypes.byref(tbias) if tbias is not None else None)
    if gemv:
        st = L.lib.nvfp4a_gemv_tc(c.m, c.n, c.k, c.alpha, ctypes.byref(tA), ctypes.byref(tB), h["ldb"], c.beta, cC, h["ldc"], ctypes.byref(tD),
                                  h["ldd"], cb, stream())
    else:
        nb = L.lib.nvfp4a_tc_image_bytes(L.TC_B, c.bt, c.n, c.k)
        imgB = torch.zeros(nb + 16, dtype=torch.uint8, device="cuda")
        L.check(L.lib.nvfp4a_tc_image(L.TC_B, ctypes.byref(tB), h["ldb"], c.n, c.k, ptr(imgB), stream()))
        tBi = L.Tensor.from_buffer_copy(tB)
        tBi.data = imgB.data_ptr()
        ws = torch.zeros(L.lib.nvfp4a_tc_workspace_bytes(), dtype=torch.uint8, device="cuda")
        st = L.lib.nvfp4a_gemm_tc(c.m, c.n, c.k, c.alpha, ctypes.byref(tA), ctypes.byref(tBi), c.beta, cC, h["ldc"], ctypes.byref(tD), h["ldd"], cb,
                                  ptr(ws), stream())
    L.check(st)
    torch.cuda.synchronize()
    return host(dD).view(h["Dinit"].dtype), float(host(damax)[0])


@pytest.mark.parametrize("bt", [L.NVFP4, L.INT8, L.BF16])
def test_image_entries_gemm_tc_and_gemv_tc(bt):
    sizes = [(37, 45, 128), (200, 300, 192), (257, 129, 256), (1100, 1300, 512), (300, 3, 1024), (1000, 8, 576), (77, 1, 128)]
    for i, (m, n, k) in enumerate(sizes):
        for fa in (0, SW, AM | PR):
            c = Case(m, n, k, bt, OUTS[i % 3], -1 if i % 4 == 1 else OUTS[i % 3], L.BF16 if i % 2 else -1, 1.25 if i % 2 else 1.0,
                     1.0 if i % 4 == 1 else 0.0, fa=fa, fb=SW if (bt == L.NVFP4 and i % 2) else 0)
            h = build_case(c, 800 + i)
            exp = oracle_case(c, h, want_ref=True)
            got, amax = run_tc(c, h, gemv=False)
            check_bound(c, h, got, amax, exp)
            if n <= 8:
                got, amax = run_tc(c, h, gemv=True)
                check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


def test_w4a4_4096_cubed_against_block_sum_oracle_sample():
    """The W4A4 GEMM 4096^3 at full size: BF16 N(0,1) operands quantized to NVFP4 (linear E4M3 scales, FP32 decode-factor
    globals), D BF16 column major.  The oracle checks a slab of 64 columns x all rows within the bound and reports the share
    within 1 BF16 ulp; linearity (alpha = 2 doubles every output exactly) is checked on the whole matrix."""
    m = n = k = 4096
    rng = np.random.default_rng(2)
    hs = []
    for seed in (2, 3):
        x = np.random.default_rng(seed).standard_normal((m, k), dtype=np.float32)
        x = O.to_f32(O.from_f32(x, L.BF16), L.BF16).reshape(m, k)
        g = np.array([np.abs(x).max() / (6.0 * 448.0)], np.float32)
        h = O.Fp4(m, k, glob=g)
        O.quantize(x, h)
        hs.append(h)
    A, B = hs
    dA, dB = DevFp4(A), DevFp4(B)
    outs = []
    for alpha in (1.0, 2.0):
        dD, damax = torch.zeros(m * n, dtype=torch.int16, device="cuda"), dev(np.zeros(1, np.float32))
        tA, tB, tD = dA.tensor(), dB.tensor(), tensor(dD, L.BF16, amax=damax)
        L.check(L.lib.nvfp4a_gemm(m, n, k, alpha, ctypes.byref(tA), k, ctypes.byref(tB), k, 0.0, None, 0, ctypes.byref(tD), m, None, stream()))
        torch.cuda.synchronize()
        outs.append((O.to_f32(host(dD).view(np.uint16), L.BF16).reshape(n, m), float(host(damax)[0])))
    assert kernel_status() == 0
    (d1, a1), (d2, a2) = outs
    assert np.array_equal(d2, 2.0 * d1) and a2 == 2.0 * a1
    # slab: columns 1000..1063
    j0, nj = 1000, 64
    Bs = O.Fp4(nj, k, glob=B.glob)
    Bs.data[:] = B.data.reshape(n, k // 2)[j0:j0 + nj].reshape(-1)
    Bs.scales[:] = B.scales.reshape(n, k // 16)[j0:j0 + nj].reshape(-1)
    exp = O.gemm(m, nj, k, A, Bs, D_dtype=L.BF16, want_ref=True)
    got = d1[j0:j0 + nj].astype(np.float64)
    assert np.all(np.abs(got - exp["ref64"]) <= exp["bound"])
    exact = O.to_f32(exp["D"], L.BF16).reshape(nj, m).astype(np.float64)
    share = frac_within_1ulp_bf16(got, exact)
    print(f"4096^3 W4A4: share of outputs within 1 BF16 ulp of the block-sum oracle = {share:.6f}; equal bits = {np.mean(got == exact):.6f}")
    assert share >= 0.999
    assert abs(a1 - np.abs(d1).max()) <= 2.0 ** -7 * a1


@pytest.mark.parametrize("bt", [L.INT8, L.NVFP4])
def test_gemv_with_block_scaled_activations_uses_the_dp4a_kernel(bt):
    """n <= 8 with INT8 / NVFP4 activations: exact integer block sums by DP4A (route 6), FP32 accumulation in the kernel's order."""
    for i, (m, n, k) in enumerate([(70, 1, 64), (515, 3, 1024), (4096, 8, 4096), (33, 5, 2304)]):
        for fa in (0, SW, AM | PR):
            c = Case(m, n, k, bt, OUTS[i % 3], OUTS[i % 3] if i % 2 else -1, L.FP32 if i % 2 else -1, 0.75, 1.0 if not i % 2 else 0.0, fa=fa,
                     fb=(SW | AM) if (bt == L.NVFP4 and i % 2) else 0)
            h = build_case(c, 1200 + i)
            exp = oracle_case(c, h, want_ref=True)
            got, amax = run_gemm(c, h)
            assert L.lib.nvfp4a_b200_last_route() == 6, c
            check_bound(c, h, got, amax, exp)


@pytest.mark.parametrize("bt", [L.INT8, L.NVFP4])
@pytest.mark.parametrize("layout", ["image", "swizzled", "linear"])
def test_blocked_gemv_at_the_edges_of_its_tiles_and_k_ranges(bt, layout):
    """Units of 128 and 256 values with remainders, one to eight warps per group of 16 rows, CTAs of 4, 8 and 16 warps (the last also because
    the activations fill shared memory), more tiles than CTAs, odd n; negative block scales; and a row's bits do not depend on the matrix around it."""
    for i, (m, n, k) in enumerate([(33, 1, 64), (77, 2, 192), (200, 3, 320), (130, 5, 576), (4900, 4, 128), (100, 7, 1088), (2500, 8, 2112), (5000, 2, 1344), (50, 8, 14400),
                                   (9700, 6, 256)]):
        c = Case(m, n, k, bt, L.FP32, -1, -1, 1.0, 0.0, fa=SW if layout == "swizzled" else 0)
        h = build_case(c, 7300 + i)
        flip = np.random.default_rng(i).integers(0, 4, h["A"].scales.size) == 0
        h["A"].scales[flip & (h["A"].scales != 0)] |= 0x80
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_tc(c, h, gemv=True) if layout == "image" else run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == 6, c
        check_bound(c, h, got, amax, exp)
        if layout == "linear" and m > 160:
            A = h["A"]
            top = O.Fp4(160, k, ld=A.ld, ld_scale=A.ld_scale, flags=A.flags, scale_max=A.scale_max, glob=0.0)
            top.data[:], top.scales[:], top.glob[:] = A.data[:160 * A.ld // 2], A.scales[:160 * A.ld_scale], A.glob
            ct, ht = Case(160, n, k, bt, L.FP32, -1, -1, 1.0, 0.0), dict(h, A=top)
            got_top, _ = run_gemm(ct, ht)
            assert np.array_equal(values(got_top, ct, ht), values(got, c, h)[:, :160])


@pytest.mark.parametrize("m,n,k", [(300, 8, 1024), (9700, 5, 1024), (130, 8, 1984), (5000, 3, 1536), (70, 6, 2048), (40, 8, 960), (4800, 7, 64), (64, 4, 2112)])
def test_blocked_gemv_where_its_units_change(m, n, k):
    """One 128-value unit per warp (k <= 1024: pairs of vectors in a loop), two of them (k < 2048), 256-value units from there on: within the bound,
    and a vector's bits are those of the vector alone."""
    c = Case(m, n, k, L.INT8, L.FP32, -1, L.BF16, 1.0, 0.0)
    h = build_case(c, 7500 + m)
    got, amax = run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == 6
    check_bound(c, h, got, amax, oracle_case(c, h, want_ref=True))
    B = h["B"]
    one = O.Q8(1, k, ld=B.ld, ld_scale=B.ld_scale)
    one.data[:], one.scales[:] = B.data[:B.ld], B.scales[:B.ld_scale]
    one.glob = B.glob
    c1, h1 = Case(m, 1, k, L.INT8, L.FP32, -1, L.BF16, 1.0, 0.0), dict(h, B=one, Dinit=h["Dinit"][:h["ldd"]])
    got1, _ = run_gemm(c1, h1)
    assert np.array_equal(values(got1, c1, h1)[0], values(got, c, h)[0])


def test_w4a8_dp4a_gemm_is_bit_exact_in_the_tiled_order():
    """INT8 activations, n > 8, with the tensor-core W4A8 GEMM switched off (nvfp4a_b200_set_route(3)): the DP4A GEMM (route 7)
    sums blocks in the reference's tiled order, so D and amax equal the oracle's bit for bit; tails in m and n, padded leading
    dimensions, every output type, bias, beta, alpha.  The default route on the same inputs stays within the bound."""
    old = L.lib.nvfp4a_b200_set_route(3)
    try:
        for i, (m, n, k) in enumerate([(128, 128, 64), (130, 9, 128), (517, 300, 1024), (1000, 129, 576), (64, 2048, 256)]):
            for fa in (0, SW, AM | PR):
                c = Case(m, n, k, L.INT8, OUTS[i % 3], OUTS[(i + 1) % 3] if i % 2 else -1, L.BF16 if i % 2 else -1, 1.25, 0.5 if i % 2 else 1.0, fa=fa)
                h = build_case(c, 1300 + i)
                exp = oracle_case(c, h, want_ref=True)
                got, amax = run_gemm(c, h)
                assert L.lib.nvfp4a_b200_last_route() == 7, c
                assert np.array_equal(got.view(np.uint8), exp["D"].view(np.uint8)), c
                assert amax == exp["amax"], c
                L.lib.nvfp4a_b200_set_route(0)
                got, amax = run_gemm(c, h)
                assert L.lib.nvfp4a_b200_last_route() == (8 if m >= 128 and n >= 64 else 7), c
                check_bound(c, h, got, amax, exp)
                L.lib.nvfp4a_b200_set_route(3)
    finally:
        L.lib.nvfp4a_b200_set_route(old)


def test_gemm_dual_forward_dgrad_and_wgrad():
    """nvfp4a_gemm_dual picks, per operand, the half whose blocks run along k (reference include/nvfp4effma.h:97-103):
    forward Y = X W^T (trans 0, 0), dgrad dX = dY W (A = W with trans_a = 1: the column half of the [k][m] weight),
    wgrad dW = dY^T X (both column halves).  Each must equal nvfp4a_gemm on the chosen halves bit for bit (the call only
    forwards) and lie within the bound of the exact definition; a missing half is INVALID_VALUE."""
    T, I, Ou = 256, 384, 192
    rng = np.random.default_rng(77)

    def dual(x):
        rows, cols = x.shape
        row = O.Fp4(rows, cols, flags=O.GLOBAL_AMAX, glob=0.0)
        col = O.Fp4(cols, rows, flags=O.GLOBAL_AMAX, glob=0.0)
        O.quantize(x, row, tile=16, compute_amax=True)
        O.quantize(x, col, transposed=True, tile=16, compute_amax=True)
        dr, dc = DevFp4(row), DevFp4(col)
        return row, col, dr, dc, L.DualTensor(dr.tensor(), dc.tensor(), cols, rows)

    W = dual(rng.standard_normal((Ou, I)).astype(np.float32))
    X = dual(rng.standard_normal((T, I)).astype(np.float32))
    dY = dual(rng.standard_normal((T, Ou)).astype(np.float32))
    cases = [("forward", Ou, T, I, W, 0, X, 0), ("dgrad", I, T, Ou, W, 1, dY, 0), ("wgrad", I, Ou, T, X, 1, dY, 1)]
    for name, m, n, k, A, ta, B, tb in cases:
        hA, hB = A[1 if ta else 0], B[1 if tb else 0]
        dA, dB = A[3 if ta else 2], B[3 if tb else 2]
        outs = []
        for use_dual in (True, False):
            dD, damax = torch.zeros(m * n, dtype=torch.float32, device="cuda"), dev(np.zeros(1, np.float32))
            tD = tensor(dD, L.FP32, amax=damax)
            if use_dual:
                st = L.lib.nvfp4a_gemm_dual(m, n, k, 1.0, ctypes.byref(A[4]), ta, ctypes.byref(B[4]), tb, 0.0, None, 0, ctypes.byref(tD), m, None, stream())
            else:
                tA, tB = dA.tensor(), dB.tensor()
                st = L.lib.nvfp4a_gemm(m, n, k, 1.0, ctypes.byref(tA), hA.ld, ctypes.byref(tB), hB.ld, 0.0, None, 0, ctypes.byref(tD), m, None, stream())
            assert st == 0, (name, L.last_error())
            torch.cuda.synchronize()
            outs.append((host(dD).copy(), float(host(damax)[0])))
        assert np.array_equal(outs[0][0], outs[1][0]) and outs[0][1] == outs[1][1], name
        exp = O.gemm(m, n, k, hA, hB, D_dtype=L.FP32, want_ref=True)
        assert np.all(np.abs(outs[0][0].reshape(n, m).astype(np.float64) - exp["ref64"]) <= exp["bound"]), name
    # 16 x 16 tiles: the column half of W decodes to the transpose of its row half, so dgrad really multiplies by W
    assert np.array_equal(O.dequantize(W[1])[0], O.dequantize(W[0])[0].T)
    lone = L.DualTensor(W[2].tensor(), L.Tensor(), I, 0)
    dD = torch.zeros(I * T, dtype=torch.float32, device="cuda")
    tD = tensor(dD, L.FP32)
    st = L.lib.nvfp4a_gemm_dual(I, T, Ou, 1.0, ctypes.byref(lone), 1, ctypes.byref(dY[4]), 0, 0.0, None, 0, ctypes.byref(tD), I, None, stream())
    assert st == L.INVALID_VALUE and "column" in L.last_error()
    assert kernel_status() == 0


@pytest.mark.parametrize("bt", [L.INT8, L.NVFP4, L.BF16, L.FP32])
def test_grouped_gemm_gives_every_group_the_bytes_of_its_own_gemm(bt):
    """nvfp4a_gemm_grouped (reference include/nvfp4effma.h:104-116): three experts of 40 weight rows stacked in A, the row counts
    of B per expert in a device array (one expert empty, rows past seg[groups] left alone); every group's rows of D are the
    bytes the oracle's tiled order gives for that group's own GEMM -- bias, beta * C and per-row globals of the stacked A included."""
    for groups, m, k, rows, seg in ((3, 40, 192, 45, [0, 19, 19, 41]), (3, 200, 256, 300, [0, 130, 130, 290])):
        _grouped_case(bt, groups, m, k, rows, np.array(seg, np.int32))


def _grouped_case(bt, groups, m, k, rows, seg):
    from util import rand_fp4, rand_q8
    rng = np.random.default_rng(4100 + bt + m)
    lda, ldb, ldd = k + 64, k + 64, m + 8
    A = rand_fp4(rng, groups * m, k, ld=lda, ld_scale=k // 16 + 4, flags=O.PER_ROW, glob=0.375)
    if bt == L.NVFP4:
        B = rand_fp4(rng, rows, k, ld=ldb, ld_scale=k // 16 + 8, flags=O.PER_ROW, glob=1.75)
    elif bt == L.INT8:
        B = rand_q8(rng, rows, k, ld=ldb, ld_scale=k // 16 + 8)
    else:
        B = O.Dense(bt, rand_dense(rng, bt, ldb * rows, 2.0), ldb)
    bias = rand_dense(rng, L.BF16, groups * m, 3.0)
    Dinit = rand_dense(rng, L.BF16, ldd * rows, 4.0)     # D is also C (beta != 0)
    alpha, beta = 1.25, 0.5

    def rows_of(t, lo, hi):
        """The sub-matrix of rows [lo, hi) of a host operand (linear scales: whole rows of every array)."""
        if isinstance(t, O.Dense):
            return O.Dense(t.dtype, t.raw[lo * t.ld: hi * t.ld], t.ld)
        if isinstance(t, O.Q8):
            q = O.Q8(hi - lo, t.cols, ld=t.ld, ld_scale=t.ld_scale)
            q.data[:], q.scales[:] = t.data[lo * t.ld: hi * t.ld], t.scales[lo * t.ld_scale: hi * t.ld_scale]
            return q
        q = O.Fp4(hi - lo, t.cols, ld=t.ld, ld_scale=t.ld_scale, flags=t.flags, scale_max=t.scale_max, glob=0.0)
        q.data[:], q.scales[:], q.glob[:] = t.data[lo * t.ld // 2: hi * t.ld // 2], t.scales[lo * t.ld_scale: hi * t.ld_scale], t.glob[lo:hi]
        return q

    want = Dinit.copy()
    amax = 0.0
    for q in range(groups):
        lo, hi = int(seg[q]), int(seg[q + 1])
        if hi == lo:
            continue
        exp = O.gemm(m, hi - lo, k, rows_of(A, q * m, (q + 1) * m), rows_of(B, lo, hi), D_dtype=L.BF16, alpha=alpha, beta=beta,
                     C=Dinit[lo * ldd: hi * ldd], C_dtype=L.BF16, ldc=ldd, ldd=ldd, bias=bias[q * m: (q + 1) * m], bias_dtype=L.BF16,
                     lda=lda, ldb=ldb, D_init=Dinit[lo * ldd: hi * ldd])
        want[lo * ldd: hi * ldd] = exp["D"]
        amax = max(amax, exp["amax"])

    dA = DevFp4(A)
    if bt == L.NVFP4:
        keep = DevFp4(B); tB = keep.tensor()
    elif bt == L.INT8:
        keep = (dev(B.data), dev(B.scales)); tB = tensor(keep[0], L.INT8, keep[1], B.ld_scale)
    else:
        keep = dev(B.raw); tB = tensor(keep, bt)
    dD, damax, dbias, dseg = dev(Dinit), dev(np.zeros(1, np.float32)), dev(bias), dev(seg)
    tA, tD, tbias = dA.tensor(), tensor(dD, L.BF16, amax=damax), tensor(dbias, L.BF16)
    st = L.lib.nvfp4a_gemm_grouped(groups, m, k, rows, alpha, ctypes.byref(tA), lda, ctypes.byref(tB), ldb, beta, ctypes.byref(tD), ldd,
                                   ctypes.byref(tD), ldd, ctypes.byref(tbias), ctypes.c_void_p(dseg.data_ptr()), stream())
    assert st == 0, L.lib.nvfp4a_last_error()
    assert L.lib.nvfp4a_b200_last_route() == (7 if bt == L.INT8 else 1)   # INT8: the 128 x 128 DP4A kernel, else the generic one
    torch.cuda.synchronize()
    got = host(dD).view(np.uint16)
    assert np.array_equal(got, want)          # groups bit for bit; padding, the empty group and the rows past seg[groups] untouched
    assert float(host(damax)[0]) == amax


def test_w4a8_on_the_tensor_cores_and_the_exact_route_beside_it():
    """INT8 activations, more than 8 tokens: by default the W4A16 tcgen05 kernel on the activations split into three BF16 planes
    (route 8; within the FP32 accumulation bound of the exact definition: one rounding of q * s_b per activation); with
    nvfp4a_b200_set_route(3) the DP4A kernel (route 7), bit-identical to the reference's tiled order.  Tails in m, n and k, padded
    leading dimensions, bias, beta * C, every output type."""
    sizes = [(128, 64, 64), (300, 200, 320), (1000, 77, 192), (2048, 512, 1024), (515, 130, 4160)]
    for i, (m, n, k) in enumerate(sizes):
        c = Case(m, n, k, L.INT8, OUTS[i % 3], OUTS[i % 3] if i % 2 else -1, L.BF16 if i % 3 == 1 else -1, 1.25 if i % 2 else 1.0, 0.5 if i % 2 else 0.0)
        h = build_case(c, 4300 + i)
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == 8, c
        check_bound(c, h, got, amax, exp)
        old = L.lib.nvfp4a_b200_set_route(3)
        try:
            got, amax = run_gemm(c, h)
            assert L.lib.nvfp4a_b200_last_route() == 7, c
        finally:
            L.lib.nvfp4a_b200_set_route(old)
        assert np.array_equal(got, exp["D"]) and amax == exp["amax"], c
    assert kernel_status() == 0
    # the planes' pool: trimmed, refilled by the next call; and the whole call (allocation, conversion, GEMM, free) inside a CUDA graph
    assert L.lib.nvfp4a_b200_trim_scratch() == 0
    c = Case(300, 200, 320, L.INT8, L.BF16, -1, -1, 1.0, 0.0)
    h = build_case(c, 4390)
    want, _ = run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == 8
    dA = DevFp4(h["A"])
    keepB, tB = device_b(c, h)
    dD = dev(h["Dinit"])
    tA, tD = dA.tensor(), tensor(dD, c.dt)

    def call():
        st = L.lib.nvfp4a_gemm(c.m, c.n, c.k, c.alpha, ctypes.byref(tA), h["lda"], ctypes.byref(tB), h["ldb"], 0.0, None, 0, ctypes.byref(tD), h["ldd"],
                               None, stream())
        assert st == 0, L.lib.nvfp4a_last_error()

    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    fresh = dev(h["Dinit"])
    for _ in range(3):
        dD.copy_(fresh)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(host(dD).view(np.uint16), want.view(np.uint16))
    assert kernel_status() == 0


def test_gemv_long_reductions_in_sections():
    """The mma.sync GEMV cuts k >= 8192 into 2 and k >= 12288 into 4 sections; a matrix of few rows gives each section to a
    CTA of a cluster (partial sums through distributed shared memory), a taller one walks them in one CTA.  Both against the
    float64 reference within the bound, images and plain operands, 1 to 8 activation vectors, tails in m; and the two forms
    agree bit for bit on the rows they share (a row's sum depends on k alone)."""
    old = L.lib.nvfp4a_b200_set_route(2)   # keep the FP4 tensor-core GEMV out of it
    try:
        for i, (m, n, k) in enumerate([(300, 1, 8192), (130, 5, 14336), (1300, 3, 14336), (77, 8, 12288), (2500, 2, 8192)]):
            c = Case(m, n, k, L.BF16, OUTS[i % 3], -1, L.BF16 if i % 2 else -1, 1.25 if i % 2 else 1.0, 0.0, fa=SW if i % 2 else 0)
            h = build_case(c, 4700 + i)
            exp = oracle_case(c, h, want_ref=True)
            got, amax = run_gemm(c, h)
            assert L.lib.nvfp4a_b200_last_route() == 2, c
            check_bound(c, h, got, amax, exp)
            got_tc, amax_tc = run_tc(c, h, gemv=True)
            assert L.lib.nvfp4a_b200_last_route() == 2, c
            check_bound(c, h, got_tc, amax_tc, exp)
        # the same rows as part of a short matrix (cluster per slice) and of a tall one (one CTA per slice): identical bytes
        k = 14336
        tall = Case(1600, 2, k, L.BF16, L.FP32, -1, -1, 1.0, 0.0)
        h = build_case(tall, 4750)
        got_tall, _ = run_gemm(tall, h)
        short = Case(160, 2, k, L.BF16, L.FP32, -1, -1, 1.0, 0.0)
        hs = dict(h)
        A = h["A"]
        As = O.Fp4(160, k, ld=A.ld, ld_scale=A.ld_scale, flags=A.flags, scale_max=A.scale_max, glob=0.0)
        As.data[:], As.scales[:], As.glob[:] = A.data[:160 * A.ld // 2], A.scales[:160 * A.ld_scale], A.glob
        hs["A"] = As
        got_short, _ = run_gemm(short, hs)
        a = values(got_tall, tall, h)[:, :160]
        b = values(got_short, short, hs)
        assert np.array_equal(a, b)
    finally:
        L.lib.nvfp4a_b200_set_route(old)
    assert kernel_status() == 0


def test_blocked_gemv_with_sixteen_and_thirty_two_rows_per_cta():
    """The DP4A GEMV for INT8 / NVFP4 activations gives a CTA 16 rows while the matrix would leave SMs without a CTA and 32 rows
    from about 4700 rows up: both against the float64 reference within the bound, and bit for bit against each other on shared rows."""
    for bt in (L.INT8, L.NVFP4):
        outs = {}
        for m in (4800, 160):
            c = Case(m, 3, 320, bt, L.FP32, -1, -1, 1.0, 0.0)
            h = build_case(c, 4800 + bt)          # the same seed: the short matrix is not a prefix of the tall one, so each is checked alone
            exp = oracle_case(c, h, want_ref=True)
            got, amax = run_gemm(c, h)
            assert L.lib.nvfp4a_b200_last_route() == 6, c
            check_bound(c, h, got, amax, exp)
            outs[m] = (c, h, got)
        # shared rows: the first 160 rows of the tall matrix as a matrix of their own (16 rows per CTA)
        c, h, got_tall = outs[4800]
        A = h["A"]
        As = O.Fp4(160, c.k, ld=A.ld, ld_scale=A.ld_scale, flags=A.flags, scale_max=A.scale_max, glob=0.0)
        As.data[:], As.scales[:], As.glob[:] = A.data[:160 * A.ld // 2], A.scales[:160 * A.ld_scale], A.glob
        cs = Case(160, 3, 320, bt, L.FP32, -1, -1, 1.0, 0.0)
        hs = dict(h, A=As)
        got_short, _ = run_gemm(cs, hs)
        assert np.array_equal(values(got_tall, c, h)[:, :160], values(got_short, cs, hs))


@pytest.mark.parametrize("m,n,k", [(1, 1, 64), (128, 8, 192), (129, 9, 320), (257, 63, 256), (300, 65, 1088), (520, 257, 576), (1100, 700, 512)])
def test_fp16_activations_on_the_tensor_cores(m, n, k):
    """FP16 activations with a 16-bit D run on the tcgen05 kernel (route 5; weights expanded to exact FP16) for every n; an FP32 D or
    UE5M3 scales keep the CUDA-core kernel.  Edges of the 256-row / 64-token tiles and of the 256-value slots of k, every epilogue input."""
    for i, (dt, fa, route) in enumerate([(L.FP16, 0, 5), (L.BF16, SW, 5), (L.FP16, AM | PR, 5), (L.FP32, 0, 1), (L.FP16, UE, 1)]):
        c = Case(m, n, k, L.FP16, dt, dt if i % 2 else -1, L.BF16 if i % 2 else -1, 1.25 if i % 2 else 1.0, 0.5 if i % 2 else 0.0, fa=fa)
        h = build_case(c, 5200 + 10 * m + i)
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == route, c
        check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


def test_w4a16_gemm_gives_the_same_bytes_every_time():
    """120 launches of a large problem with an FP32 D (whose stores queue up in the load / store unit next to the weight expansion's reads
    of shared memory): a slot of weights handed back while reads of it are still queued shows as a few wrong rows in one launch of
    fifteen.  Every launch has to give the first one's bytes."""
    m, n, k = 28672, 2048, 4096
    gen = torch.Generator(device="cuda").manual_seed(9)
    img = torch.randint(0, 256, (L.lib.nvfp4a_tc_image_bytes(L.TC_A16, L.NVFP4, m, k),), generator=gen, device="cuda", dtype=torch.uint8)
    img.view(-1, 18432)[:, 16384:] = torch.randint(0x30, 0x48, (img.numel() // 18432, 2048), generator=gen, device="cuda", dtype=torch.uint8)
    x = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
    ws = torch.zeros(L.lib.nvfp4a_tc_workspace_bytes(), dtype=torch.uint8, device="cuda")
    D = torch.empty(n, m, dtype=torch.float32, device="cuda")
    ta, tb, td = tensor(img, L.NVFP4), tensor(x, L.BF16), tensor(D, L.FP32)
    first, differs = None, []
    for _ in range(120):
        L.check(L.lib.nvfp4a_gemm_tc(m, n, k, 1.0, ctypes.byref(ta), ctypes.byref(tb), 0.0, None, 0, ctypes.byref(td), m, None, ptr(ws), stream()))
        if first is None:
            assert L.lib.nvfp4a_b200_last_route() == 5
            first = D.clone()
        else:
            differs.append((D != first).any())
    assert not bool(torch.stack(differs).any())
    assert kernel_status() == 0


@pytest.mark.parametrize("k", [512, 576, 1024, 4096])
@pytest.mark.parametrize("kind", ["fp16", "grouped_int8"])
def test_long_sums_on_the_tensor_cores_are_joined_in_fp32(kind, k):
    """The tensor cores truncate the running sum at every instruction, so that one chain over k = 4096 loses about 1e-5 of a sum of positive
    terms, always downwards; the ordered CUDA-core kernels lose a few 1e-7.  FP16 activations and INT8 groups therefore sum segments of 256
    values (128 below k = 1024).  The largest result before its rounding (amax) against 64 bits: at most one unit in the last place (2^-23)
    of the segment's running sum, on average half of the segment's, for each of its 16 instructions, as much again for the FP32
    additions of up to 16 segments, four more for the small terms, scales and the quantities rounded on the way."""
    m, n = 300, 70
    gen = torch.Generator(device="cuda").manual_seed(k)
    w = torch.randint(1, 8, (m, k), generator=gen, device="cuda", dtype=torch.uint8)             # positive codes
    ws = torch.randint(0x28, 0x48, (m, k // 16), generator=gen, device="cuda", dtype=torch.uint8)
    packed = (w[:, 0::2] | (w[:, 1::2] << 4)).contiguous()
    W = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device="cuda")[w.long()]
    W = (W.view(m, k // 16, 16) * ws.view(torch.float8_e4m3fn).double().unsqueeze(-1)).view(m, k)
    ta, amax = tensor(packed, L.NVFP4, ws, k // 16), torch.zeros(1, dtype=torch.float32, device="cuda")
    D = torch.zeros(n, m, dtype=torch.bfloat16, device="cuda")
    td = tensor(D, L.BF16, amax=amax)
    if kind == "fp16":
        x = (torch.rand(n, k, generator=gen, device="cuda") + 0.01).half()
        X, tb = x.double(), tensor(x, L.FP16)
        L.check(L.lib.nvfp4a_gemm(m, n, k, 1.0, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), m, None, stream()))
        assert L.lib.nvfp4a_b200_last_route() == 5
    else:
        x, xs = torch.randint(1, 128, (n, k), generator=gen, device="cuda", dtype=torch.int8), torch.rand(n, k // 16, generator=gen, device="cuda") + 0.01
        X = (x.double().view(n, k // 16, 16) * xs.double().unsqueeze(-1)).view(n, k)
        tb, seg = tensor(x, L.INT8, xs, k // 16), torch.tensor([0, n], dtype=torch.int32, device="cuda")
        L.check(L.lib.nvfp4a_gemm_grouped(1, m, k, n, 1.0, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), m, None,
                                          ctypes.c_void_p(seg.data_ptr()), stream()))
        assert L.lib.nvfp4a_b200_last_route() == 8
    want = X @ W.t()
    assert abs(float(amax.double()) / float(want.max()) - 1.0) <= (16 + 16 + 4) * 2.0 ** -24
    assert torch.allclose(D.double(), want, rtol=2.0 ** -8, atol=0.0)
    assert kernel_status() == 0


@pytest.mark.parametrize("case", ["odd_row_tiles", "swiglu", "grouped"])
def test_tma_stored_tiles_equal_plain_stores_on_every_launch(case):
    """A 16-bit D leaves through two alternating staging tiles and TMA stores.  Short reductions (the next tile's results arrive soon), several
    tiles per CTA pair and turns that store nothing by TMA -- an odd number of 128-row tiles, the last tokens of a group -- against the
    same launch with a leading dimension that TMA cannot store (plain stores, no staging tile in flight), 60 launches each."""
    m, k = (2048, 512) if case == "grouped" else (33 * 128, 64)
    gen = torch.Generator(device="cuda").manual_seed(11)
    ints = lambda lo, hi, shape: torch.randint(lo, hi, shape, generator=gen, device="cuda", dtype=torch.uint8)
    if case == "grouped":
        sizes = torch.randint(1, 250, (40,), generator=torch.Generator().manual_seed(3))
        seg = torch.cat([torch.zeros(1, dtype=torch.int64), sizes.cumsum(0)]).to(torch.int32).cuda()
        groups, n = 40, int(sizes.sum())
        x, xs = ints(0, 256, (n, k)).view(torch.int8), torch.rand(n, k // 16, generator=gen, device="cuda") + 0.5
        tb = tensor(x, L.INT8, xs, k // 16)
    else:
        groups, n = 1, 2048
        x = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
        tb = tensor(x, L.BF16)
    w, ws = ints(0, 256, (groups * m, k // 2)), ints(0x30, 0x48, (groups * m, k // 16))
    ta = tensor(w, L.NVFP4, ws, k // 16)
    mo = m // 2 if case == "swiglu" else m
    ex = L.Epilogue()
    ex.swiglu = int(case == "swiglu")

    def launch(out):
        td, ld = tensor(out, L.BF16), out.stride(0)
        if case == "grouped":
            return L.lib.nvfp4a_gemm_grouped(groups, m, k, n, 2.0 ** -10, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), ld, None,
                                             ctypes.c_void_p(seg.data_ptr()), stream())
        return L.lib.nvfp4a_gemm_ex(m, n, k, 0.25, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), ld, None, ctypes.byref(ex), stream())

    plain, out = torch.zeros(n, mo + 1, dtype=torch.bfloat16, device="cuda"), torch.zeros(n, mo, dtype=torch.bfloat16, device="cuda")
    L.check(launch(plain))
    assert L.lib.nvfp4a_b200_last_route() == (8 if case == "grouped" else 5)
    assert bool(torch.isfinite(plain.float()).all()) and bool(plain.any())
    want, differs = plain[:, :mo].contiguous().view(torch.int16), []
    for _ in range(60):
        out.zero_()
        L.check(launch(out))
        differs.append((out.view(torch.int16) != want).any())
    assert not bool(torch.stack(differs).any())
    assert kernel_status() == 0


@pytest.mark.parametrize("seg,m,k", [([0, 1, 1, 64], 128, 512), ([0, 65, 130, 131], 130, 576), ([0, 0, 0, 257], 300, 1088), ([3, 3, 100, 400], 257, 512)])
def test_grouped_w4a8_on_the_tensor_cores(seg, m, k):
    """INT8 activations, 16-bit D, k >= 512: nvfp4a_gemm_grouped runs the tcgen05 kernel (route 8), every group within the bound of its own
    GEMM; nvfp4a_b200_set_route(3) gives the DP4A kernel's bytes.  Empty groups, groups of one token, partial 64-token tiles, row tiles
    that cross into the next group's weight, rows before seg[0] and past seg[groups] left alone, per-row globals, bias, beta * C."""
    groups, rows = len(seg) - 1, seg[-1] + 5
    rng = np.random.default_rng(6100 + m + k)
    lda, ldb, ldd = k + 64, k + 64, m + 8
    A = rand_fp4(rng, groups * m, k, ld=lda, ld_scale=k // 16 + 4, flags=O.PER_ROW, glob=0.375)
    B = rand_q8(rng, rows, k, ld=ldb, ld_scale=k // 16 + 8)
    bias = rand_dense(rng, L.BF16, groups * m, 3.0)
    dA, dB, dS, dbias, dseg = DevFp4(A), dev(B.data), dev(B.scales), dev(bias), dev(np.array(seg, np.int32))
    for dt, pad, alpha, beta in ((L.BF16, 8, 1.25, 0.5), (L.FP16, 3, 0.0078125, 0.0)):   # ldd = m + 3: D that TMA cannot store; FP16: stays in range
        ldd = m + pad
        Dinit = rand_dense(rng, dt, ldd * rows, 4.0)
        for route in (0, 3):
            old = L.lib.nvfp4a_b200_set_route(route)
            try:
                dD, damax = dev(Dinit), dev(np.zeros(1, np.float32))
                tA, tB, tD, tb = dA.tensor(), tensor(dB, L.INT8, dS, B.ld_scale), tensor(dD, dt, amax=damax), tensor(dbias, L.BF16)
                st = L.lib.nvfp4a_gemm_grouped(groups, m, k, rows, alpha, ctypes.byref(tA), lda, ctypes.byref(tB), ldb, beta, ctypes.byref(tD), ldd,
                                               ctypes.byref(tD), ldd, ctypes.byref(tb), ctypes.c_void_p(dseg.data_ptr()), stream())
                assert st == 0, L.lib.nvfp4a_last_error()
                assert L.lib.nvfp4a_b200_last_route() == (8 if route == 0 else 7)
            finally:
                L.lib.nvfp4a_b200_set_route(old)
            torch.cuda.synchronize()
            raw = host(dD).view(np.uint16).reshape(rows, ldd)
            init = Dinit.reshape(rows, ldd)
            assert np.array_equal(raw[:, m:], init[:, m:]) and np.array_equal(raw[seg[-1]:], init[seg[-1]:]) and np.array_equal(raw[:seg[0]], init[:seg[0]])
            for q in range(groups):
                lo, hi = seg[q], seg[q + 1]
                if hi == lo:
                    continue
                Aq = O.Fp4(m, k, ld=lda, ld_scale=A.ld_scale, flags=A.flags, scale_max=A.scale_max, glob=0.0)
                Aq.data[:], Aq.scales[:] = A.data[q * m * lda // 2:(q + 1) * m * lda // 2], A.scales[q * m * A.ld_scale:(q + 1) * m * A.ld_scale]
                Aq.glob[:] = A.glob[q * m:(q + 1) * m]
                Bq = O.Q8(hi - lo, k, ld=ldb, ld_scale=B.ld_scale)
                Bq.data[:], Bq.scales[:] = B.data[lo * ldb:hi * ldb], B.scales[lo * B.ld_scale:hi * B.ld_scale]
                exp = O.gemm(m, hi - lo, k, Aq, Bq, D_dtype=dt, alpha=alpha, beta=beta, C=Dinit[lo * ldd:hi * ldd], C_dtype=dt, ldc=ldd, ldd=ldd,
                             bias=bias[q * m:(q + 1) * m], bias_dtype=L.BF16, lda=lda, ldb=ldb, D_init=Dinit[lo * ldd:hi * ldd], want_ref=True)
                got = O.to_f32(np.ascontiguousarray(raw[lo:hi, :m]).reshape(-1), dt).reshape(hi - lo, m).astype(np.float64)
                if route == 3:
                    assert np.array_equal(raw[lo:hi], exp["D"].reshape(hi - lo, ldd))
                else:
                    assert np.all(np.abs(got - exp["ref64"]) <= exp["bound"]), (q, np.max(np.abs(got - exp["ref64"]) / exp["bound"]))
    assert kernel_status() == 0


@pytest.mark.parametrize("bt", [L.BF16, L.FP16])
def test_w4a16_gemm_decodes_signed_block_scales(bt):
    """Negative E4M3 block-scale codes are legal for the reference; the expansion to 16-bit weights keeps their sign."""
    for i, (m, n, k) in enumerate([(200, 150, 256), (300, 33, 576)]):
        c = Case(m, n, k, bt, L.BF16, -1, L.BF16, 1.25, 0.0, fa=SW if i else 0)
        h = build_case(c, 6600 + i)
        rng = np.random.default_rng(6600 + i)
        flip = rng.integers(0, 3, h["A"].scales.size) == 0
        h["A"].scales[flip & (h["A"].scales != 0)] |= 0x80
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == 5
        check_bound(c, h, got, amax, exp)


@pytest.mark.parametrize("spread,exponent", [(0, 0), (11, 0), (12, 0), (13, 0), (40, 0), (5, 100), (5, 101), (5, -94), (5, -102)])
@pytest.mark.parametrize("grouped", [False, True])
def test_w4a8_planes_at_the_edges_of_their_range(grouped, spread, exponent):
    """INT8 activations are two FP16 planes while a token's scales lie within 2^12 of each other (and near enough to one for the planes' scale to be a
    float), else three BF16 planes for every token: scales 2^spread apart around a power of two, q = -128 .. 127, a token of zeros, one whose large
    blocks meet zero weights only, negative scales.  Against 64 bits: (k + 2) 2^-24 of the sum of the terms' magnitudes (the FP32 accumulation bound)
    and half a unit of the 16-bit result."""
    m, n, k = 256, 96, 512
    gen = torch.Generator(device="cuda").manual_seed(100 + spread)
    ints = lambda lo, hi, shape, t: torch.randint(lo, hi, shape, generator=gen, device="cuda", dtype=t)
    w, ws = ints(0, 16, (m, k), torch.uint8), ints(0x28, 0x48, (m, k // 16), torch.uint8)
    w[:, :32] = 0
    x = ints(-128, 128, (n, k), torch.int8)
    s = (1.0 + torch.rand(n, k // 16, generator=gen, device="cuda", dtype=torch.float64) * (1 - 2.0 ** -23)).float()
    s[:, 1] = 2.0 - 2.0 ** -23
    x[:, 16] = -128
    s = (s.double() * 2.0 ** (exponent - spread * ints(0, 2, (n, k // 16), torch.int32).double())).float()
    s[:, 5] *= -1.0
    s[3] = 0.0
    s[4] *= 2.0 ** -9
    s[4, :2] = 2.0 ** exponent        # meets zero weights
    W = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device="cuda")[(w & 7).long()] * (1.0 - 2.0 * (w >> 3).double())
    W = (W.view(m, k // 16, 16) * ws.view(torch.float8_e4m3fn).double().unsqueeze(-1)).view(m, k)
    packed = (w[:, 0::2] | (w[:, 1::2] << 4)).contiguous()
    X = (x.double().view(n, k // 16, 16) * s.double().unsqueeze(-1)).view(n, k)
    alpha = 2.0 ** -exponent   # the results near one
    D = torch.zeros(n, m, dtype=torch.bfloat16, device="cuda")
    ta, tb, td = tensor(packed, L.NVFP4, ws, k // 16), tensor(x, L.INT8, s, k // 16), tensor(D, L.BF16)
    if grouped:
        seg = torch.tensor([0, 40, n], dtype=torch.int32, device="cuda")
        packed2, ws2 = torch.cat([packed, packed]), torch.cat([ws, ws])
        ta = tensor(packed2, L.NVFP4, ws2, k // 16)
        L.check(L.lib.nvfp4a_gemm_grouped(2, m, k, n, alpha, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), m, None,
                                          ctypes.c_void_p(seg.data_ptr()), stream()))
    else:
        L.check(L.lib.nvfp4a_gemm(m, n, k, alpha, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), m, None, stream()))
    assert L.lib.nvfp4a_b200_last_route() == 8
    want, size = X @ W.t() * alpha, X.abs() @ W.abs().t() * alpha
    assert bool(((D.double() - want).abs() <= (k + 2) * 2.0 ** -24 * size + 2.0 ** -8 * want.abs()).all())
    assert kernel_status() == 0


@pytest.mark.parametrize("m,n,k,out", [(300, 64, 512, "bf16"), (512, 200, 1088, "fp16"), (640, 1000, 2048, "fp32"), (300, 130, 4096, "bf16"), (768, 449, 1024, "swiglu")])
def test_w4a8_result_of_a_token_does_not_depend_on_its_neighbours(m, n, k, out):
    """Tokens whose scales lie more than 2^12 apart are BF16 planes, the others FP16 planes: whichever tokens of a call are of which kind -- one, the first
    and the last of a tile, every third, all -- a token's outputs are the bytes that it has among tokens of its own kind, and they keep the bound."""
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    w = torch.randint(0, 16, (m, k), generator=gen, device="cuda", dtype=torch.uint8)
    ws = torch.randint(0x28, 0x48, (m, k // 16), generator=gen, device="cuda", dtype=torch.uint8)
    W = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device="cuda")[(w & 7).long()] * (1.0 - 2.0 * (w >> 3).double())
    W = (W.view(m, k // 16, 16) * ws.view(torch.float8_e4m3fn).double().unsqueeze(-1)).view(m, k)
    packed = (w[:, 0::2] | (w[:, 1::2] << 4)).contiguous()
    x = torch.randint(-127, 128, (n, k), generator=gen, device="cuda", dtype=torch.int8)
    s = torch.exp2(-3.0 * torch.rand(n, k // 16, generator=gen, device="cuda")) * 2.0 ** -8
    wide_s = s.clone()
    wide_s[:, 3::7] *= 2.0 ** -14
    dt = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "swiglu": torch.bfloat16}[out]
    code = {"bf16": L.BF16, "fp16": L.FP16, "fp32": L.FP32, "swiglu": L.BF16}[out]
    ta = tensor(packed, L.NVFP4, ws, k // 16)

    def run(wide):
        sc = torch.where(wide.unsqueeze(1), wide_s, s).contiguous()
        d = torch.zeros(n, m // 2 if out == "swiglu" else m, dtype=dt, device="cuda")
        tb, td = tensor(x, L.INT8, sc, k // 16), tensor(d, code)
        if out == "swiglu":
            ex = L.Epilogue()
            ex.swiglu = 1
            L.check(L.lib.nvfp4a_gemm_ex(m, n, k, 2.0 ** -6, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), m // 2, None, ctypes.byref(ex), stream()))
        else:
            L.check(L.lib.nvfp4a_gemm(m, n, k, 1.0, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), m, None, stream()))
            X = (x.double().view(n, k // 16, 16) * sc.double().unsqueeze(-1)).view(n, k)
            want, size = X @ W.t(), X.abs() @ W.abs().t()
            assert bool(((d.double() - want).abs() <= (k + 2) * 2.0 ** -24 * size + (0.0 if out == "fp32" else 2.0 ** -8) * want.abs()).all())
        assert L.lib.nvfp4a_b200_last_route() == 8
        return d.view(torch.int32 if out == "fp32" else torch.int16)

    index = torch.arange(n, device="cuda")
    none, every = run(index < 0), run(index >= 0)
    for wide in (index == 7, (index == 0) | (index == n - 1), index % 3 == 1, index >= n // 2, index != 63):
        got = run(wide)
        assert torch.equal(got[~wide], none[~wide]) and torch.equal(got[wide], every[wide])
    assert kernel_status() == 0


def test_w4a8_planes_with_ue5m3_weight_scales():
    """Products with UE5M3 scales do not fit FP16: three BF16 planes."""
    c = Case(256, 96, 512, L.INT8, L.FP32, -1, L.BF16, 1.25, 0.0, fa=UE)
    h = build_case(c, 4395)
    exp = oracle_case(c, h, want_ref=True)
    got, amax = run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == 8
    check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("bt", [L.BF16, L.FP16, L.INT8])
def test_w4a16_units_of_two_stages_at_the_ends_of_k(bt):
    """The tcgen05 kernel works in units of eight MMAs: two stages of 64 values of k (one where FP16 sums segments of 64), or two planes of one stage.  Odd
    numbers of stages, a single one, segments that end in half a unit; one tile and several per CTA pair."""
    for i, k in enumerate([64, 128, 192, 448, 512, 576, 960, 1088, 1344]):
        for m, n in [(300, 70), (130, 700)] + ([(4500, 1100)] if k in (192, 576) else []):
            c = Case(m, n, k, bt, L.FP16 if i % 2 else L.BF16, -1, L.BF16 if i % 3 == 1 else -1, 1.25, 0.0, fa=SW if i % 2 else 0)
            h = build_case(c, 4800 + i)
            exp = oracle_case(c, h, want_ref=True)
            got, amax = run_gemm(c, h)
            assert L.lib.nvfp4a_b200_last_route() == (8 if bt == L.INT8 else 5), c
            check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("bt", [L.BF16, L.FP16, L.INT8])
@pytest.mark.parametrize("case", ["plain", "bias", "swiglu", "grouped"])
def test_w4a16_epilogues_compiled_for_plain_calls_equal_the_general_one(bt, case):
    """Calls with a 16-bit D and nothing but scales, bias and SwiGLU take an epilogue of their own; an amax wish brings the general one: the same bytes.
    D that TMA stores and D that it does not, ragged tiles, -0 results without a bias."""
    if (case == "swiglu" and bt == L.FP16) or (case == "grouped" and bt != L.INT8):
        pytest.skip("not a combination the entry points take")
    m, n, k = 528, 300, 640
    gen = torch.Generator(device="cuda").manual_seed(17)
    ints = lambda lo, hi, shape, t=torch.uint8: torch.randint(lo, hi, shape, generator=gen, device="cuda", dtype=t)
    groups = 3 if case == "grouped" else 1
    w, ws = ints(0, 256, (groups * m, k // 2)), ints(0x28, 0x48, (groups * m, k // 16))
    ta, x, xs = tensor(w, L.NVFP4, ws, k // 16), None, None
    if bt == L.INT8:
        x, xs = ints(-127, 128, (n, k), torch.int8), torch.rand(n, k // 16, generator=gen, device="cuda") + 0.1
        x[7] = 0
        tb = tensor(x, L.INT8, xs, k // 16)
    else:
        x = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16 if bt == L.BF16 else torch.float16)
        x[7] = -0.0
        tb = tensor(x, bt)
    bias = torch.randn(groups * m, generator=gen, device="cuda").to(torch.bfloat16)
    tbias = tensor(bias, L.BF16) if case in ("bias", "grouped") else None
    seg = torch.tensor([0, 65, 66, n], dtype=torch.int32, device="cuda")
    ex = L.Epilogue()
    ex.swiglu = int(case == "swiglu")
    mo = m // 2 if case == "swiglu" else m
    for dt in (torch.bfloat16, torch.float16):
        for ld in (mo, mo + 3):
            outs = []
            for amax in (None, torch.zeros(1, dtype=torch.float32, device="cuda")):
                D = torch.zeros(n, ld, dtype=dt, device="cuda")
                td = tensor(D, L.BF16 if dt == torch.bfloat16 else L.FP16, amax=amax)
                pb = ctypes.byref(tbias) if tbias is not None else None
                if case == "grouped":
                    L.check(L.lib.nvfp4a_gemm_grouped(groups, m, k, n, -0.01, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), ld, pb,
                                                      ctypes.c_void_p(seg.data_ptr()), stream()))
                elif case == "swiglu":
                    L.check(L.lib.nvfp4a_gemm_ex(m, n, k, -0.01, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), ld, pb, ctypes.byref(ex), stream()))
                else:
                    L.check(L.lib.nvfp4a_gemm(m, n, k, -0.01, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), ld, pb, stream()))
                assert L.lib.nvfp4a_b200_last_route() == (8 if bt == L.INT8 else 5)
                outs.append(D.view(torch.int16))
            assert bool(outs[0].any()) and torch.equal(outs[0], outs[1])
    assert kernel_status() == 0


@pytest.mark.parametrize("bt", [L.BF16, L.INT8])
@pytest.mark.parametrize("case", ["norm_swiglu", "out2", "norm", "add"])
def test_w4a16_epilogues_compiled_for_the_mlp_equal_the_general_one(bt, case):
    """RMSNorm scale with or without SwiGLU, the second output with sums of squares, and beta * C have epilogues of their own where D has 16 bits; an FP32 D
    takes the general one: the 16-bit D is its rounding, the other outputs and the amax are the same bytes.  With and without bias and amax, D that TMA stores or not, ragged tiles."""
    m, n, k = 528, 300, 640
    glu = case == "norm_swiglu"
    gen = torch.Generator(device="cuda").manual_seed(18)
    ints = lambda lo, hi, shape, t=torch.uint8: torch.randint(lo, hi, shape, generator=gen, device="cuda", dtype=t)
    w, ws = ints(0, 256, (m, k // 2)), ints(0x28, 0x48, (m, k // 16))
    ta = tensor(w, L.NVFP4, ws, k // 16)
    if bt == L.INT8:
        x, xs = ints(-127, 128, (n, k), torch.int8), torch.rand(n, k // 16, generator=gen, device="cuda") + 0.1
        tb = tensor(x, L.INT8, xs, k // 16)
    else:
        x = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
        tb = tensor(x, bt)
    bias, w2 = (torch.randn(m, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2))
    parts = torch.rand(n, 8, generator=gen, device="cuda")
    C = torch.randn(n, m, generator=gen, device="cuda").to(torch.bfloat16)
    tc = tensor(C, L.BF16)
    mo = m // 2 if glu else m

    def run(dt, ld, use_bias, use_amax):
        D, amax = torch.zeros(n, ld, dtype=dt, device="cuda"), torch.zeros(1, dtype=torch.float32, device="cuda")
        d2, sq = torch.zeros(n, m, dtype=torch.bfloat16, device="cuda"), torch.zeros(n, m // 16, dtype=torch.float32, device="cuda")
        ex = L.Epilogue()
        if case.startswith("norm"):
            ex.norm_parts, ex.norm_nparts, ex.norm_ld, ex.norm_inv_n, ex.norm_eps, ex.swiglu = parts.data_ptr(), 8, 8, 1.0 / 64.0, 1e-6, int(glu)
        elif case == "out2":
            ex.d2, ex.d2_dtype, ex.ldd2, ex.w2, ex.w2_dtype, ex.sq, ex.ld_sq = d2.data_ptr(), L.BF16, m, w2.data_ptr(), L.BF16, sq.data_ptr(), m // 16
        td = tensor(D, {torch.bfloat16: L.BF16, torch.float16: L.FP16, torch.float32: L.FP32}[dt], amax=amax if use_amax else None)
        tbias = tensor(bias, L.BF16)
        L.check(L.lib.nvfp4a_gemm_ex(m, n, k, -0.01, ctypes.byref(ta), k, ctypes.byref(tb), k, *(ctypes.c_float(0.5), ctypes.byref(tc), m) if case == "add" else (0.0, None, 0),
                                     ctypes.byref(td), ld, ctypes.byref(tbias) if use_bias else None, ctypes.byref(ex) if case != "add" else None, stream()))
        assert L.lib.nvfp4a_b200_last_route() == (8 if bt == L.INT8 else 5)
        return D, d2.view(torch.int16), sq.view(torch.int32), amax.view(torch.int32)

    for dt in (torch.bfloat16, torch.float16):
        for ld in (mo, mo + 3):
            for use in (False, True):
                got, want = run(dt, ld, use, use), run(torch.float32, ld, use, use)
                assert bool(want[0].any()) and torch.equal(got[0].view(torch.int16), want[0].to(dt).view(torch.int16))
                for a, b in zip(got[1:], want[1:]):
                    assert torch.equal(a, b)
    assert kernel_status() == 0


@pytest.mark.parametrize("k", [512, 576, 1088, 4096])
def test_w4a8_of_9_to_63_tokens_is_summed_in_segments(k):
    """INT8 activations of fewer than 64 tokens (k >= 512, 16-bit D, plain epilogue): the tcgen05 kernel in segments (route 8), within the bound; sums of
    positive terms as close to 64 bits as test_long_sums_on_the_tensor_cores_are_joined_in_fp32 asks.  Plain operands and images."""
    for i, (m, n) in enumerate([(128, 9), (300, 33), (515, 63), (130, 16)]):
        c = Case(m, n, k, L.INT8, L.FP16 if i % 2 else L.BF16, -1, L.BF16 if i % 2 else -1, 1.25, 0.0, fa=SW if i == 1 else 0)
        h = build_case(c, 4900 + i)
        exp = oracle_case(c, h, want_ref=True)
        for run in (run_gemm, lambda c, h: run_tc(c, h, gemv=False)):
            got, amax = run(c, h)
            assert L.lib.nvfp4a_b200_last_route() == 8, c
            check_bound(c, h, got, amax, exp)
    m, n = 300, 40
    gen = torch.Generator(device="cuda").manual_seed(k)
    w = torch.randint(1, 8, (m, k), generator=gen, device="cuda", dtype=torch.uint8)
    ws = torch.randint(0x28, 0x48, (m, k // 16), generator=gen, device="cuda", dtype=torch.uint8)
    W = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device="cuda")[w.long()]
    W = (W.view(m, k // 16, 16) * ws.view(torch.float8_e4m3fn).double().unsqueeze(-1)).view(m, k)
    packed, D, amax = (w[:, 0::2] | (w[:, 1::2] << 4)).contiguous(), torch.zeros(n, m, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, device="cuda")
    x, xs = torch.randint(1, 128, (n, k), generator=gen, device="cuda", dtype=torch.int8), torch.rand(n, k // 16, generator=gen, device="cuda") + 0.01
    ta, tb, td = tensor(packed, L.NVFP4, ws, k // 16), tensor(x, L.INT8, xs, k // 16), tensor(D, L.BF16, amax=amax)
    L.check(L.lib.nvfp4a_gemm(m, n, k, 1.0, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), m, None, stream()))
    assert L.lib.nvfp4a_b200_last_route() == 8
    want = (x.double().view(n, k // 16, 16) * xs.double().unsqueeze(-1)).view(n, k) @ W.t()
    assert abs(float(amax.double()) / float(want.max()) - 1.0) <= (16 + 16 + 4) * 2.0 ** -24
    assert torch.allclose(D.double(), want, rtol=2.0 ** -8, atol=0.0)
    assert kernel_status() == 0


@pytest.mark.parametrize("bt", [L.BF16, L.FP16, L.INT8])
def test_gemm_ex_and_its_twin_without_allocations_give_the_same_bytes(bt):
    """Up to 63 tokens whatever the activations are, with a reduction that nvfp4a_gemm would cut into parts or take to the planes."""
    for m, n, k in ((300, 16, 1024), (512, 33, 8192), (130, 63, 4096)):
        c = Case(m, n, k, bt, L.BF16, -1, -1, 1.0, 0.0)
        h = build_case(c, 5100 + n)
        A = DevFp4(rand_fp4(np.random.default_rng(n), m, k, glob=0.375))
        keep, tb = device_b(c, h)
        ta, ex, outs = A.tensor(), L.Epilogue(), []
        for entry in (L.lib.nvfp4a_gemm_ex, L.lib.nvfp4a_b200_gemm_ex_static):
            d = torch.zeros(n, m, dtype=torch.bfloat16, device="cuda")
            td = tensor(d, L.BF16)
            L.check(entry(m, n, k, 1.0, ctypes.byref(ta), k, ctypes.byref(tb), h["ldb"], 0.0, None, 0, ctypes.byref(td), m, None, ctypes.byref(ex), stream()))
            outs.append(d.view(torch.int16))
        assert torch.equal(*outs) and bool(outs[0].any())
    assert kernel_status() == 0


@pytest.mark.parametrize("bt", [L.BF16, L.FP16, L.INT8])
def test_long_reductions_of_few_tiles_in_parts_of_k(bt):
    """Few tiles and a long k: several CTA pairs take a run of k each, a small kernel adds their sums and runs the plain epilogue.  Every layout, runs of unequal
    length, odd numbers of stages, tails in m and n, bias, beta, every output type and amax; the same bytes on every call; and, captured in a graph
    (where BF16 and FP16 keep k whole), the bound again."""
    for i, (m, n, k) in enumerate([(512, 33, 8192), (130, 9, 4160), (300, 200, 6144 + 64), (700, 64, 4096 + 448), (128, 130, 16384)]):
        for fa, out in ((0, L.BF16), (SW, L.FP16), (AM | PR, L.FP32)):
            if bt == L.FP16 and out == L.FP32 or bt == L.INT8 and n < 64 and out == L.FP32:
                continue      # (other kernels)
            c = Case(m, n, k, bt, out, out if i % 2 else -1, L.BF16 if i % 2 else -1, 1.25, 0.5 if i % 2 else 0.0, fa=fa)
            h = build_case(c, 5000 + i)
            exp = oracle_case(c, h, want_ref=True)
            got, amax = run_gemm(c, h)
            assert L.lib.nvfp4a_b200_last_route() == (8 if bt == L.INT8 else 5) and L.lib.nvfp4a_b200_last_parts() > 1, c
            check_bound(c, h, got, amax, exp)
            again, amax2 = run_gemm(c, h)
            assert np.array_equal(got.view(np.uint8), again.view(np.uint8)) and amax == amax2, c
            if bt == L.INT8:
                got, amax = run_tc(c, h, gemv=False)
                check_bound(c, h, got, amax, exp)
    dA = DevFp4(h["A"])
    keepB, tB = device_b(c, h)
    dD, damax = dev(h["Dinit"]), torch.zeros(1, device="cuda")
    tA, tD = dA.tensor(), tensor(dD, c.dt, amax=damax)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert L.lib.nvfp4a_gemm(c.m, c.n, c.k, c.alpha, ctypes.byref(tA), h["lda"], ctypes.byref(tB), h["ldb"], 0.0, None, 0, ctypes.byref(tD), h["ldd"], None, stream()) == 0
    assert (L.lib.nvfp4a_b200_last_parts() > 1) == (bt == L.INT8)
    graph.replay()
    torch.cuda.synchronize()
    assert c.beta == 0.0 and c.bias < 0
    if bt == L.BF16:      # nvfp4a_gemm_ex keeps k whole: the bytes of the entry that must not allocate
        outs, ex = [], L.Epilogue()
        for entry in (L.lib.nvfp4a_gemm_ex, L.lib.nvfp4a_b200_gemm_ex_static):
            d = torch.zeros(c.n, c.m, dtype=torch.bfloat16, device="cuda")
            td = tensor(d, L.BF16)
            A0 = DevFp4(rand_fp4(np.random.default_rng(1), c.m, c.k, glob=0.375))
            ta = A0.tensor()
            L.check(entry(c.m, c.n, c.k, 1.0, ctypes.byref(ta), c.k, ctypes.byref(tB), h["ldb"], 0.0, None, 0, ctypes.byref(td), c.m, None, ctypes.byref(ex), stream()))
            assert L.lib.nvfp4a_b200_last_parts() == 1
            outs.append(d.view(torch.int16))
        assert torch.equal(*outs) and bool(outs[0].any())
    check_bound(c, h, host(dD).view(h["Dinit"].dtype), float(damax), exp)
    assert kernel_status() == 0


def graph_node_types(graph):
    from cuda.bindings import runtime
    raw = runtime.cudaGraph_t(graph.raw_cuda_graph())
    err, nodes, count = runtime.cudaGraphGetNodes(raw)
    err, nodes, count = runtime.cudaGraphGetNodes(raw, count)
    assert err == runtime.cudaError_t.cudaSuccess and count > 0
    return [runtime.cudaGraphNodeGetType(node)[1] for node in nodes], runtime, raw


@pytest.mark.parametrize("bt,n", [(L.INT8, 9), (L.INT8, 40), (L.BF16, 46), (L.FP16, 33)])
def test_captured_calls_leave_no_allocation_in_the_graph(bt, n):
    """nvfp4a_gemm where eager calls take scratch from the library's pool: a capture has no allocation node, so that the graph can be instantiated twice and be a
    child of another, and gives results within the bound.  INT8: the exact kernel's bytes."""
    c = Case(512, n, 4096, bt, L.BF16, -1, -1, 1.0, 0.0)
    h = build_case(c, 5200 + n)
    exp = oracle_case(c, h, want_ref=True)
    run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == (8 if bt == L.INT8 else 5)
    dA, (keep, tB), dD, damax = DevFp4(h["A"]), device_b(c, h), dev(h["Dinit"]), torch.zeros(1, device="cuda")
    tA, tD = dA.tensor(), tensor(dD, c.dt, amax=damax)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        assert L.lib.nvfp4a_gemm(c.m, c.n, c.k, 1.0, ctypes.byref(tA), h["lda"], ctypes.byref(tB), h["ldb"], 0.0, None, 0, ctypes.byref(tD), h["ldd"], None, stream()) == 0
    assert L.lib.nvfp4a_b200_last_route() == (7 if bt == L.INT8 else 5)
    types, runtime, raw = graph_node_types(graph)
    assert runtime.cudaGraphNodeType.cudaGraphNodeTypeMemAlloc not in types
    execs = []
    for _ in range(2):
        err, ex = runtime.cudaGraphInstantiate(raw, 0)
        assert err == runtime.cudaError_t.cudaSuccess
        execs.append(ex)
    err, parent = runtime.cudaGraphCreate(0)
    err, node = runtime.cudaGraphAddChildGraphNode(parent, None, 0, raw)
    assert err == runtime.cudaError_t.cudaSuccess
    err, ex = runtime.cudaGraphInstantiate(parent, 0)
    assert err == runtime.cudaError_t.cudaSuccess
    for e in execs + [ex]:
        dD.copy_(dev(h["Dinit"]))
        damax.zero_()
        assert runtime.cudaGraphLaunch(e, torch.cuda.current_stream().cuda_stream)[0] == runtime.cudaError_t.cudaSuccess
        torch.cuda.synchronize()
        check_bound(c, h, host(dD).view(h["Dinit"].dtype), float(damax), exp)
        if bt == L.INT8:
            old = L.lib.nvfp4a_b200_set_route(3)
            exact = run_gemm(c, h)[0]
            L.lib.nvfp4a_b200_set_route(old)
            assert np.array_equal(host(dD).view(np.uint8), exact.view(np.uint8))
    for e in execs + [ex]:
        runtime.cudaGraphExecDestroy(e)
    runtime.cudaGraphDestroy(parent)
    assert kernel_status() == 0


def test_scratch_from_the_callers_allocator_and_without_any():
    """nvfp4a_b200_set_scratch_alloc: the bytes of the pool's calls, one request a call, nothing from the pool; where the allocator has nothing, 16-bit activations keep
    k whole, 9 to 63 INT8 tokens take the exact kernel and 64 INT8 tokens report it."""
    kind = ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t)
    held, asked = [], []

    def give(ctx, size):
        asked.append(size)
        held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        return held[-1].data_ptr()

    def none(ctx, size):
        asked.append(size)
        return None

    give_c, none_c = kind(give), kind(none)
    for bt, n, route in ((L.INT8, 16, 8), (L.INT8, 130, 8), (L.BF16, 46, 5), (L.FP16, 33, 5)):
        c = Case(512, n, 8192, bt, L.BF16, -1, -1, 1.0, 0.0)
        h = build_case(c, 5300 + n)
        exp = oracle_case(c, h, want_ref=True)
        pool = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == route and L.lib.nvfp4a_b200_last_parts() > 1
        try:
            L.lib.nvfp4a_b200_set_scratch_alloc(give_c, None)
            del asked[:]
            got = run_gemm(c, h)
            assert len(asked) == 1 and L.lib.nvfp4a_b200_last_route() == route and L.lib.nvfp4a_b200_last_parts() > 1
            assert np.array_equal(got[0].view(np.uint8), pool[0].view(np.uint8)) and got[1] == pool[1]
            L.lib.nvfp4a_b200_set_scratch_alloc(none_c, None)
            del asked[:]
            if bt == L.INT8 and n >= 64:
                with pytest.raises(AssertionError, match="memory"):
                    run_gemm(c, h)
            else:
                got = run_gemm(c, h)
                assert L.lib.nvfp4a_b200_last_route() == (7 if bt == L.INT8 else 5)
                assert bt == L.INT8 or L.lib.nvfp4a_b200_last_parts() == 1
                check_bound(c, h, got[0], got[1], exp)
            assert 1 <= len(asked) <= 2
        finally:
            L.lib.nvfp4a_b200_set_scratch_alloc(None, None)
        assert np.array_equal(run_gemm(c, h)[0].view(np.uint8), pool[0].view(np.uint8))
        del held[:]
    assert kernel_status() == 0
