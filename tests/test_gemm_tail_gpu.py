"""The tensor-core kernel's last round of tiles in parts of k beside whole tiles, against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

import nvfp4effma_b200.api as nf
from nvfp4effma_b200 import _lib as L
from test_gemm_gpu import Case, DevFp4, build_case, check_bound, dev, device_b, host, kernel_status, oracle_case, run_tc, stream, tensor

pytestmark = pytest.mark.gpu
SW = L.SCALES_SWIZZLED


def run_plain(c, h):
    """nvfp4a_gemm without an amax (the plain epilogue)."""
    dA, (keep, tB), dD = DevFp4(h["A"]), device_b(c, h), dev(h["Dinit"])
    bias = dev(h["bias"]) if h["bias"] is not None else None
    tA, tD, tbias = dA.tensor(), tensor(dD, c.dt), tensor(bias, c.bias) if bias is not None else None
    L.check(L.lib.nvfp4a_gemm(c.m, c.n, c.k, c.alpha, ctypes.byref(tA), h["lda"], ctypes.byref(tB), h["ldb"], 0.0, None, 0, ctypes.byref(tD), h["ldd"],
                              ctypes.byref(tbias) if tbias is not None else None, stream()))
    return host(dD).view(h["Dinit"].dtype)


# (74 SM pairs; tiles of 256 rows and at most 256 tokens, 128 with FP16.  FP16: an output pitch that TMA stores take and one that they do not; the other rows are no whole 16
# bytes and take plain stores)
@pytest.mark.parametrize("bt,m,n,k", [
    (L.INT8, 2500, 1793, 4096 + 192),  # a last token alone in its tile, rows past the matrix, an odd number of stages
    (L.BF16, 18997, 250, 7168),       # one tile more than a round
    (L.FP16, 4864, 600, 6144 + 64),
])
@pytest.mark.parametrize("fa,out,bias,pitch", [(0, L.BF16, -1, 8), (SW, L.FP16, L.BF16, 3)])
def test_last_round_in_parts_of_k(bt, m, n, k, fa, out, bias, pitch):
    """Whole tiles and parts both within the bound of one sum over k, every output written, the same bytes on every call."""
    c = Case(m, n, k, bt, out, -1, bias, 2.0 ** -12 if out == L.FP16 else 1.25, 0.0, fa=fa)   # (FP16: inside its range)
    h = build_case(c, 5400)
    h["ldd"] = (m + 7) // 8 * 8 + pitch
    h["Dinit"] = np.resize(h["Dinit"], n * h["ldd"])
    exp = oracle_case(c, h, want_ref=True)
    got = run_plain(c, h)
    assert L.lib.nvfp4a_b200_last_route() == (8 if bt == L.INT8 else 5) and L.lib.nvfp4a_b200_last_parts() > 1
    check_bound(c, h, got, float(exp["amax"]), exp)
    assert np.array_equal(got.view(np.uint8), run_plain(c, h).view(np.uint8))
    assert kernel_status() == 0


TAILS = [(torch.bfloat16, "int8", 2504, 1793, 4288), (torch.bfloat16, "exact", 19000, 250, 7168), (torch.float16, "exact", 4864, 600, 6208)]


def operands(dtype, m, n, k):
    gen = torch.Generator(device="cuda").manual_seed(54)
    w = nf.quantize((torch.randn(m, k, generator=gen, device="cuda") * 0.02).to(torch.bfloat16), swizzled=True)
    return torch.randn(n, k, generator=gen, device="cuda").to(dtype), w


@pytest.mark.parametrize("dtype,act,m,n,k", TAILS)
def test_what_is_asked_for_beside_the_product_changes_no_bits(dtype, act, m, n, k):
    """The amax, beta * out and (where this kernel writes it) an FP32 result: the same sums as the plain call, in parts of k for the same outputs."""
    x, w = operands(dtype, m, n, k)
    y = nf.linear(x, w, act=act)
    assert L.lib.nvfp4a_b200_last_parts() > 1
    amax = torch.zeros(1, device="cuda")
    assert torch.equal(nf.linear(x, w, act=act, amax_out=amax), y)
    out = torch.zeros_like(y)
    assert torch.equal(nf.linear(x, w, act=act, out=out, beta=1.0), y)
    assert L.lib.nvfp4a_b200_last_parts() > 1
    if dtype == torch.bfloat16:
        wide = nf.linear(x, w, act=act, out_dtype=torch.float32)
        assert torch.equal(wide.to(dtype), y) and float(amax) == float(wide.abs().max())
    assert kernel_status() == 0


@pytest.mark.parametrize("bt,m,n,k,form", [
    (L.INT8, 2504, 1793, 4096 + 192, "plain"),
    (L.INT8, 2504, 1793, 4096 + 192, "image"),
    (L.INT8, 2504, 1793, 4096 + 192, "wide tokens"),   # every third token is three BF16 planes, the others two FP16 planes
    (L.INT8, 2504, 1793, 4096 + 192, "ue5m3"),         # three planes for all of them
    (L.BF16, 19000, 250, 7168, "plain"),
])
def test_last_round_in_parts_of_k_beside_tiles_that_tma_stores(bt, m, n, k, form):
    """A pitch and rows of whole 16 bytes: TMA stores the whole tiles, whose last tokens do not fill a tile; image tiles and scales at a part's first stage."""
    c = Case(m, n, k, bt, L.BF16, -1, L.BF16, 1.25, 0.0, fa=L.SCALES_UE5M3 if form == "ue5m3" else SW)
    h = build_case(c, 5450)
    h["ldd"] = m
    h["Dinit"] = np.resize(h["Dinit"], n * m)
    if form == "wide tokens":
        h["B"].scales.reshape(n, -1)[1::3, 3::7] *= np.float32(2.0 ** -14)
    exp = oracle_case(c, h, want_ref=True)
    got, amax = run_tc(c, h, gemv=False) if form == "image" else (run_plain(c, h), float(exp["amax"]))
    assert L.lib.nvfp4a_b200_last_route() == (8 if bt == L.INT8 else 5) and L.lib.nvfp4a_b200_last_parts() > 1
    check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0
