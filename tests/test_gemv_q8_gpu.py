"""The INT8 / NVFP4 GEMV (csrc/gemv_q8.cu): long reductions in sections, rounds of slices, and dense activations that it makes INT8 itself."""
import ctypes

import numpy as np
import pytest
import torch

import nvfp4effma_b200.api as nf
import oracle as O
from nvfp4effma_b200 import _lib as L
from test_gemm_gpu import SW, UE, Case, build_case, check_bound, kernel_status, oracle_case, run_gemm, run_tc, values
from util import DevFp4, dev, host, stream, tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bt", [L.INT8, L.NVFP4])
@pytest.mark.parametrize("n,k", [(1, 17408), (3, 9216), (8, 20032)])
def test_long_reductions_in_sections(bt, n, k):
    """Clusters of two and four CTAs, the last section short, its last chunk ragged; E4M3 and UE5M3 scales."""
    for fa in (SW, UE):
        c = Case(70, n, k, bt, L.FP32, -1, L.BF16, 1.0, 0.0, fa=fa)
        h = build_case(c, 6100 + n)
        got, amax = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == 6
        check_bound(c, h, got, amax, oracle_case(c, h, want_ref=True))
    assert kernel_status() == 0


def test_bits_of_a_row_do_not_depend_on_rounds_of_slices():
    """Eight vectors and so many rows that a CTA's sums do not fit shared memory at once: the first rows' bytes over and over."""
    base, times, n, k = 1024, 60, 8, 2048
    c = Case(base, n, k, L.INT8, L.FP32, -1, -1, 1.0, 0.0)
    h = build_case(c, 6200)
    first = values(run_gemm(c, h)[0], c, h)
    A = DevFp4(h["A"])
    data, scales, m = A.data.repeat(times), A.scales.repeat(times), base * times
    y = torch.zeros(n, m, dtype=torch.float32, device="cuda")
    q, s, gb = dev(h["B"].data), dev(h["B"].scales), dev(h["B"].glob)
    ta, tb, td = tensor(data, L.NVFP4, scales, h["A"].ld_scale, A.glob, flags=h["A"].flags), tensor(q, L.INT8, s, h["B"].ld_scale, gb), tensor(y, L.FP32)
    L.check(L.lib.nvfp4a_gemm(m, n, k, 1.0, ctypes.byref(ta), h["lda"], ctypes.byref(tb), h["ldb"], 0.0, None, 0, ctypes.byref(td), m, None, stream()))
    assert L.lib.nvfp4a_b200_last_route() == 6
    got = host(y).astype(np.float64).reshape(n, times, base)
    assert np.array_equal(got, np.broadcast_to(first[:, None], got.shape))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("image", [False, True])
def test_dense_activations_give_the_bytes_of_quantizing_first(dtype, image):
    """nvfp4a_b200_gemv_w4a8 against nvfp4a_quantize to INT8 and nvfp4a_gemm / nvfp4a_gemv_tc: ragged k, one to eight vectors, zeros, infinities, NaNs, blocks whose
    scale takes the IEEE divisions."""
    gen = torch.Generator(device="cuda").manual_seed(62)
    for m, n, k in ((17, 1, 64), (200, 3, 320), (300, 8, 1088), (128, 5, 4096), (130, 2, 14400)):
        w = nf.quantize(torch.randn(m, k, generator=gen, device="cuda"), swizzled=n % 2 == 0)
        op = w._operand()
        x = torch.randn(n, k, generator=gen, device="cuda")
        x[:, :16] = 0
        x[0, 16:32] *= 1e-30
        if dtype != torch.float16:
            x[-1, 32:48] *= 1e30
        if n == 3:
            x[1, 50], x[2, 51] = float("inf"), float("nan")
        x = x.to(dtype)
        xq = nf.quantize_int8(x)
        img = nf.TCWeight(w, "int8").image if image else None
        code = {torch.bfloat16: L.BF16, torch.float16: L.FP16, torch.float32: L.FP32}[dtype]
        ta = tensor(img if image else op.data, L.NVFP4, None if image else op.scales, 0 if image or op.flags & SW else op.scales.stride(0), op.glob, flags=op.flags)
        tx, tq = tensor(x, code), tensor(xq.data, L.INT8, xq.scales, k // 16)
        bias = torch.randn(m, generator=gen, device="cuda")
        out = [torch.zeros(n, m, device="cuda") for _ in range(2)]
        amax = [torch.zeros(1, device="cuda") for _ in range(2)]
        td, tbias = [tensor(o, L.FP32, amax=a) for o, a in zip(out, amax)], tensor(bias, L.FP32)
        L.check(L.lib.nvfp4a_b200_gemv_w4a8(m, n, k, 0.5, ctypes.byref(ta), k, int(image), ctypes.byref(tx), k, 0.0, None, 0, ctypes.byref(td[0]), m, ctypes.byref(tbias),
                                            stream()))
        assert L.lib.nvfp4a_b200_last_route() == 6
        if image:
            L.check(L.lib.nvfp4a_gemv_tc(m, n, k, 0.5, ctypes.byref(ta), ctypes.byref(tq), k, 0.0, None, 0, ctypes.byref(td[1]), m, ctypes.byref(tbias), stream()))
        else:
            L.check(L.lib.nvfp4a_gemm(m, n, k, 0.5, ctypes.byref(ta), k, ctypes.byref(tq), k, 0.0, None, 0, ctypes.byref(td[1]), m, ctypes.byref(tbias), stream()))
        assert torch.equal(out[0].view(torch.int32), out[1].view(torch.int32)), (m, n, k)
        assert torch.equal(amax[0].view(torch.int32), amax[1].view(torch.int32))
    assert kernel_status() == 0


def test_what_the_fused_entry_leaves_to_two_calls():
    """Nine vectors, more values than one CTA after another should quantize, and the CUDA-core route: not supported, nothing written."""
    w = nf.quantize(torch.ones(64, 8192, device="cuda"))
    op = w._operand()
    ta = tensor(op.data, L.NVFP4, op.scales, op.scales.stride(0), op.glob, flags=op.flags)
    x, y = torch.ones(9, 8192, dtype=torch.bfloat16, device="cuda"), torch.zeros(9, 64, device="cuda")
    tx, td = tensor(x, L.BF16), tensor(y, L.FP32)

    def call(n):
        return L.lib.nvfp4a_b200_gemv_w4a8(64, n, 8192, 1.0, ctypes.byref(ta), 8192, 0, ctypes.byref(tx), 8192, 0.0, None, 0, ctypes.byref(td), 64, None, stream())

    assert call(9) == L.NOT_SUPPORTED and call(5) == L.NOT_SUPPORTED
    old = L.lib.nvfp4a_b200_set_route(1)
    assert call(2) == L.NOT_SUPPORTED
    L.lib.nvfp4a_b200_set_route(old)
    assert not bool(y.any()) and call(4) == L.OK and bool(y[:4].all()) and not bool(y[4:].any())


@pytest.mark.parametrize("flags,one", [(0, 0x38), (UE, 0x78)])
@pytest.mark.parametrize("n", [1, 4, 7])
def test_sums_of_the_smallest_activations_keep_their_bits(n, flags, one):
    """INT8 activations whose scales are 2^-140: every product with a weight and its block scale is a whole number of 2^-144, so that FP32, whose smallest number is
    2^-149, holds every sum exactly, and the weight's decode factor of 2^100 brings the result back.  No tolerance."""
    m, k = 40, 192
    rng = np.random.default_rng(63)
    codes, scodes = rng.integers(0, 16, (m, k)).astype(np.uint8), rng.integers(one, one + 16, (m, k // 16)).astype(np.uint8)     # (scales of 1 to 3.75)
    q = rng.integers(-127, 128, (n, k)).astype(np.int8)
    e2m1 = np.array([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0])
    w = np.where(codes & 8, -1.0, 1.0) * e2m1[codes & 7] * np.repeat((1.0 + (scodes & 7) / 8.0) * 2.0 ** ((scodes >> 3) - float(one >> 3)), 16, axis=1)
    want = q.astype(np.float64) @ w.T * 2.0 ** -40
    data, scales, glob = dev((codes[:, 0::2] | codes[:, 1::2] << 4).reshape(-1)), dev(scodes.reshape(-1)), dev(np.array([2.0 ** 100], np.float32))
    values8, scales8, ones = dev(q.reshape(-1)), dev(np.full(n * k // 16, 2.0 ** -140, np.float32)), dev(np.ones(1, np.float32))
    ta, tb = tensor(data, L.NVFP4, scales, k // 16, glob, flags=flags), tensor(values8, L.INT8, scales8, k // 16, ones)
    y = torch.zeros(n, m, device="cuda")
    td = tensor(y, L.FP32)
    L.check(L.lib.nvfp4a_gemm(m, n, k, 1.0, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), m, None, stream()))
    assert L.lib.nvfp4a_b200_last_route() == 6
    assert np.array_equal(host(y).astype(np.float64).reshape(n, m), want)


def test_activations_that_the_fused_entry_leaves_to_two_calls_cost_no_try():
    """Five vectors of 8192 values: the INT8 values, their scales, the result and the amax are all that a call allocates."""
    gen = torch.Generator(device="cuda").manual_seed(64)
    w, x, amax = nf.quantize(torch.randn(64, 8192, generator=gen, device="cuda")), torch.randn(5, 8192, generator=gen, device="cuda").to(torch.bfloat16), torch.zeros(1, device="cuda")
    y = nf.linear(x, w, act="int8", amax_out=amax)
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    again = nf.linear(x, w, act="int8", amax_out=amax)
    assert torch.cuda.memory_stats()["allocation.all.allocated"] - before == 4
    assert torch.equal(y, again) and torch.equal(y, nf.linear(nf.quantize_int8(x), w, out_dtype=torch.bfloat16)) and float(amax.to(torch.bfloat16)) == float(y.abs().max())
