"""The GEMV of one and two BF16 vectors below the FP4 tensor-core GEMV's sizes (csrc/gemv_stream.cu) against the CPU oracle: where its units, warps,
slices and sections end, activations that need more than one FP16 plane, and the independence of a row's bits from the matrix around it."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from nvfp4effma_b200 import _lib as L
from test_epilogue_gpu import run_case
from test_gemm_gpu import AM, OUTS, PR, SW, Case, build_case, check_bound, kernel_status, oracle_case, run_gemm, run_tc, values
from util import DevFp4, dev, host, stream, tensor

pytestmark = pytest.mark.gpu
GEMV = 2


def run(layout, c, h):
    got = run_tc(c, h, gemv=True) if layout == "image" else run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == GEMV, c
    return got


@pytest.mark.parametrize("layout", ["image", "swizzled", "linear"])
@pytest.mark.parametrize("n", [1, 2])
def test_edges_of_units_slices_and_tiles(layout, n):
    """One unit and less, remainders of 64 values, one to sixteen warps per slice, tails in m, several slices per CTA, negative scales, 0x7F."""
    for i, (m, k) in enumerate([(1, 64), (15, 128), (17, 192), (127, 256), (129, 320), (300, 1088), (2500, 64), (5000, 448), (2400, 2112), (130, 4160), (200, 14400)]):
        c = Case(m, n, k, L.BF16, OUTS[i % 3], -1 if i % 4 == 1 else OUTS[i % 3], L.BF16 if i % 2 else -1, 1.25 if i % 2 else 1.0, 1.0 if i % 4 == 1 else 0.0,
                 fa=(SW if layout == "swizzled" else 0) | (AM | PR if i % 3 == 2 else 0))
        h = build_case(c, 5100 + i)
        rng = np.random.default_rng(i)
        codes = h["A"].scales
        codes[(rng.integers(0, 4, codes.size) == 0) & (codes != 0)] |= 0x80
        if layout != "image":
            codes[rng.integers(0, codes.size, 3)] = 0x7E
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run(layout, c, h)
        check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("layout", ["image", "linear"])
@pytest.mark.parametrize("n", [1, 2])
@pytest.mark.parametrize("spread", [2.0 ** -31, 2.0 ** -36, 2.0 ** -70, 2.0 ** -115])
def test_values_of_further_planes_count_where_large_ones_meet_zeros(layout, n, spread):
    """Every tenth activation is of the order of 1 and meets a zero weight in every row, the others are `spread` times smaller (and some of them another 2^-33
    below): the result consists of values that the first plane of their chunk cannot hold."""
    m, k = 200, 1344
    c = Case(m, n, k, L.BF16, L.FP32, -1, -1, 1.0, 0.0)
    h = build_case(c, 5200)
    rng = np.random.default_rng(5201)
    big = np.arange(0, k, 10)
    a = h["A"].data.reshape(m, h["lda"] // 2)
    for kk in big:
        a[:, kk // 2] &= 0xF0 if kk % 2 == 0 else 0x0F
    x = (rng.standard_normal((n, h["ldb"])) * spread).astype(np.float32)
    x[:, 5::7] *= np.float32(2.0 ** -33) if spread > 2.0 ** -80 else np.float32(1.0)
    x[:, big] = rng.choice([-1.0, 1.0, 1.9], (n, big.size))
    x[:, 300:320] = 0
    h["B"] = O.Dense(L.BF16, O.from_f32(x.reshape(-1), L.BF16), h["ldb"])
    exp = oracle_case(c, h, want_ref=True)
    got, amax = run(layout, c, h)
    check_bound(c, h, got, amax, exp)
    small = h["B"].raw.copy().reshape(n, -1)
    small[:, big] = 0                                  # the same without the large ones: they contribute nothing
    hs = dict(h, B=O.Dense(L.BF16, small.reshape(-1), h["ldb"]))
    alone = oracle_case(c, hs, want_ref=True)
    err = np.abs(values(got, c, h) - alone["ref64"])
    assert (err <= alone["bound"]).all(), float((err / alone["bound"]).max())
    assert kernel_status() == 0


def test_subnormal_huge_infinite_and_nan_activations():
    m, n, k = 64, 2, 512
    c = Case(m, n, k, L.BF16, L.FP32, -1, -1, 1.0, 0.0)
    h = build_case(c, 5300)
    rng = np.random.default_rng(5301)
    for scale in (2.0 ** -126, 2.0 ** -133, 2.0 ** 100):
        x = (rng.integers(-100, 101, (n, h["ldb"])) * scale).astype(np.float32)
        hx = dict(h, B=O.Dense(L.BF16, O.from_f32(x.reshape(-1), L.BF16), h["ldb"]))
        exp = oracle_case(c, hx, want_ref=True)
        got, _ = run("linear", c, hx)
        err = np.abs(values(got, c, hx) - exp["ref64"])
        assert (err <= exp["bound"] + 2.0 ** -149 * k).all()        # (products and partial sums below FP32's normal range round to multiples of 2^-149)
    x = rng.standard_normal((n, h["ldb"])).astype(np.float32)
    x[0, 77], x[1, 300] = np.inf, np.nan
    hx = dict(h, B=O.Dense(L.BF16, O.from_f32(x.reshape(-1), L.BF16), h["ldb"]))
    got = values(run("linear", c, hx)[0], c, hx)
    a = h["A"].data.reshape(m, -1)[:, 77 // 2] >> 4                  # the weights that meet the infinity
    sc = h["A"].scales.reshape(m, -1)[:, 77 // 16] & 0x7F
    zero = ((a & 7) == 0) | (sc == 0)
    assert np.isnan(got[0][zero]).all() and np.isinf(got[0][~zero]).all() and np.isnan(got[1]).all()


@pytest.mark.parametrize("n,k", [(1, 65536), (2, 36864), (2, 100032)])
def test_long_reductions_in_sections(n, k):
    """Activations of 128 KiB in one CTA; a cluster of two and of four CTAs, the last section short and its last chunk ragged."""
    c = Case(50, n, k, L.BF16, L.FP32, -1, L.BF16, 1.0, 0.0, fa=SW)
    h = build_case(c, 5400)
    exp = oracle_case(c, h, want_ref=True)
    for layout in ("swizzled", "image"):
        got, amax = run(layout, c, h)
        check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("n,k,sections", [(2, 2048, 1), (2, 36864, 2)])
def test_bits_of_a_row_do_not_depend_on_the_matrix(n, k, sections):
    """A matrix so tall that a CTA's slices take several rounds (or a cluster several slices) repeats the first rows' bytes."""
    base = 1024 if sections == 1 else 128
    times = 230 if sections == 1 else 40
    c = Case(base, n, k, L.BF16, L.FP32, -1, -1, 1.0, 0.0)
    h = build_case(c, 5500)
    first = values(run_gemm(c, h)[0], c, h)
    assert L.lib.nvfp4a_b200_last_route() == GEMV
    old = L.lib.nvfp4a_b200_set_route(2)               # (a matrix of this size would go to the FP4 tensor-core GEMV)
    try:
        A = DevFp4(h["A"])
        data, scales = A.data.repeat(times), A.scales.repeat(times)
        x, m = dev(h["B"].raw), base * times
        y = torch.zeros(n, m, dtype=torch.float32, device="cuda")
        ta = tensor(data, L.NVFP4, scales, h["A"].ld_scale, A.glob, flags=h["A"].flags)
        tb, td = tensor(x, L.BF16), tensor(y, L.FP32)
        L.check(L.lib.nvfp4a_gemm(m, n, k, 1.0, ctypes.byref(ta), h["lda"], ctypes.byref(tb), h["ldb"], 0.0, None, 0, ctypes.byref(td), m, None, stream()))
        assert L.lib.nvfp4a_b200_last_route() == GEMV
        got = host(y).astype(np.float64).reshape(n, times, base)
        assert np.array_equal(got, np.broadcast_to(first[:, None], got.shape))
    finally:
        L.lib.nvfp4a_b200_set_route(old)


@pytest.mark.parametrize("mask", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("image", [False, True])
def test_extended_epilogue(mask, image):
    for i, (m, n, k) in enumerate([(48, 1, 320), (528, 2, 2304), (2400, 2, 64)]):
        run_case(m, n, k, L.BF16, (L.BF16, L.FP32)[i % 2], mask, i > 0, i == 1 and not mask & 2, image)
    assert L.lib.nvfp4a_b200_last_route() == GEMV and kernel_status() == 0
