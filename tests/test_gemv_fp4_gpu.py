"""The FP4 tensor-core GEMV (BF16 activation vectors: a kernel for n <= 2, another for 3 <= n <= 8; weights fed to tcgen05 as stored, activations as FP4 digit
planes) against the CPU oracle: plain epilogue within the FP32-accumulation bound, extended epilogue bit for bit given the
kernel's own accumulators -- the checks of test_gemm_gpu / test_epilogue_gpu, with the kernel pinned by
nvfp4a_b200_set_gemv_splits and its use confirmed by nvfp4a_b200_last_route."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from nvfp4effma_b200 import _lib as L
from test_epilogue_gpu import run_case
from test_gemm_gpu import AM, OUTS, PR, SW, Case, build_case, check_bound, kernel_status, oracle_case, run_gemm, run_tc
from util import DevFp4, dev, host, stream, tensor

pytestmark = pytest.mark.gpu
FP4_GEMV = 3


@pytest.fixture
def pin():
    def set_splits(s):
        assert L.lib.nvfp4a_b200_set_gemv_splits(s) == 0
    yield set_splits
    L.lib.nvfp4a_b200_set_gemv_splits(0)


@pytest.mark.parametrize("splits", [1, 2, 4, 8])
def test_image_operand_all_splits(pin, splits):
    pin(splits)
    sizes = [(77, 1, 2048), (300, 2, 2048), (256, 1, 4096), (515, 2, 2048), (1100, 1, 2304), (4096, 2, 2048)]
    for i, (m, n, k) in enumerate(sizes):
        for fa in (0, AM | PR):
            c = Case(m, n, k, L.BF16, OUTS[i % 3], -1 if i % 4 == 1 else OUTS[i % 3], L.BF16 if i % 2 else -1, 1.25 if i % 2 else 1.0,
                     1.0 if i % 4 == 1 else 0.0, fa=fa)
            h = build_case(c, 900 + i)
            exp = oracle_case(c, h, want_ref=True)
            got, amax = run_tc(c, h, gemv=True)
            assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV, c
            check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


def test_plain_operand_with_swizzled_scales(pin):
    pin(2)
    for i, (m, n, k) in enumerate([(200, 1, 512), (513, 2, 1024), (2048, 1, 4096)]):
        c = Case(m, n, k, L.BF16, OUTS[i % 3], OUTS[i % 3], L.FP32, 0.5, 0.0, fa=SW | (AM if i else 0))
        h = build_case(c, 950 + i)
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV, c
        check_bound(c, h, got, amax, exp)
    # linear scales are left to the mma.sync GEMV
    c = Case(200, 1, 512, L.BF16, L.BF16, L.BF16, -1, 1.0, 0.0)
    run_gemm(c, build_case(c, 960))
    assert L.lib.nvfp4a_b200_last_route() == 2
    assert kernel_status() == 0


def test_automatic_route_by_size():
    c = Case(300, 1, 2048, L.BF16, L.BF16, L.BF16, -1, 1.0, 0.0, fa=SW)
    run_gemm(c, build_case(c, 961))
    assert L.lib.nvfp4a_b200_last_route() == 2          # small: the mma.sync GEMV
    c = Case(8192, 1, 8192, L.BF16, L.BF16, L.BF16, -1, 1.0, 0.0, fa=SW)
    h = build_case(c, 962)
    exp = oracle_case(c, h, want_ref=True)
    got, amax = run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV   # 38 MB of weights
    check_bound(c, h, got, amax, exp)


@pytest.mark.parametrize("spread", [0, 12, 23, 31, 60, 120])
def test_activations_with_a_wide_dynamic_range(pin, spread):
    """|x| spread over 2^-spread .. 1 (and exact zeros): up to 2^-24 of the largest element the digit planes hold every bit;
    a CTA that meets anything smaller computes its share on the CUDA cores instead."""
    pin(2)
    m, n, k = 384, 2, 2048
    c = Case(m, n, k, L.BF16, L.FP32, L.FP32, -1, 1.0, 0.0, fa=SW)
    h = build_case(c, 970 + spread)
    rng = np.random.default_rng(spread)
    x = rng.standard_normal(h["ldb"] * n).astype(np.float32) * np.exp2(-rng.integers(0, spread + 1, h["ldb"] * n)).astype(np.float32)
    x[rng.random(x.size) < 0.1] = 0.0
    h["B"] = O.Dense(L.BF16, O.from_f32(x, L.BF16), h["ldb"])
    exp = oracle_case(c, h, want_ref=True)
    got, amax = run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV
    check_bound(c, h, got, amax, exp)


@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("linear", [False, True])
def test_large_activations_that_meet_zero_weights(pin, linear, splits):
    """A few activations of magnitude 1 at positions where every weight is zero, all others near 2^-40: the result consists of
    the small terms alone, so bits dropped relative to the LARGEST activation would show (the FP32 accumulation bound is
    relative to sum |a_i x_i|).  Both tokens; swizzled and linear block scales; one token left narrow."""
    from util import rand_fp4
    pin(splits)   # one CTA per row tile: sixteen chunks through a ring of four stages, the eight consumer warps far apart
    m, n, k = 640, 2, 4096
    c = Case(m, n, k, L.BF16, L.FP32, L.FP32, -1, 1.0, 0.0, fa=0 if linear else SW)
    h = build_case(c, 990)
    rng = np.random.default_rng(991)
    if linear:
        h["A"] = rand_fp4(rng, m, k, ld=h["lda"], ld_scale=k // 16, glob=0.375)
    big = rng.choice(k, 9, replace=False)
    a = h["A"].data.reshape(m, h["lda"] // 2)
    for kk in big:                                    # zero nibble kk of every weight row
        a[:, kk // 2] &= 0xF0 if kk % 2 == 0 else 0x0F
    x = (rng.standard_normal(h["ldb"] * n) * 2.0 ** -40).astype(np.float32)
    x[big] = rng.choice([-1.0, 1.0, 1.5], big.size)   # token 0 only; token 1 stays within a few binades
    x[h["ldb"]:] *= 2.0 ** 40
    h["B"] = O.Dense(L.BF16, O.from_f32(x, L.BF16), h["ldb"])
    exp = oracle_case(c, h, want_ref=True)
    got, amax = run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV
    check_bound(c, h, got, amax, exp)
    assert np.abs(exp["ref64"][0]).max() < 1e-6       # token 0's outputs really are made of the small terms
    assert kernel_status() == 0


def test_linear_scales_back_to_back_at_the_benchmark_size():
    """8192 x 8192 weights with linear block scales, automatic split, 300 launches back to back in one CUDA graph (as a decode
    step issues them): every launch gives the bytes of the first, and those are within the bound of the oracle.  The stages of
    the weight ring land in any order here; a warp that re-tiles scales must not take a stage's second fill for its first."""
    from util import rand_fp4
    m, n, k = 8192, 1, 8192
    c = Case(m, n, k, L.BF16, L.BF16, -1, -1, 1.0, 0.0)
    h = build_case(c, 995)
    rng = np.random.default_rng(996)
    h["A"] = rand_fp4(rng, m, k, ld=h["lda"], ld_scale=k // 16, glob=0.375)
    exp = oracle_case(c, h, want_ref=True)
    got, amax = run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV
    check_bound(c, h, got, amax, exp)
    dA = DevFp4(h["A"])
    tA, x = dA.tensor(), dev(h["B"].raw)
    tx = tensor(x, L.BF16)
    outs = [torch.zeros(h["ldd"], dtype=torch.int16, device="cuda") for _ in range(50)]
    touts = [tensor(o, L.BF16) for o in outs]

    def launch(i):
        st = L.lib.nvfp4a_gemm(m, n, k, 1.0, ctypes.byref(tA), h["lda"], ctypes.byref(tx), h["ldb"], 0.0, None, 0, ctypes.byref(touts[i]), h["ldd"],
                               None, stream())
        assert st == 0, L.lib.nvfp4a_last_error()

    launch(0)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for i in range(50):
            launch(i)
    for _ in range(6):
        g.replay()
    torch.cuda.synchronize()
    assert kernel_status() == 0
    first = outs[0][:m].cpu()
    assert np.array_equal(first.numpy().view(np.uint16), got.reshape(-1)[:m])
    assert all(torch.equal(o[:m].cpu(), first) for o in outs[1:])


def test_extended_epilogue(pin):
    pin(2)
    v = 0
    for (m, n, k) in [(64, 1, 512), (1024, 1, 1024), (528, 2, 2304), (4096, 2, 1024)]:
        for mask in range(1, 6):
            glu = bool(mask & 2)
            run_case(m, n, k, L.BF16, L.FP32 if v % 2 else L.BF16, mask, (not glu) and v % 3 == 1, (not glu) and v % 4 == 2, True)
            assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV
            v += 1
    assert kernel_status() == 0


def test_plain_operand_with_linear_scales(pin):
    """Linear block scales with a 16-byte aligned pitch: a TMA box brings [256 rows][16 bytes] per chunk, four warps re-tile it."""
    from util import rand_dense, rand_fp4
    pin(2)
    for i, (m, n, k) in enumerate([(300, 1, 512), (1000, 2, 2048), (4096, 1, 4096)]):
        c = Case(m, n, k, L.BF16, OUTS[i % 3], OUTS[i % 3], L.BF16 if i % 2 else -1, 1.0, 0.0)
        h = build_case(c, 980 + i)
        rng = np.random.default_rng(981 + i)
        h["A"] = rand_fp4(rng, m, k, ld=h["lda"], ld_scale=k // 16, glob=0.375)   # compact scale rows: pitch k / 16, a multiple of 16
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV, c
        check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("layout", ["image", "swizzled", "linear"])
def test_three_to_eight_activation_vectors(pin, splits, layout):
    """The digit planes of up to eight tokens fill the MMA's 128 rows: every n from 3 to 8, all cuts of k (at most seven or fourteen 256-value
    chunks per CTA), row remainders, and matrices with more 256-row tiles than clusters run at once, whose clusters take two tiles."""
    from util import rand_fp4
    pin(splits)
    sizes = [(77, 3, 2048), (300, 8, 256 * splits), (515, 5, 1536 if splits < 8 else 2048), (1100, 4, 256 * (14 if splits == 1 else splits + 1)), (256, 7, 256 * 7 * splits),
             (33, 6, 2304 if splits > 1 else 1792)]
    if splits == 8:
        sizes.append((4096 + 300, 8, 2048))       # 18 tiles on 15 clusters
    if splits == 4:
        sizes.append((8704 + 200, 6, 1024))       # 35 tiles on 33 clusters
    for i, (m, n, k) in enumerate(sizes):
        c = Case(m, n, k, L.BF16, OUTS[i % 3], OUTS[i % 3] if i % 2 else -1, L.BF16 if i % 2 else -1, 1.25 if i % 2 else 1.0, 0.5 if i % 2 else 0.0,
                 fa=SW if layout == "swizzled" else 0)
        h = build_case(c, 1200 + 10 * splits + i)
        if layout == "linear":
            h["A"] = rand_fp4(np.random.default_rng(i), m, k, ld=h["lda"], ld_scale=-(-k // 256) * 16, glob=0.375)
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_tc(c, h, gemv=True) if layout == "image" else run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV, c
        check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("linear", [False, True])
def test_eight_vectors_of_which_one_does_not_fit_the_digit_planes(pin, linear):
    """One token spread over 2^-60 .. 1: the CTAs that meet it consume the weight ring on the CUDA cores, two tiles each."""
    from util import rand_fp4
    pin(8)
    m, n, k = 4096 + 300, 8, 2048
    c = Case(m, n, k, L.BF16, L.FP32, L.FP32, -1, 1.0, 0.0, fa=0 if linear else SW)
    h = build_case(c, 1300)
    rng = np.random.default_rng(1301)
    if linear:
        h["A"] = rand_fp4(rng, m, k, ld=h["lda"], ld_scale=k // 16, glob=0.375)
    x = rng.standard_normal((n, h["ldb"])).astype(np.float32)
    x[5, :700] *= np.exp2(-rng.integers(0, 61, 700)).astype(np.float32)
    h["B"] = O.Dense(L.BF16, O.from_f32(x.reshape(-1), L.BF16), h["ldb"])
    exp = oracle_case(c, h, want_ref=True)
    got, amax = run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV
    check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


def test_extended_epilogue_of_several_vectors(pin):
    v = 0
    for splits, (m, n, k) in [(2, (64, 3, 512)), (4, (1024, 8, 1024)), (8, (528, 5, 2304)), (1, (4096, 4, 1024)), (8, (4096 + 256, 8, 2048))]:
        pin(splits)
        for mask in range(1, 6):
            glu = bool(mask & 2)
            run_case(m, n, k, L.BF16, L.FP32 if v % 2 else L.BF16, mask, (not glu) and v % 3 == 1, (not glu) and v % 4 == 2, True)
            assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV
            v += 1
    assert kernel_status() == 0


@pytest.mark.parametrize("layout", ["image", "swizzled", "linear"])
def test_negative_block_scales_of_several_vectors(pin, layout):
    """Negative E4M3 block scales are legal for the reference: they keep their sign on the FP4 tensor cores, whose scales are unsigned, and
    where the CUDA cores take over (the last size, a token spread over 2^-60 .. 1)."""
    from util import rand_fp4
    for i, (splits, m, n, k) in enumerate([(1, 300, 5, 768), (2, 515, 3, 1024), (8, 4096 + 300, 8, 2048), (4, 300, 4, 1024)]):
        pin(splits)
        c = Case(m, n, k, L.BF16, L.FP32, -1, L.BF16, 1.25, 0.0, fa=SW if layout == "swizzled" else 0)
        h = build_case(c, 1400 + i)
        rng = np.random.default_rng(1400 + i)
        if layout == "linear":
            h["A"] = rand_fp4(rng, m, k, ld=h["lda"], ld_scale=k // 16, glob=0.375)
        flip = rng.integers(0, 3 if i else 200, h["A"].scales.size) == 0
        h["A"].scales[flip & (h["A"].scales != 0)] |= 0x80
        if i == 3:
            x = rng.standard_normal((n, h["ldb"])).astype(np.float32)
            x[2, :700] *= np.exp2(-rng.integers(0, 61, 700)).astype(np.float32)
            h["B"] = O.Dense(L.BF16, O.from_f32(x.reshape(-1), L.BF16), h["ldb"])
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_tc(c, h, gemv=True) if layout == "image" else run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV, c
        check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("layout", ["image", "swizzled", "linear"])
def test_block_scale_code_7f_of_several_vectors(pin, layout):
    """Codes 0x7F and 0xFF decode as +-480 (a NaN to the tensor cores) in a few blocks, in the first and last row and in the last block of a row."""
    from util import rand_fp4
    for i, (splits, m, n, k) in enumerate([(1, 300, 5, 768), (2, 515, 3, 1024), (8, 4096 + 300, 8, 2048)]):
        pin(splits)
        c = Case(m, n, k, L.BF16, L.FP32, -1, L.BF16, 1.25, 0.0, fa=SW if layout == "swizzled" else 0)
        h = build_case(c, 1500 + i)
        rng = np.random.default_rng(1500 + i)
        if layout == "linear":
            h["A"] = rand_fp4(rng, m, k, ld=h["lda"], ld_scale=k // 16, glob=0.375)
        sc = h["A"].scales
        sc[rng.integers(0, sc.size, 1 + sc.size // 500)] = 0x7F
        sc[rng.integers(0, sc.size, 1 + sc.size // 500)] = 0xFF
        sc[0] = 0x7F
        if layout == "linear":
            sc[(m - 1) * (k // 16) + k // 16 - 1] = 0xFF
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_tc(c, h, gemv=True) if layout == "image" else run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV, c
        assert np.isfinite(exp["ref64"]).all()
        check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("spread", [0, 23, 24, 25, 31, 200])
def test_digit_planes_at_the_edges_of_their_range(pin, spread):
    """Activations whose largest and smallest magnitudes are 2^spread apart, around the last digit plane, with subnormals, signed zeros and a token of
    zeros; and tokens too small for the planes' scale to be a float (eb < 31)."""
    for i, (n, top) in enumerate([(1, 1.0), (2, 2.0 ** -100), (8, 2.0 ** 100), (5, 2.0 ** -120)]):
        pin(2)
        m, k = 300, 1024
        c = Case(m, n, k, L.BF16, L.FP32, -1, -1, 1.0, 0.0, fa=SW)
        h = build_case(c, 1700 + i)
        rng = np.random.default_rng(1700 + spread + i)
        x = (rng.uniform(1, 2, (n, h["ldb"])) * rng.choice([-1.0, 1.0], (n, h["ldb"]))).astype(np.float32) * np.float32(top)
        x[:, ::3] *= np.float32(2.0) ** -spread
        x[:, 5] = -0.0
        if n == 5:
            x[2] = 0.0
        h["B"] = O.Dense(L.BF16, O.from_f32(x.reshape(-1), L.BF16), h["ldb"])
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV, c
        check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("layout", ["image", "swizzled", "linear"])
def test_signed_and_largest_block_scale_codes_of_one_and_two_vectors(pin, layout):
    """Negative block scales keep their sign and codes 0x7F / 0xFF are +-480, on the tensor cores and where the CUDA cores take over (the last size, a
    vector spread over 2^-60 .. 1); row remainders with and without a second 128-row half."""
    from util import rand_fp4
    for i, (splits, m, n, k) in enumerate([(1, 300, 1, 768), (2, 515, 2, 1024), (4, 77, 2, 2048), (8, 1100, 1, 2048), (2, 300, 2, 1024)]):
        pin(splits)
        c = Case(m, n, k, L.BF16, L.FP32, -1, L.BF16, 1.25, 0.0, fa=SW if layout == "swizzled" else 0)
        h = build_case(c, 1600 + i)
        rng = np.random.default_rng(1600 + i)
        if layout == "linear":
            h["A"] = rand_fp4(rng, m, k, ld=h["lda"], ld_scale=k // 16, glob=0.375)
        sc = h["A"].scales
        sc[(rng.integers(0, 3 if i else 200, sc.size) == 0) & (sc != 0)] |= 0x80
        if i % 2:
            sc[rng.integers(0, sc.size, 1 + sc.size // 500)] = 0x7F
            sc[rng.integers(0, sc.size, 1 + sc.size // 500)] = 0xFF
        if i == 4:
            x = rng.standard_normal((n, h["ldb"])).astype(np.float32)
            x[1, :700] *= np.exp2(-rng.integers(0, 61, 700)).astype(np.float32)
            h["B"] = O.Dense(L.BF16, O.from_f32(x.reshape(-1), L.BF16), h["ldb"])
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_tc(c, h, gemv=True) if layout == "image" else run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV, c
        assert np.isfinite(exp["ref64"]).all()
        check_bound(c, h, got, amax, exp)
    assert kernel_status() == 0


@pytest.mark.parametrize("few", [1, 7, 31, 32, 33, 40])
def test_activations_of_which_the_planes_drop_bits(pin, few):
    """`few` activations per vector far below the last digit plane and nothing else beside large ones that meet zero weights, so that the result is made of
    what the planes drop: up to 64 a CTA adds by itself, more it leaves to the CUDA cores.  The same bytes on every launch."""
    for i, (splits, n, layout) in enumerate([(1, 1, SW), (2, 2, 0), (4, 2, SW)]):
        pin(splits)
        m, k = 300, 4096
        c = Case(m, n, k, L.BF16, L.FP32, -1, -1, 1.0, 0.0, fa=layout)
        h = build_case(c, 1800 + few + i)
        rng = np.random.default_rng(1801 + few)
        if not layout:
            from util import rand_fp4
            h["A"] = rand_fp4(rng, m, k, ld=h["lda"], ld_scale=k // 16, glob=0.375)
        big = rng.choice(k, 8, replace=False)
        a = h["A"].data.reshape(m, h["lda"] // 2)
        for kk in big:
            a[:, kk // 2] &= 0xF0 if kk % 2 == 0 else 0x0F
        x = np.zeros((n, h["ldb"]), dtype=np.float32)
        x[:, big] = rng.choice([-1.0, 1.5], (n, big.size))
        small = rng.choice(np.setdiff1d(np.arange(k), big), few, replace=False)
        x[:, small] = rng.standard_normal((n, few)) * np.exp2(-rng.integers(22, 90, (n, few)))
        h["B"] = O.Dense(L.BF16, O.from_f32(x.reshape(-1), L.BF16), h["ldb"])
        exp = oracle_case(c, h, want_ref=True)
        got, amax = run_gemm(c, h)
        assert L.lib.nvfp4a_b200_last_route() == FP4_GEMV
        check_bound(c, h, got, amax, exp)
        for _ in range(5):
            assert np.array_equal(run_gemm(c, h)[0].view(np.uint8), got.view(np.uint8))
    assert kernel_status() == 0


def test_one_and_two_vectors_take_the_tensor_cores_from_32_megabytes_up():
    """Below that the mma.sync GEMV, whose time and bytes do not depend on how far the activations spread: one vector whose tail lies 2^-30 below its
    largest value, through the plain and the image entry, gives the bytes of the mma.sync GEMV asked for by name."""
    for m, k, route in ((6144, 4096, 2), (4096, 14336, 2), (1024, 1024, 2), (8192, 8192, FP4_GEMV)):
        for n in (1, 2):
            c = Case(m, n, k, L.BF16, L.BF16, -1, -1, 1.0, 0.0, fa=SW)
            h = build_case(c, 1900)
            x = O.to_f32(h["B"].raw, L.BF16).reshape(n, -1).copy()
            x[:, 1::2] *= np.float32(2.0 ** -30)
            h["B"] = O.Dense(L.BF16, O.from_f32(x.reshape(-1), L.BF16), h["ldb"])
            exp = oracle_case(c, h, want_ref=True) if n == 1 else None
            for run in (run_gemm, lambda c, h: run_tc(c, h, gemv=True)):
                got, amax = run(c, h)
                assert L.lib.nvfp4a_b200_last_route() == route, c
                if exp is not None:
                    check_bound(c, h, got, amax, exp)
                if route == 2:
                    old = L.lib.nvfp4a_b200_set_route(2)
                    named = run(c, h)[0]
                    L.lib.nvfp4a_b200_set_route(old)
                    assert np.array_equal(got.view(np.uint8), named.view(np.uint8))
    assert kernel_status() == 0


def test_which_matrices_several_vectors_take_to_the_tensor_cores():
    """8192 x 8192 with up to four vectors, not with more: there the mma.sync GEMV, whose time does not depend on the activations, is near enough."""
    for m, k, n, route in ((8192, 8192, 4, FP4_GEMV), (8192, 8192, 6, 2), (8192, 8192, 8, 2), (14336, 4096, 8, FP4_GEMV), (4096, 14336, 3, 2), (4096, 4096, 8, 2)):
        A = DevFp4(O.Fp4(m, k, flags=SW))
        x, y = torch.ones(n, k, dtype=torch.bfloat16, device="cuda"), torch.ones(n, m, dtype=torch.bfloat16, device="cuda")
        ta, tb, td = A.tensor(), tensor(x, L.BF16), tensor(y, L.BF16)
        L.check(L.lib.nvfp4a_gemm(m, n, k, 1.0, ctypes.byref(ta), k, ctypes.byref(tb), k, 0.0, None, 0, ctypes.byref(td), m, None, stream()))
        assert L.lib.nvfp4a_b200_last_route() == route, (m, k, n)
        assert not bool(y.any())
    assert kernel_status() == 0
