"""The weights that the tensor-core GEMM expands to FP16, one by one."""
import numpy as np
import pytest

from nvfp4effma_b200 import _lib as L
from test_gemm_gpu import Case, build_case, kernel_status, oracle_case, run_gemm, values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bt,out,n,k", [(L.FP16, L.FP16, 64, 64), (L.FP16, L.BF16, 300, 320), (L.INT8, L.BF16, 64, 64), (L.INT8, L.BF16, 300, 320)])
def test_every_value_under_every_scale_code(bt, out, n, k):
    """Row r has scale code r (negative codes, subnormals, 0x7F among them) and the nibbles of a block are all sixteen; token j is one in place j % k, so that an
    output is one weight: at most 6 significant bits, exact in every type.  A tile of part of a stage pair, an odd number of stages, several tiles of tokens."""
    c = Case(256, n, k, bt, out, -1, -1, 1.0, 0.0)
    h = build_case(c, 5500)
    A, B = h["A"], h["B"]
    A.data[:] = np.resize(np.arange(0x10, 0x100, 0x22, dtype=np.uint8), A.data.size)   # bytes 0x10, 0x32, ... 0xfe: nibbles 0 to 15 in order
    A.scales.reshape(256, A.ld_scale)[:] = np.arange(256, dtype=np.uint8)[:, None]
    A.glob[:] = 1.0
    one = np.zeros((n, h["ldb"]), np.float32)
    one[np.arange(n), np.arange(n) % k] = 1.0
    if bt == L.INT8:
        B.data[:] = one.astype(np.int8).reshape(B.data.shape)
        B.scales[:] = 1.0
        B.glob[:] = 1.0
    else:
        B.raw[:] = one.astype(np.float16).view(B.raw.dtype).reshape(B.raw.shape)
    got, _ = run_gemm(c, h)
    assert L.lib.nvfp4a_b200_last_route() == (8 if bt == L.INT8 else 5)
    e2m1 = np.array([0, 0.5, 1, 1.5, 2, 3, 4, 6, 0, -0.5, -1, -1.5, -2, -3, -4, -6])
    code = np.arange(128)
    mag = np.where(code < 8, (code & 7) * 2.0 ** -9, (8 + (code & 7)) * 2.0 ** ((code >> 3) - 10.0))
    want = e2m1[np.arange(n) % k % 16][:, None] * np.concatenate([mag, -mag])[None, :]
    assert np.array_equal(values(got, c, h), want)
    assert np.array_equal(values(got, c, h), values(oracle_case(c, h)["D"], c, h))
    assert kernel_status() == 0
