"""A tensor-core product whose waits run out (their limit is zero, so the first operand copies are in flight):
it reports the error, and products, network passes and steps after it are right. Narrow and wide tiles, fewer
and more chunks than the operand ring holds, one tile and several to a CTA."""
import ctypes

import numpy as np
import pytest

from arbo_gpu_fit_gb300.surrogate import tc_gemm
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(16, 16, 16), (64, 512, 512), (300, 128, 2048), (4096, 1024, 1024), (20000, 512, 128)])
def test_product_that_gives_up(gpu, M, N, K):
    rng = np.random.default_rng(M + K)
    a = mlp_ref.bf16(rng.standard_normal((M, K)).astype(np.float32))
    b = mlp_ref.bf16(rng.standard_normal((N, K)).astype(np.float32))
    want, _ = tc_gemm(a, b)
    for _ in range(3):
        err = ctypes.c_uint32(0)
        assert gpu.arbo_selftest_stalled_product(M, N, K, ctypes.byref(err)) == 0, gpu.arbo_last_error()
        assert err.value == 1
        np.testing.assert_array_equal(tc_gemm(a, b)[0], want)
    # FP32 accumulation of K exact products (as in the test of the tiles' edges).
    bound = K * 2.0 ** -24 * (np.abs(a).astype(np.float64) @ np.abs(b).T.astype(np.float64))
    assert np.all(np.abs(want - a.astype(np.float64) @ b.T.astype(np.float64)) <= np.maximum(bound, 1e-30))


def test_bad_shapes_are_refused(gpu):
    err = ctypes.c_uint32(0)
    for shape in ((0, 16, 16), (16, 8, 16), (16, 16, 24)):
        assert gpu.arbo_selftest_stalled_product(*shape, ctypes.byref(err)) != 0
