"""The tensor-core product at the edges of its tiles: every tile width, part-filled tiles in both
directions, K below, at and past one chunk and past the operand ring, and the fused epilogues on
widths and row counts that are no multiple of a tile."""
import numpy as np
import pytest

from arbo_gpu_fit_gb300.surrogate import MLP, tc_gemm
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 16, 16), (129, 48, 80), (33, 112, 656), (4000, 592, 64), (8192, 1040, 48),
                                   (20000, 512, 128)])
def test_product_matches_numpy(gpu, M, N, K):
    rng = np.random.default_rng(M + N + K)
    a = mlp_ref.bf16(rng.standard_normal((M, K)).astype(np.float32))
    b = mlp_ref.bf16(rng.standard_normal((N, K)).astype(np.float32))
    c, _ = tc_gemm(a, b)
    # FP32 accumulation of K exact products: each addition rounds to half a unit of the partial sum,
    # which the sum of the products' magnitudes bounds.
    bound = K * 2.0 ** -24 * (np.abs(a).astype(np.float64) @ np.abs(b).T.astype(np.float64))
    err = np.abs(c - a.astype(np.float64) @ b.T.astype(np.float64))
    assert np.all(err <= np.maximum(bound, 1e-30))


@pytest.mark.parametrize("hidden,layers,n_out,rows", [(16, 1, 1, 16), (48, 2, 7, 144), (272, 1, 100, 400), (656, 2, 33, 208)])
def test_epilogues_match_restatement(gpu, hidden, layers, n_out, rows):
    rng = np.random.default_rng(hidden + rows)
    net = MLP(6, hidden, layers, n_out, max_batch=rows + 32, seed=7)
    x = rng.uniform(-1, 1, (rows, 6)).astype(np.float32)
    t = rng.standard_normal((rows, n_out)).astype(np.float32)
    loss = net.gradients(x, t)
    ws = [net.layer(l)[0] for l in range(net.layers)]
    bs = [net.layer(l)[1] for l in range(net.layers)]
    want_loss, dws, dbs, y = mlp_ref.forward_backward(x, t, ws, bs, net.dims, n_out)
    # The restatement rounds to BF16 at the same places; an FP32 sum that lands on the other side of
    # a rounding boundary moves one operand by 2^-8, which stays below 2e-3 in the norm of a gradient.
    assert loss == pytest.approx(want_loss, rel=1e-4)
    for l in range(net.layers):
        _, _, dw, db = net.layer(l)
        assert np.linalg.norm(dw - dws[l]) <= 2e-3 * np.linalg.norm(dws[l])
        assert np.linalg.norm(db - dbs[l]) <= 2e-3 * np.linalg.norm(dbs[l])
    assert np.abs(net.forward(x) - y[:, :n_out]).max() <= 1e-3 * max(1.0, np.abs(y).max())


def test_row_counts_past_the_captured_ones(gpu):
    """More row counts than captured sequences are kept: the first, the captured and the evicted call of each
    give the same outputs and gradients, bit for bit."""
    rng = np.random.default_rng(5)
    net = MLP(6, 64, 2, 30, max_batch=192, seed=3)
    x = rng.uniform(-1, 1, (192, 6)).astype(np.float32)
    t = rng.standard_normal((192, 30)).astype(np.float32)
    first = {}
    for turn in range(3):
        for rows in range(16, 192, 16):
            for _ in range(1 + turn):
                net.gradients(x[:rows], t[:rows])
                got = [net.forward(x[:rows])] + [net.layer(l)[k] for l in range(net.layers) for k in (2, 3)]
                for a, b in zip(first.setdefault(rows, got), got):
                    np.testing.assert_array_equal(a, b)
