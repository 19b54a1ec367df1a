"""GPU parity tests of single kernels, called through the C ABI and compared with the CPU
checker on the same seeded inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,K,N", [(1, 64, 128), (12, 128, 512), (60, 1000, 4000), (768, 2000, 1000), (131, 257, 391)])
def test_gemm_simt_vs_checker(oracle, cuda_lib, R, K, N):
    from linmt_b200 import decoder
    rng = np.random.default_rng(R * 7 + K)
    X = rng.uniform(-1, 1, (R, K)).astype(np.float32)
    W = rng.uniform(-0.08, 0.08, (K, N)).astype(np.float32)
    Y = decoder.k_gemm(X, W, "simt", "fp32")
    ref = oracle.gemm(X, W)
    scale = np.abs(X).astype(np.float64) @ np.abs(W).astype(np.float64)
    # fp32 sums in a different order: error bounded by a few ulps of the absolute-value sum
    assert (np.abs(Y - ref) <= 4e-6 * scale + 1e-7).all()


@pytest.mark.parametrize("R,V,kk", [(4, 1000, 2), (24, 30000, 13), (7, 80000, 6), (3, 37, 5)])
def test_softmax_topk_vs_checker(oracle, cuda_lib, R, V, kk):
    from linmt_b200 import decoder
    rng = np.random.default_rng(V + kk)
    z = rng.normal(0, 0.5, (R, V)).astype(np.float32)
    idx, lp, eos = decoder.k_softmax_topk(z, kk)
    ridx, rlp = oracle.softmax_topk(z, kk)
    assert (idx == ridx).all()          # bit-exact indices
    np.testing.assert_allclose(lp, rlp, rtol=1e-5, atol=1e-6)
    z64 = z.astype(np.float64)
    lse = np.log(np.exp(z64 - z64.max(1, keepdims=True)).sum(1)) + z64.max(1)
    np.testing.assert_allclose(eos, z64[:, 1] - lse, rtol=1e-5, atol=1e-6)


def test_softmax_topk_ties_lowest_index(oracle, cuda_lib):
    from linmt_b200 import decoder
    V, kk = 30000, 13
    z = np.zeros((3, V), np.float32)                 # all equal: ids 0..kk-1
    z[1, [29999, 5, 17000, 17001]] = 2.0             # four-way tie on top, then zeros
    z[2] = np.repeat(np.arange(V // 4, dtype=np.float32)[::-1], 4)[:V] * 0.25  # groups of 4 equal values
    idx, lp, _ = decoder.k_softmax_topk(z, kk)
    ridx, _ = oracle.softmax_topk(z, kk)
    assert idx[0].tolist() == list(range(kk))
    assert idx[1].tolist() == [5, 17000, 17001, 29999] + list(range(0, 5)) + list(range(6, 10))
    assert (idx == ridx).all()


@pytest.mark.parametrize("R,K,N", [(12, 128, 512), (72, 1000, 30000), (768, 3000, 4000), (131, 257, 391)])
@pytest.mark.parametrize("path,prec,tol", [("tensor", "fp32", 1e-6), ("tensor3", "fp32", 1e-6), ("tensor2", "fp32", 4e-6), ("tensor", "bf16", 4e-3)])
def test_gemm_tensor_vs_checker(oracle, cuda_lib, R, K, N, path, prec, tol):
    """tcgen05 GEMM on split operands against a float64 product: the fp16 pair (default) and three
    bf16 planes give the error of an fp32 FMA loop, two bf16 planes ~2^-17 per product, one plane is
    plain bf16."""
    from linmt_b200 import decoder
    rng = np.random.default_rng(R + K + N)
    X = rng.uniform(-1, 1, (R, K)).astype(np.float32)
    W = rng.uniform(-0.08, 0.08, (K, N)).astype(np.float32)
    Y = decoder.k_gemm(X, W, path, prec)
    ref = X.astype(np.float64) @ W.astype(np.float64)
    scale = np.abs(X).astype(np.float64) @ np.abs(W).astype(np.float64)
    assert (np.abs(Y - ref) <= tol * scale + 1e-7).all(), float((np.abs(Y - ref) / scale).max())


def test_gemm_on_cta_pairs_vs_float64_and_one_tile(cuda_lib):
    """The decoder's gate product at full width (768 x 2048 times 2048 x 4096) picks 176-wide tiles, which as one
    tile per CTA leave room for two stages only: the library then runs CTA pairs (tcgen05 cta_group::2, each CTA
    loading half of the weight tile).  Against a float64 product the error is that of an fp32 FMA loop, and the
    bits are those of the one-tile kernel (LINMT_TC_PAIR=0): the same products accumulate in the same order."""
    import os
    from linmt_b200 import decoder
    rng = np.random.default_rng(11)
    R, K, N = 768, 2048, 4096
    X = rng.uniform(-1, 1, (R, K)).astype(np.float32)
    W = rng.uniform(-0.08, 0.08, (K, N)).astype(np.float32)
    Y = decoder.k_gemm(X, W, "tensor", "fp32")
    ref = X.astype(np.float64) @ W.astype(np.float64)
    scale = np.abs(X).astype(np.float64) @ np.abs(W).astype(np.float64)
    assert (np.abs(Y - ref) <= 1e-6 * scale + 1e-7).all(), float((np.abs(Y - ref) / scale).max())
    old = os.environ.get("LINMT_TC_PAIR")
    os.environ["LINMT_TC_PAIR"] = "0"
    try:
        Y1 = decoder.k_gemm(X, W, "tensor", "fp32")
    finally:
        if old is None:
            os.environ.pop("LINMT_TC_PAIR", None)
        else:
            os.environ["LINMT_TC_PAIR"] = old
    assert np.array_equal(Y, Y1)
    # a last row tile that is partly empty (700 = 5 x 128 + 60 rows)
    Y5 = decoder.k_gemm(X[:700], W, "tensor", "fp32")
    assert (np.abs(Y5 - ref[:700]) <= 1e-6 * scale[:700] + 1e-7).all()


@pytest.mark.parametrize("prec,tol", [("fp32", 1e-6), ("bf16", 4e-3)])
@pytest.mark.parametrize("R,K,N", [(1, 64, 128), (3, 200, 130), (16, 2048, 4096), (17, 1000, 3000), (32, 130, 20000), (33, 2048, 4096),
                                   (49, 700, 20000), (64, 1024, 391), (65, 256, 512), (96, 2048, 4096), (128, 1024, 3000), (129, 2048, 4096),
                                   (500, 1000, 4096)])
def test_gemm_few_rows_vs_float64(cuda_lib, R, K, N, prec, tol):
    """The weight-streaming product for few rows: edges of its row groups (4), MMA widths (16), of the change from half to
    whole SMs and to one MMA per product (65), to the other kernels (49 rows of many columns, 65 / 129), K slices of unequal
    length; and narrow tiles beyond."""
    from linmt_b200 import decoder
    rng = np.random.default_rng(R + K + N)
    X = rng.uniform(-1, 1, (R, K)).astype(np.float32)
    W = rng.uniform(-0.08, 0.08, (K, N)).astype(np.float32)
    Y = decoder.k_gemm(X, W, "tensor", prec)
    ref = X.astype(np.float64) @ W.astype(np.float64)
    scale = np.abs(X).astype(np.float64) @ np.abs(W).astype(np.float64)
    assert (np.abs(Y - ref) <= tol * scale + 1e-7).all(), float((np.abs(Y - ref) / scale).max())


@pytest.mark.parametrize("path,prec,R,K,V,kernel", [
    # one fp16 product, logits rounded to fp16, candidates recomputed (the default): a single column tile, unit edges,
    # the statistics of 80,000 classes and the activations of 7800 units that leave no room for the sums (the latter's
    # sweep passes 48 KB of shared memory), a partly empty row tile, an odd number of them
    ("auto", "fp32", 1, 64, 37, "rows"), ("auto", "fp32", 12, 1000, 30000, "rows"), ("auto", "fp32", 64, 1000, 5003, "rows"),
    ("auto", "fp32", 6, 1000, 80000, "rows"), ("auto", "fp32", 2, 7800, 300, "rows"), ("auto", "fp32", 65, 1000, 5003, "tile"), ("auto", "fp32", 128, 1000, 30000, "tile"),
    ("auto", "fp32", 100, 1000, 40000, "persist"), ("auto", "fp32", 129, 1000, 40000, "persist_pair"), ("auto", "fp32", 300, 1000, 30000, "persist_pair"),
    # three products
    ("tensor", "fp32", 12, 1000, 30000, "rows"), ("tensor", "fp32", 128, 1000, 5003, "rows"), ("tensor", "fp32", 65, 1000, 30000, "tile"),
    ("tensor", "fp32", 129, 1000, 30000, "persist"), ("tensor", "fp32", 768, 1000, 5003, "pair"),
    # bf16
    ("auto", "bf16", 48, 1000, 30000, "rows"), ("auto", "bf16", 49, 1000, 30000, "rows"), ("auto", "bf16", 70, 1000, 5003, "tile"),
    ("auto", "bf16", 100, 1000, 40000, "persist"), ("auto", "bf16", 700, 300, 30000, "persist_pair")])
def test_vocabulary_product_statistics_and_softmax(cuda_lib, path, prec, R, K, V, kernel):
    """Every GEMM form a vocabulary product takes: the logits against float64, the maximum of every block of columns (of
    the values as they are stored) and its sum of exponentials, each column in one block, and the top-kk behind them."""
    from linmt_b200 import decoder
    rng = np.random.default_rng(R + K + V)
    X = rng.uniform(-1, 1, (R, K)).astype(np.float32)
    W = rng.uniform(-0.08, 0.08, (K, V)).astype(np.float32)
    bias = rng.uniform(-0.5, 0.5, V).astype(np.float32)
    kk = min(13, V)
    out = decoder.k_logits(X, W, bias, kk, path, prec)
    assert out["kernel"] == kernel
    ref = X.astype(np.float64) @ W.astype(np.float64) + bias
    scale = np.abs(X).astype(np.float64) @ np.abs(W).astype(np.float64)
    Y = out["Y"].astype(np.float64)
    # both operands rounded to 8 bits (bf16) or 11 (fp16, and the stored value); otherwise 22, and the tensor core's
    # truncation of a 1000-term sum (2.4e-6 of 3072 terms was measured)
    if prec == "bf16":
        bound = 2.0 ** -8 * scale + 1e-6
    elif path == "auto":
        bound = 2.0 ** -10 * scale + 2.0 ** -11 * np.abs(ref) + 1e-6
    else:
        bound = 2e-6 * scale + 1e-6
    assert (np.abs(Y - ref) <= bound).all(), float((np.abs(Y - ref) / bound).max())
    seen = np.zeros(V, int)
    for i, (c0, c1) in enumerate(out["blocks"]):
        if c0 >= c1:
            assert (out["block_max"][:, i] == -np.inf).all()
            continue
        seen[c0:c1] += 1
        m = Y[:, c0:c1].max(1)
        assert (out["block_max"][:, i] == m).all(), i
        if out["block_sum"] is not None:
            np.testing.assert_allclose(out["block_sum"][:, i], np.exp(Y[:, c0:c1] - m[:, None]).sum(1), rtol=1e-5)
    assert (seen == 1).all()
    assert (out["block_sum"] is None) == (V == 80000 or K == 7800)
    # with recomputed candidates the result is the exact product's (1e-4 of a row's log-probabilities), otherwise the stored values'
    z = ref if path == "auto" and prec == "fp32" else Y
    lp = z - z.max(1, keepdims=True)
    lp -= np.log(np.exp(lp).sum(1, keepdims=True))
    tol = 1e-4 * np.abs(lp).max() if z is ref else 1e-5 * np.abs(lp).max()
    got = np.take_along_axis(lp, out["idx"].astype(np.int64), 1)
    assert (np.abs(out["logp"] - got) <= tol).all()
    assert (np.abs(out["logp"] - (-np.sort(-lp, 1)[:, :kk])) <= tol).all()
    assert (np.sort(out["idx"], 1)[:, 1:] != np.sort(out["idx"], 1)[:, :-1]).all()
    assert (np.abs(out["eos"] - lp[:, 1]) <= tol).all()
