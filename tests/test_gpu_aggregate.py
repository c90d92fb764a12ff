"""Block-at-a-time aggregation (csrc/aggregate.cu) against the oracle, bit for
bit, on random match sets: every region size of the launch rule (8, 16 and 24
pixels a side, chosen by the image's size), images that end inside a region,
patches 8 and 16, dense and tiled reference grids, partial groups."""
import numpy as np
import pytest

from gbm3d_b200 import options
from gbm3d_b200.api import _as_set

pytestmark = pytest.mark.gpu


def _opts(d, s, K, d2=32):
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=d, blockSizeWie=d, matchSize=d2, refStride=s, refStrideWie=s, numMax=K, numMin=K, levels=1,
             cycleSpin=1)
    return o


def _sets(rng, K, M, N, d2):
    S = rng.integers(1, d2 * d2 + 1, (K, M, N)).astype(np.uint32)
    S[0] = d2 * d2 // 2 + d2 // 2 + 1
    return np.asfortranarray(S)


@pytest.mark.parametrize("m,n,d,s,d2", [
    (61, 70, 8, 3, 32), (65, 49, 8, 8, 24), (96, 80, 16, 5, 32),   # 8-pixel regions
    (485, 500, 8, 7, 32), (480, 496, 16, 16, 16),                 # 16-pixel regions
    (945, 931, 8, 6, 32), (960, 944, 16, 16, 32),                 # 24-pixel regions
])
def test_wiener_aggregation(gpu, oracle, m, n, d, s, d2):
    rng = np.random.default_rng(m + n)
    K = 8
    M, N = (m - d) // s + 1, (n - d) // s + 1
    S = _sets(rng, K, M, N, d2)
    V1 = np.asfortranarray(rng.uniform(0, 255, (d, d, K, M, N)).astype(np.float32))
    V2 = np.asfortranarray(V1 + 25 * rng.standard_normal(V1.shape).astype(np.float32))
    o = _opts(d, s, K, d2)
    U, W = gpu.denoiseAndAggregateWieFast(V1, V2, _as_set(S), 25.0, o)
    Uo, Wo = oracle.denoiseAndAggregateWieFast(V1, V2, S, 25.0, o, prec=32)
    assert np.array_equal(U, Uo) and np.array_equal(W, Wo)


@pytest.mark.parametrize("m,n,d,s,d2", [
    (61, 70, 8, 3, 32), (96, 80, 16, 5, 24), (485, 500, 8, 8, 32), (945, 931, 8, 7, 32), (960, 944, 16, 16, 32),
])
def test_hard_threshold_aggregation(gpu, oracle, m, n, d, s, d2):
    rng = np.random.default_rng(m * n)
    K = 8
    M, N = (m - d) // s + 1, (n - d) // s + 1
    S = _sets(rng, K, M, N, d2)
    cnt = np.asfortranarray(rng.integers(1, K + 1, (M, N)).astype(np.int32))
    V = np.asfortranarray(rng.uniform(0, 255, (M * d, N * d, K)).astype(np.float32))
    o = _opts(d, s, K, d2)
    tau = 25.0 * options.getTau(1, 1)
    Psi, Psi2 = options.bank_from_factors(options.bior_factors())
    U, W = gpu.denoiseAndAggregateGPU(V, _as_set(S, cnt), tau, Psi, Psi2, o)
    Uo, Wo = oracle.denoiseAndAggregateGPU(V, S, tau, o, cnt=cnt, filters=oracle.bior_filters(), prec=32)
    assert np.array_equal(U, Uo) and np.array_equal(W, Wo)


@pytest.mark.parametrize("m,n,d,s,K", [(40, 33, 8, 1, 32), (48, 41, 16, 1, 16), (33, 32, 8, 8, 8)])
def test_full_and_empty_lists(gpu, oracle, m, n, d, s, K):
    """Every match at its own reference: rounds of candidates that all hit or all miss."""
    rng = np.random.default_rng(m + n + K)
    M, N = (m - d) // s + 1, (n - d) // s + 1
    m, n = (M - 1) * s + d, (N - 1) * s + d
    S = np.full((K, M, N), 32 * 16 + 17, dtype=np.uint32, order="F")
    V1 = np.asfortranarray(rng.uniform(0, 255, (d, d, K, M, N)).astype(np.float32))
    V2 = np.asfortranarray(V1 + 25 * rng.standard_normal(V1.shape).astype(np.float32))
    o = _opts(d, s, K)
    U, W = gpu.denoiseAndAggregateWieFast(V1, V2, _as_set(S), 25.0, o)
    Uo, Wo = oracle.denoiseAndAggregateWieFast(V1, V2, S, 25.0, o, prec=32)
    assert np.array_equal(U, Uo) and np.array_equal(W, Wo)
