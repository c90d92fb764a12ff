"""The marching wavelet kernels (csrc/wavelet.cu) against the oracle, bit for
bit, at the sizes where they can go wrong: coarse levels at and around the
filter length (below it the generic kernels run), strips of 27, 28 and 32
coefficient rows and their remainders, segments of a few columns, one to three
cycle spins (odd shifts; a cycle count that is no power of two), both pipeline
banks and the video's."""
import numpy as np
import pytest

from gbm3d_b200 import api, options
from gbm3d_b200.api import _as_set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wav", ["bior", "haar"])
@pytest.mark.parametrize("M,N,K,levels,cycles", [
    (1, 2, 2, 1, 1), (2, 3, 4, 1, 2), (3, 2, 8, 2, 2), (5, 4, 8, 3, 3), (7, 8, 16, 3, 2), (8, 9, 2, 1, 3),
    (13, 14, 8, 1, 1), (14, 13, 8, 2, 2), (16, 5, 16, 3, 1), (27, 6, 8, 3, 2), (28, 29, 4, 2, 3), (65, 3, 8, 3, 2),
    (4, 67, 32, 3, 2),
])
def test_wavelet_sizes(gpu, oracle, M, N, K, levels, cycles, wav):
    d = 8
    rng = np.random.default_rng(M * 100 + N)
    V = np.asfortranarray(rng.uniform(0, 255, (M * d, N * d, K)).astype(np.float32))
    S = np.full((K, M, N), 529, dtype=np.uint32, order="F")
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=d, blockSizeWie=d, matchSize=32, numMax=K, numMin=K, levels=levels, cycleSpin=cycles)
    tau = 25.0 * options.getTau(levels, 1)
    fac = options.bior_factors() if wav == "bior" else options.haar_factors()
    Psi, Psi2 = options.bank_from_factors(fac)
    U, W = gpu.denoiseAndAggregateGPU(V, _as_set(S), tau, Psi, Psi2, o)
    f = oracle.bior_filters() if wav == "bior" else oracle.haar_filters()
    Uo, Wo = oracle.denoiseAndAggregateGPU(V, S, tau, o, filters=f, prec=32)
    assert np.array_equal(U, Uo) and np.array_equal(W, Wo)


@pytest.mark.parametrize("M,N,levels,cycles", [(2, 2, 1, 2), (3, 5, 2, 3), (9, 7, 3, 2), (29, 8, 3, 1), (8, 33, 2, 2)])
def test_video_wavelet_sizes(gpu, oracle, M, N, levels, cycles):
    d, K, F = 8, 8, 3
    rng = np.random.default_rng(M * 10 + N)
    V = np.asfortranarray(rng.uniform(0, 1, (M * d, N * d, K)).astype(np.float32))
    S = np.asfortranarray(rng.integers(1, d * d * F + 1, (K, M, N)).astype(np.uint32))
    o = dict(blockSize=d, numMax=K, numMin=K, levels=levels, cycleSpin=cycles, nF=F)
    U, out = api.denoiseAndAggregateV(None, V, np.zeros((M * d, N * d, F)), S, 0.1, o)
    tau = np.asfortranarray(0.1 * options.getTau(levels, 2))
    Uo, Wo = oracle.denoiseAndAggregateV(V, S, d, F, tau, levels, cycles, prec=32)
    assert np.array_equal(U, Uo) and np.array_equal(out["K"], Wo)
