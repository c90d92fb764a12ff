"""Cycle spins that share the launches of the coarse wavelet levels: any number
of them, their results and their workspace."""
import numpy as np
import pytest

from gbm3d_b200 import options
from gbm3d_b200.api import _as_set

pytestmark = pytest.mark.gpu


def test_more_spins_than_a_launch_can_hold(gpu, oracle):
    """8200 spins of 8 slot pairs at the second level: more than 65535 slices of a grid."""
    d, K, levels, cycles = 8, 32, 2, 8200
    V = np.asfortranarray(np.random.default_rng(2).uniform(0, 255, (d, d, K)).astype(np.float32))
    S = np.full((K, 1, 1), 529, dtype=np.uint32, order="F")
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=d, blockSizeWie=d, matchSize=32, numMax=K, numMin=K, levels=levels, cycleSpin=cycles)
    tau = 25.0 * options.getTau(levels, 1)
    Psi, Psi2 = options.bank_from_factors(options.haar_factors())
    U, W = gpu.denoiseAndAggregateGPU(V, _as_set(S), tau, Psi, Psi2, o)
    Uo, Wo = oracle.denoiseAndAggregateGPU(V, S, tau, o, filters=oracle.haar_filters(), prec=32)
    assert np.array_equal(U, Uo) and np.array_equal(W, Wo)
