"""Split exhaustive matching of large patches (csrc/match.cu, k_match_split)
against the oracle: the largest number of references that takes it, one more
(one warp per reference), partial searches and the tolerance branch."""
import numpy as np
import pytest

from gbm3d_b200 import options, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,d,s,d2,numMin", [
    (256, 296, 16, 16, 32, 16),   # 288 references: split
    (16 * 37, 128, 16, 16, 32, 16),  # 296: the last split size
    (16 * 27, 176, 16, 16, 32, 16),  # 297: one warp per reference
    (96, 80, 16, 5, 24, 16), (64, 64, 16, 16, 16, 16), (70, 90, 32, 8, 32, 16), (64, 96, 32, 32, 24, 16),
    (96, 96, 16, 16, 32, 4),
])
def test_split_matching(gpu, oracle, m, n, d, s, d2, numMin):
    _, noisy = synth.noisy_image(m, n, 10.0, seed=m + n)
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=d, matchSize=d2, refStride=s, numMin=numMin)
    S, V = gpu.matchBlocksCPU(noisy, 10.0, o)
    So, Vo, co = oracle.matchBlocksCPU(noisy, 10.0, o, prec=32)
    assert np.array_equal(np.asarray(S), So) and np.array_equal(S.count, co) and np.array_equal(V, Vo)
