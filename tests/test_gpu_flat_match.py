"""Windows of one value (an empty border, a mask, saturation) in the bounded matchers, where
every distance is zero: alone, beside textured windows, one value off in a window's corner, at
the ends of the value range, next to the grid's end; against the oracle."""
import numpy as np
import pytest

from gbm3d_b200 import options, synth

pytestmark = pytest.mark.gpu


def _part_flat(m, n, value, r0, c0):
    I = synth.noisy_image(m, n, 25.0, seed=m + n)[1]
    I[r0:, c0:] = value
    return I


@pytest.mark.parametrize("value", [0.0, 90.1, 1e-30, -3.7, 5e4, 1e30])
@pytest.mark.parametrize("m,n,s,K,r0,c0", [(96, 131, 8, 16, 0, 0), (120, 140, 3, 32, 10, 21), (90, 121, 7, 1, 0, 40),
                                           (110, 130, 5, 8, 33, 0)])
def test_flat_windows(gpu, oracle, value, m, n, s, K, r0, c0):
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=8, blockSizeWie=8, matchSize=32, refStride=s, refStrideWie=s, numMax=K, numMin=K)
    I = _part_flat(m, n, value, r0, c0)
    for odd in (False, True):
        if odd:  # the smallest change of one pixel, at a window's last row and column
            f = np.float32(value)
            I[72 if m > 100 else 38, 77] = np.nextafter(f, np.float32(np.inf)) if f else np.float32(1e-45)
        S, V = gpu.matchBlocksCPU(I, 25.0, o)
        So, Vo, co = oracle.matchBlocksCPU(I, 25.0, o, prec=32)
        assert np.array_equal(np.asarray(S), So) and np.array_equal(S.count, co) and np.array_equal(V, Vo)


@pytest.mark.parametrize("value", [0.0, 0.7, 1e-30])
@pytest.mark.parametrize("m,n,F,K,r0", [(96, 96, 3, 16, 0), (128, 64, 5, 32, 40), (100, 70, 3, 1, 30)])
def test_flat_video_windows(gpu, oracle, value, m, n, F, K, r0):
    from gbm3d_b200 import api
    I = np.stack([_part_flat(m, n, value, r0, 0) for _ in range(F)], axis=2)
    for odd in (False, True):
        if odd:  # one pixel of the last frame
            f = np.float32(value)
            I[r0 + 20, 20, F - 1] = np.nextafter(f, np.float32(np.inf)) if f else np.float32(1e-45)
        S, V = api.matchBlocksV(I, 0.1, {"blockSize": 32, "numMax": K, "numMin": K, "nF": F})
        So, Vo = oracle.matchBlocksV(I, 32, K, prec=32)
        assert np.array_equal(np.asarray(S), So) and np.array_equal(V, Vo)
