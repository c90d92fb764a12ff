"""Colour images whose group columns, laid side by side, are more than 65535:
the interior columns of such an image equal those of its right-hand crop (group
grid, search windows and wavelet filters are local; the crop starts on a
reference column)."""
import numpy as np
import pytest

from gbm3d_b200 import options, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,s,d2", [(24600, 3, 32), (8300, 1, 16)])
def test_wide_colour_image(gpu, n, s, d2):
    from gbm3d_b200 import api
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=8, blockSizeWie=8, matchSize=d2, refStride=s, refStrideWie=s)
    m, c0, edge = 32, 3 * (n // 4), 300
    x = np.stack([np.tile(synth.noisy_image(m, 500, 25.0, seed=q)[1], (1, n // 500 + 1))[:, :n] for q in range(3)], axis=2)
    x = x + np.random.default_rng(1).standard_normal(x.shape)
    wide, crop = api.GBM3D_rgb(x, 25.0, o), api.GBM3D_rgb(x[:, c0:], 25.0, o)
    assert wide.shape == x.shape
    assert np.array_equal(wide[:, c0 + edge:n - edge], crop[:, edge:-edge])
