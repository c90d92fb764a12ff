"""The tcgen05 matcher's own sets against the oracle, at every search size: at 32 a wait
limit selects it (a call without one takes the bounded matcher), and an image whose candidate
lists overflow sends its references to the exhaustive list kernel."""
import numpy as np
import pytest

from gbm3d_b200 import options, synth

pytestmark = pytest.mark.gpu


def _image(kind, m, n):
    if kind == "noisy":
        return synth.noisy_image(m, n, 25.0, seed=m + n)[1]
    I = np.full((m, n), 90.0)
    if kind == "step":  # flat parts overflow their lists, the edge's references do not
        I[m // 3:2 * m // 3, n // 4:n // 2] = 140.0
        I += 1e-3 * np.random.default_rng(3).standard_normal((m, n)) * (np.arange(n) > 2 * n // 3)
    return I


@pytest.mark.parametrize("form", ["precision", "tensor"])
@pytest.mark.parametrize("kind,m,n,d2,s", [
    ("noisy", 96, 104, 16, 3), ("noisy", 96, 104, 24, 5), ("noisy", 96, 104, 32, 3), ("noisy", 104, 96, 32, 8),
    ("noisy", 90, 75, 32, 7), ("noisy", 64, 72, 32, 1), ("step", 96, 104, 16, 8), ("step", 96, 104, 24, 3),
    ("step", 96, 104, 32, 8), ("step", 96, 104, 32, 3), ("flat", 64, 72, 32, 8),
])
def test_tcgen05_match_sets(gpu, oracle, form, kind, m, n, d2, s):
    I = _image(kind, m, n)
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=8, blockSizeWie=8, matchSize=d2, refStride=s, refStrideWie=s, form=form)
    ctx = gpu.context()
    ctx.tc_stats(True)
    ctx.set_tc_wait(4_000_000_000)  # the default limit, stated
    try:
        S, V = gpu.matchBlocksCPU(I, 25.0, o)
    finally:
        ctx.set_tc_wait(0)
        hist = ctx.tc_stats(False)
    assert sum(hist) == S.shape[1] * S.shape[2]  # this kernel made them
    So, Vo, co = oracle.matchBlocksCPU(I, 25.0, dict(o, form="plain"), prec=32)
    assert np.array_equal(np.asarray(S), So) and np.array_equal(S.count, co) and np.array_equal(V, Vo)
