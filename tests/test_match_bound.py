"""Block matching at patch 8 / search 32 with f16 tensor-core distances as a
bound (csrc/match_bound.cu): the match sets and the gathered volume equal the
exhaustive search's (the oracle's), bit for bit, wherever the bound can go
wrong: strides 1 to 8, grids whose last tile of four references is partial,
small and large value ranges (f16 subnormals, f16 overflow), smooth images
whose distances nearly tie, flat ones whose lists overflow, every group size.
"""
import numpy as np
import pytest

from gbm3d_b200 import options, synth


def _opts(s=8, K=16, **kw):
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=8, blockSizeWie=8, matchSize=32, refStride=s, refStrideWie=s, numMax=K, numMin=K)
    o.update(kw)
    return o


def _image(kind, m, n, seed):
    clean, noisy = synth.noisy_image(m, n, 25.0, seed=seed)
    if kind == "noisy":
        return noisy
    if kind == "unit":          # the [0, 1] scale
        return noisy / 255.0
    if kind == "tiny":          # f16 subnormals after centring
        return noisy * 1e-7
    if kind == "overflow":      # centred values beyond the f16 range
        return noisy * 2000.0
    if kind == "smooth":        # a step-2 pilot: distances nearly tie
        return clean + 0.02 * np.cos(np.arange(m)[:, None] / 7.0) * np.arange(n)[None, :] % 3
    if kind == "flat":          # every distance ties
        return np.full((m, n), 90.0)
    step = np.full((m, n), 90.0)  # a mix of tied and distinct distances
    step[m // 3:m // 2, n // 4:] = 140.0
    return step + 1e-3 * (noisy - clean)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,m,n,s,K", [
    ("noisy", 64, 72, 8, 16), ("noisy", 57, 61, 1, 16), ("noisy", 80, 67, 2, 16), ("noisy", 96, 75, 3, 16),
    ("noisy", 70, 81, 4, 16), ("noisy", 68, 90, 5, 16), ("noisy", 100, 77, 6, 16), ("noisy", 64, 99, 7, 16),
    ("noisy", 64, 40, 8, 1), ("noisy", 64, 48, 8, 8), ("noisy", 64, 56, 3, 32), ("noisy", 32, 32, 8, 16),
    ("unit", 72, 67, 3, 16), ("tiny", 64, 64, 8, 16), ("overflow", 64, 70, 3, 16), ("smooth", 96, 90, 7, 16),
    ("smooth", 90, 96, 3, 32), ("flat", 64, 64, 8, 16), ("step", 96, 88, 3, 16), ("step", 96, 88, 8, 8),
])
def test_bounded_matching_equals_the_exhaustive_search(gpu, oracle, kind, m, n, s, K):
    I = _image(kind, m, n, seed=m + n + s)
    o = _opts(s, K)
    S, V = gpu.matchBlocksCPU(I, 25.0, o)
    So, Vo, co = oracle.matchBlocksCPU(I, 25.0, o, prec=32)
    assert np.array_equal(np.asarray(S), So), f"{int((np.asarray(S) != So).any(axis=0).sum())} match sets differ"
    assert np.array_equal(S.count, co) and np.array_equal(V, Vo)


def _threshold(T, nx):
    """candidate_threshold() of csrc/match_bound.cu in float32."""
    f = np.float32
    U, ETA2, KAPPA, GAMMA2 = f(4.8852e-4), f(4.8e-7), f(2.2e-5), f(1.0e-5)
    X = np.sqrt(nx) * (f(1) + f(2) * U) + ETA2
    A = np.sqrt((np.maximum(T, f(0)) + f(3) * KAPPA * nx) * (f(1) + f(3) * KAPPA))
    R = (A + f(2) * U * X + ETA2) * (f(1) + f(2) * U) * (f(1) + GAMMA2)
    R16 = R * (f(1) + U) + f(2) * U * X + ETA2
    return (R16 * R16 * (f(1) + f(2) * KAPPA) + f(3) * KAPPA * nx) * (f(1) + f(1e-6))


@pytest.mark.parametrize("scale", [1e-7, 1e-3, 1.0, 100.0])
@pytest.mark.parametrize("contrast,noise", [(0.0, 1.0), (50.0, 1.0), (50.0, 0.02), (200.0, 1e-4)])
def test_threshold_keeps_the_exact_top_k(scale, contrast, noise):
    """Patches around a common structure, rounded to f16: every member of the
    exact top K lies within the threshold derived from the K-th best rounded
    distance, also when that distance is off by the largest error allowed."""
    rng = np.random.Generator(np.random.PCG64(5))
    K = 16
    for _ in range(40):
        base = contrast * rng.standard_normal(64) + 30 * rng.standard_normal()
        w = ((base + noise * rng.standard_normal((1024, 64))) * scale).astype(np.float32)
        x = ((base + noise * rng.standard_normal(64)) * scale).astype(np.float32)
        exact = np.zeros(1024, np.float32)
        for k in range(64):  # serial FP32 chain
            t = x[k] - w[:, k]
            exact = (t.astype(np.float64) ** 2 + exact).astype(np.float32)
        if max(np.abs(x).max(), np.abs(w).max()) >= 60000:
            continue  # the kernel's f16 overflow guard: searched exhaustively
        x16, w16 = x.astype(np.float16).astype(np.float64), w.astype(np.float16).astype(np.float64)
        d = ((x16 - w16) ** 2).sum(1)
        nx, nw = (x16 ** 2).sum(), (w16 ** 2).sum(1)
        d = d + 1.9e-5 * (nx + nw) * rng.choice([-1.0, 1.0], 1024)  # the MMA's error at its bound
        theta = _threshold(np.float32(np.sort(d)[K - 1]), np.float32(nx))
        top = np.argsort(exact, kind="stable")[:K]
        assert np.all(d[top] <= theta)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,m,n,F,K", [
    ("noisy", 64, 96, 3, 16), ("noisy", 96, 64, 5, 8), ("noisy", 64, 64, 7, 32), ("noisy", 64, 64, 9, 16),
    ("noisy", 64, 96, 11, 1), ("noisy", 64, 64, 13, 16), ("smooth", 96, 96, 3, 16), ("tiny", 64, 64, 3, 16),
    ("overflow", 64, 64, 3, 16), ("flat", 64, 96, 3, 16), ("step", 96, 96, 3, 16),
])
def test_bounded_video_matching_equals_the_direct_search(gpu, oracle, kind, m, n, F, K):
    """Patch 32 (csrc/video_bound.cu): windows of 3 to 11 frames, and one beyond."""
    from gbm3d_b200 import api
    base = _image(kind, m, n, seed=m + F)
    I = np.stack([np.roll(base, f, axis=0) + (0 if kind in ("flat", "step") else f * 1e-3 * base) for f in range(F)], axis=2)
    S, V = api.matchBlocksV(I, 0.1, {"blockSize": 32, "numMax": K, "numMin": K, "nF": F})
    So, Vo = oracle.matchBlocksV(I, 32, K, prec=32)
    assert np.array_equal(np.asarray(S), So), f"{int((np.asarray(S) != So).any(axis=0).sum())} match sets differ"
    assert np.array_equal(V, Vo)
