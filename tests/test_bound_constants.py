"""The error bound of the f16 matchers with the constants and the formula that the kernels
compile (csrc/bound.cuh is compiled for the host here): every member of the exact top K lies
within the threshold derived from the K-th best rounded distance, for 8 x 8 and 32 x 32
patches, when the computed distances are off by the largest errors that the bound allows.
The constants cover the sums they are derived from."""
import ctypes as C
import os
import re
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BOUND = os.path.join(ROOT, "gbm3d_b200", "csrc", "bound.cuh")


def _source():
    with open(BOUND) as f:
        return f.read()


def constants(name):
    body = re.search(r"struct " + name + r" \{[^}]*\}", _source()).group(0)
    return {k: float(v) for k, v in re.findall(r"(\w+) = ([0-9.e+-]+)f", body)}


@pytest.fixture(scope="module")
def threshold(tmp_path_factory):
    """candidate_threshold() and the two constant sets as a host library."""
    src = _source()
    parts = [re.search(r"struct " + n + r" \{.*?\n\};", src, re.S).group(0) for n in ("Bound8", "Bound32")]
    fn = re.search(r"template <class B>\n__device__ __forceinline__ float candidate_threshold.*?\n\}", src, re.S).group(0)
    d = tmp_path_factory.mktemp("bound")
    (d / "b.cpp").write_text("#include <cmath>\nusing std::sqrt;\nstatic inline float sqrtf_(float x) { return std::sqrt(x); }\n"
                             "static inline float fmaxf_(float a, float b) { return a > b ? a : b; }\n"
                             "#define sqrtf sqrtf_\n#define fmaxf fmaxf_\n" + "\n".join(parts) + "\n"
                             + fn.replace("__device__ __forceinline__", "static")
                             + '\nextern "C" float t8(float T, float nx) { return candidate_threshold<Bound8>(T, nx); }'
                             '\nextern "C" float t32(float T, float nx) { return candidate_threshold<Bound32>(T, nx); }\n')
    lib = str(d / "b.so")
    subprocess.run(["g++", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-o", lib, str(d / "b.cpp")], check=True)
    L = C.CDLL(lib)
    for f in (L.t8, L.t32):
        f.restype, f.argtypes = C.c_float, [C.c_float, C.c_float]
    return {8: L.t8, 32: L.t32}


@pytest.mark.parametrize("name,side,steps,addends,largest,norm_adds",
                         [("Bound8", 8, 8, 9, 2, 6), ("Bound32", 32, 96, 17, 1, 64)])
def test_constants_cover_their_sums(name, side, steps, addends, largest, norm_adds):
    c = constants(name)
    # two roundings of side^2 subnormal parts of 2^-25 each
    assert c["ETA2"] >= 2 * side * 2.0 ** -25
    # 2 v: each step's nonzero addends truncated at 2^-23 of the largest, which is a sum of products
    # (at most (||x||^2 + ||w||^2) / 2), at patch 8 less ||w||^2 / 2, where the sums start; and the
    # FP32 sums of the squared norms
    assert c["KAPPA"] >= largest * steps * addends * 2.0 ** -23 + norm_adds * 2.0 ** -24
    # r from the serial chain of side^2 squares of rounded differences
    assert c["GAMMA2"] >= (side * side + 3) * 2.0 ** -24


@pytest.mark.parametrize("side", [8, 32])
@pytest.mark.parametrize("scale", [1e-7, 1e-3, 1.0, 100.0])
@pytest.mark.parametrize("contrast,noise", [(0.0, 1.0), (50.0, 1.0), (50.0, 0.02), (200.0, 1e-4)])
def test_threshold_keeps_the_exact_top_k(threshold, side, scale, contrast, noise):
    rng = np.random.default_rng(side)
    kappa = constants(f"Bound{side}")["KAPPA"]
    K, n, N = 16, side * side, 1024
    for trial in range(12 if side == 8 else 3):
        base = contrast * rng.standard_normal(n) + 30 * rng.standard_normal()
        w = ((base + noise * rng.standard_normal((N, n))) * scale).astype(np.float32)
        x = ((base + noise * rng.standard_normal(n)) * scale).astype(np.float32)
        if max(np.abs(x).max(), np.abs(w).max()) >= 60000:
            continue  # beyond f16: searched exhaustively
        exact = np.zeros(N, np.float32)
        for k in range(n):  # the serial FP32 chain of the ranking
            t = x[k] - w[:, k]
            exact = (t.astype(np.float64) ** 2 + exact).astype(np.float32)
        x16, w16 = x.astype(np.float16).astype(np.float64), w.astype(np.float16).astype(np.float64)
        nx, nw = (x16 ** 2).sum(), (w16 ** 2).sum(1)
        d = ((x16 - w16) ** 2).sum(1)
        top = np.argsort(exact, kind="stable")[:K]
        sign = rng.choice([-1.0, 1.0], N)
        if trial % 3 == 0:  # the worst case: the top K off to the far side, all others to the near one
            sign[:] = -1.0
            sign[top] = 1.0
        d = d + kappa * (nx + nw) * sign
        theta = threshold[side](np.sort(d)[K - 1], nx)
        assert np.all(d[top] <= theta)
