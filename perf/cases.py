"""Performance cases: the work that users have this library do, through its
public entry points, from the smallest calls to the largest.

A case is a dict of plain values:

  kind    "grey"    one image resident on the device      api.GBM3D_device
          "host"    one image in host memory, whole call  api.GBM3D
          "stream"  one pinned host image of a stream     api.GBM3D_async
          "rgb"     one colour image on the device        api.GBM3D_mixed
          "video"   a device video through VBM3D          api.GBM3D_mixed
          "batch"   uneven images as one CUDA graph       api.GBM3D_mixed
  m, n    rows and columns; sigma the noise on the 0-255 scale
  config  a reference profile ("default", "fast", "accuracy"), "dense" (patch
          8 at stride 3, the benchmark's workload) or "tuned" (the calibrated
          profile for the image's size and noise)
  form    "plain", "tensor" or "precision"

listed() and draw() give cases, prepare() and run() execute one, work() counts
the bytes and operations that no implementation can leave out, and exact()
restates the algorithm in 64 bits with plain torch operations.
"""
import math
import random

import torch

from gbm3d_b200 import api, options
from gbm3d_b200._lib import Context

K = 16  # group size of every option set used here


def _case(name, kind, m, n, sigma, config, form="plain", **more):
    return dict(name=name, kind=kind, m=m, n=n, sigma=float(sigma), config=config, form=form, **more)


def listed():
    return [
        # the smallest whole denoise: a thumbnail with the reference's default
        # profile, where launches and host work count as much as kernels
        _case("grey-128x96-default", "grey", 128, 96, 25, "default"),
        # the smallest image of the mixed batch workload, odd on both sides
        _case("grey-301x203-tuned", "grey", 301, 203, 25, "tuned"),
        # the drop-in call of a MATLAB or numpy user: host arrays in and out,
        # the reference's default profile on a photo-sized image
        _case("host-512-default", "host", 512, 512, 25, "default"),
        # the dense configuration on a mid-sized image at low noise
        _case("grey-1024-dense-s10", "grey", 1024, 1024, 10, "dense"),
        # a ragged size of the mixed workload; its class keeps stride 3
        _case("grey-1677x1531-tuned-s11", "grey", 1677, 1531, 11.4, "tuned"),
        # the benchmark's chosen form: a 16-megapixel image, calibrated options
        _case("grey-4096-tuned", "grey", 4096, 4096, 25, "tuned"),
        # the benchmark's plain workload: the largest call
        _case("grey-4096-dense", "grey", 4096, 4096, 25, "dense"),
        # one image of a stream through pinned host buffers, copies overlapped
        _case("stream-2048-tuned", "stream", 2048, 2048, 25, "tuned"),
        # the same option class with tensor-core matching
        _case("grey-2048-tensor", "grey", 2048, 2048, 25, "tuned", form="tensor"),
        # a colour image: luma-driven matching, three filtered channels
        _case("rgb-1024-tuned", "rgb", 1024, 1024, 25, "tuned"),
        # 720p video through VBM3D's defaults (patch 32) with a 3-frame window
        _case("video-720p-8f", "video", 720, 1280, 25, "video", frames=8, patch=32),
        # a batch server's submission: uneven grey and colour images, each with
        # its own option set, replayed as one CUDA graph on four lanes
        _case("batch-8grey-2rgb", "batch", 900, 700, 25, "tuned", grey=8, rgb=2, layout=1),
    ]


def _side(rng, lo, hi):
    """A side between lo and hi, uniform in its logarithm."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(max(v, lo), hi)


def draw(rng):
    kind = rng.choice(["grey"] * 6 + ["host", "stream", "rgb", "video", "batch"])
    sigma = round(rng.uniform(5, 50), 2)
    if kind == "grey":
        config, form = rng.choice([("default", "plain"), ("fast", "plain"), ("accuracy", "plain"), ("dense", "plain"),
                                   ("tuned", "plain"), ("tuned", "plain"), ("tuned", "tensor"), ("tuned", "precision")])
        hi = {"tuned": 4096 if form == "plain" else 2048, "dense": 2048}.get(config, 1024)
        lo = 200 if config == "tuned" else 96
        c = _case("", kind, _side(rng, lo, hi), _side(rng, lo, hi), sigma, config, form)
    elif kind == "host":
        c = _case("", kind, _side(rng, 96, 768), _side(rng, 96, 768), sigma, rng.choice(["default", "fast"]))
    elif kind == "stream":
        c = _case("", kind, _side(rng, 512, 3000), _side(rng, 512, 3000), sigma, "tuned")
    elif kind == "rgb":
        c = _case("", kind, _side(rng, 200, 1024), _side(rng, 200, 1024), sigma, rng.choice(["tuned", "dense"]))
    elif kind == "video":
        c = _case("", kind, _side(rng, 96, 720), _side(rng, 128, 1280), sigma, "video", frames=rng.randint(4, 8),
                  patch=rng.choice([16, 32, 32]))
    else:
        c = _case("", kind, _side(rng, 300, 1200), _side(rng, 300, 1200), sigma, "tuned", grey=rng.randint(3, 10),
                  rgb=rng.randint(0, 2), layout=rng.randint(1, 10 ** 6))
    del c["name"]
    return c


def _opts(case):
    c = case["config"]
    if c == "dense":
        o = dict(options.setBM3Dopts("default"), **options.DENSE)
        o["form"] = case["form"]
        return o
    return {"profile": c, "form": case["form"]} if c == "tuned" else {"profile": c}


def _video_opts(case):
    return {"nF": 3, "blockSize": case["patch"]}


def _batch_items(case):
    """(grey sizes and sigmas, colour sizes and sigmas) of a batch: sides from
    a third to the whole of (m, n), noise between 5 and 50."""
    rng = random.Random(case["layout"])

    def item():
        return (max(200, int(case["m"] * rng.uniform(0.33, 1.0))), max(200, int(case["n"] * rng.uniform(0.33, 1.0))),
                round(rng.uniform(5, 50), 2))

    return [item() for _ in range(case["grey"])], [item() for _ in range(case["rgb"])]


# ---- inputs -----------------------------------------------------------------------

def _noisy(m, n, sigma, seed, shift=(0.0, 0.0)):
    """A noisy m x n image on the device, 0-255 scale: a gradient, 40 ellipses
    and 3 sinusoidal textures plus white noise.  Stored as a contiguous (n, m)
    float64 tensor, which is the column-major m x n array the library takes."""
    rng = random.Random(seed)
    y = torch.arange(m, device="cuda", dtype=torch.float64)[None, :]
    x = torch.arange(n, device="cuda", dtype=torch.float64)[:, None]
    img = rng.uniform(40, 120) + rng.uniform(-60, 60) * y / max(m - 1, 1) + rng.uniform(-60, 60) * x / max(n - 1, 1)
    for _ in range(40):
        cy, cx, ry, rx = rng.uniform(0, m), rng.uniform(0, n), rng.uniform(0.02, 0.2) * m, rng.uniform(0.02, 0.2) * n
        th, val, vy, vx = rng.uniform(0, math.pi), rng.uniform(0, 255), rng.uniform(-3, 3), rng.uniform(-3, 3)
        dy, dx = y - (cy + vy * shift[0]), x - (cx + vx * shift[1])
        c, s = math.cos(th), math.sin(th)
        inside = ((dy * c + dx * s) / ry) ** 2 + ((dx * c - dy * s) / rx) ** 2 <= 1.0
        img = torch.where(inside, torch.full_like(img, val), img)
    for _ in range(3):
        h, w = int(rng.uniform(0.1, 0.3) * m) + 1, int(rng.uniform(0.1, 0.3) * n) + 1
        y0, x0 = rng.randint(0, max(m - h, 1) - 1), rng.randint(0, max(n - w, 1) - 1)
        period, th, amp, base = rng.uniform(4, 16), rng.uniform(0, math.pi), rng.uniform(20, 60), rng.uniform(60, 190)
        phase = 2 * math.pi * (y[:, :h] * math.cos(th) + x[:w] * math.sin(th)) / period
        img[x0:x0 + w, y0:y0 + h] = base + amp * torch.sin(phase)
    gen = torch.Generator(device="cuda").manual_seed(seed * 1009 + 7 + int(shift[0]))
    return (img.clamp(0, 255) + sigma * torch.randn((n, m), generator=gen, device="cuda", dtype=torch.float64)).contiguous()


def _inputs(case, seed):
    """The case's input tensors: one image, three planes, frames or a batch's lists."""
    m, n, sigma, kind = case["m"], case["n"], case["sigma"], case["kind"]
    if kind == "rgb":
        return [_noisy(m, n, sigma, 3 * seed + q) for q in range(3)]
    if kind == "video":
        return torch.stack([_noisy(m, n, sigma, seed, shift=(f, f)) for f in range(case["frames"])]) / 255.0
    if kind == "batch":
        grey, rgb = _batch_items(case)
        return ([_noisy(a, b, s, 101 * seed + k) for k, (a, b, s) in enumerate(grey)],
                [tuple(_noisy(a, b, s, 101 * seed + 31 + 3 * k + q) for q in range(3)) for k, (a, b, s) in enumerate(rgb)])
    return _noisy(m, n, sigma, seed)


def prepare(case, seed):
    kind, x = case["kind"], _inputs(case, seed)
    st = dict(case=case, x=x, opts=_opts(case) if kind != "video" else None)
    if kind == "grey":
        st["out"] = torch.empty_like(x)
    elif kind == "host":
        st["x"] = x.cpu().numpy().T  # m x n, column-major
    elif kind == "stream":
        st["x"] = x.cpu().pin_memory()
        st["out"] = torch.empty(x.shape, dtype=torch.float64).pin_memory()
    elif kind == "rgb":
        st["out"] = tuple(torch.empty_like(p) for p in x)
    elif kind == "video":
        st["vopts"] = _video_opts(case)
        st["out"] = torch.empty((case["frames"] - 2,) + tuple(x.shape[1:]), dtype=torch.float64, device="cuda")
    else:
        # the graph belongs to the context a batch server keeps for this batch
        st["ctx"] = Context(0)
        st["ctx"].set_lanes(4)
        st["out"] = ([torch.empty_like(v) for v in x[0]], [tuple(torch.empty_like(p) for p in t) for t in x[1]], None)
    torch.cuda.synchronize()
    return st


def run(st):
    c, x = st["case"], st["x"]
    m, n, sigma, kind = c["m"], c["n"], c["sigma"], c["kind"]
    if kind == "grey":
        api.GBM3D_device(x.data_ptr(), m, n, sigma, st["out"].data_ptr(), st["opts"])
        return st["out"]
    if kind == "host":
        U, out = api.GBM3D(x, sigma, st["opts"])
        return [U, out["U1"]]
    if kind == "stream":
        api.GBM3D_async(x.data_ptr(), m, n, sigma, st["out"].data_ptr(), st["opts"])
        return st["out"]
    if kind == "rgb":
        _, out, _ = api.GBM3D_mixed(rgb=[x], rgb_sigma=[sigma], opts=st["opts"], use_graph=False,
                                    outputs=([], [st["out"]], None))
        return list(out[0])
    if kind == "video":
        return api.GBM3D_mixed(video=x, video_sigma=sigma / 255.0, vopts=st["vopts"], use_graph=False,
                               outputs=([], [], st["out"]))[2]
    grey, rgb = _batch_items(c)
    g, r, _ = api.GBM3D_mixed(x[0], [s for _, _, s in grey], x[1], [s for _, _, s in rgb], opts=st["opts"],
                              ctx=st["ctx"], outputs=st["out"])
    return list(g) + [p for t in r for p in t]


# ---- work -------------------------------------------------------------------------

def _resolved(case, m, n, sigma):
    return options.resolve_opts(_opts(case), shape=(m, n), sigma=sigma)


def _image_work(o, m, n, channels=1):
    """Image in and out once (float64); per reference block the d2^2 squared
    distances (3 operations per pixel), per group the transforms there and
    back and the weighted sums of its K blocks."""
    d, dw, w2 = o["blockSize"], o["blockSizeWie"], o["matchSize"] ** 2
    s1, s2 = options.strides(o)
    mp, np_ = _padded(m, o), _padded(n, o)
    g1 = options.grid_count(mp, d, s1) * options.grid_count(np_, d, s1) * len(o["matchSpins"])
    flops = g1 * (3 * w2 * d * d + channels * K * d * d * (o["cycleSpin"] * 2 * 2 * 14 * 8 / 7 + 4))
    if o["Wiener"]:
        g2 = options.grid_count(mp, dw, s2) * options.grid_count(np_, dw, s2) * len(o["matchSpinsWie"])
        flops += g2 * (3 * w2 * dw * dw + channels * K * dw * dw * (3 * (4 * dw + 6) + 10))
    return {"bytes": 16.0 * m * n * channels, "flops": float(flops)}


def work(case):
    m, n, sigma, kind = case["m"], case["n"], case["sigma"], case["kind"]
    if kind == "batch":
        grey, rgb = _batch_items(case)
        ws = [_image_work(_resolved(case, *it), it[0], it[1]) for it in grey]
        ws += [_image_work(_resolved(case, *it), it[0], it[1], 3) for it in rgb]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if kind == "video":
        d, frames = case["patch"], case["frames"]
        g = math.ceil(m / d) * math.ceil(n / d) * (frames - 2) * 2  # two match spins
        flops = g * (3 * 3 * d ** 4 + K * d * d * (2 * 2 * 2 * 18 * 8 / 7 + 4))
        return {"bytes": 8.0 * m * n * (2 * frames - 2), "flops": float(flops)}
    w = _image_work(_resolved(case, m, n, sigma), m, n, 3 if kind == "rgb" else 1)
    if kind == "host":
        w["bytes"] += 8.0 * m * n  # the step-1 estimate is returned too
    return w


# ---- the same results in 64 bits ----------------------------------------------------
# Images are m x n float64 device tensors here (row index first).  The search
# of a block runs over the d2 x d2 offsets of the circularly padded image; the
# groups pass a 3D wavelet hard threshold (step 1) or a DCT x Haar Wiener gain
# (step 2) and are averaged with their weights.

def _padded(L, o):
    d, dw = o["blockSize"], o["blockSizeWie"]
    s1, s2 = options.strides(o)
    if s1 == d and (not o["Wiener"] or (s2 == dw and d % dw == 0)):
        return -(-L // d) * d
    p = max(L, d, dw)
    while (p - d) % s1 or (o["Wiener"] and (p - dw) % s2):
        p += 1
    return p


def _mirror(img, M, N):
    m, n = img.shape
    r = torch.cat([torch.arange(m), m - 1 - torch.arange(M - m)]).to(img.device)
    c = torch.cat([torch.arange(n), n - 1 - torch.arange(N - n)]).to(img.device)
    return img[r][:, c]


def _search_index(L, d2, device):
    """Image row (column) that each row (column) of the search image holds."""
    h = d2 // 2
    r = torch.arange(L + d2, device=device)
    return torch.where(r < h, r + h, (r - h) % L)


def _search_image(img, d2):
    return img[_search_index(img.shape[0], d2, img.device)][:, _search_index(img.shape[1], d2, img.device)]


def _smallest(dist, k):
    """Indices of the k smallest per row, ties by index, in row chunks."""
    out = torch.empty((dist.shape[0], k), dtype=torch.int64, device=dist.device)
    for a in range(0, dist.shape[0], 1 << 17):
        out[a:a + (1 << 17)] = torch.sort(dist[a:a + (1 << 17)], dim=1, stable=True).indices[:, :k]
    return out


def _match(img, d, d2, s):
    """(M N) x K match indices a + b d2; groups ordered i + M j."""
    m, n = img.shape
    M, N = (m - d) // s + 1, (n - d) // s + 1
    pad = _search_image(img, d2)
    dist = torch.empty((M * N, d2 * d2), dtype=torch.float64, device=img.device)
    for b in range(d2):
        for a in range(d2):
            e = (img - pad[a:a + m, b:b + n]).square()
            box = torch.nn.functional.avg_pool2d(e[None, None], d, stride=s, divisor_override=1)[0, 0]
            dist[:, a + b * d2] = box.T.reshape(-1)
    S = _smallest(dist, K)
    S[:, 0] = d2 // 2 + (d2 // 2) * d2
    return S, M, N


def _origins(S, M, N, d2, s):
    g = torch.arange(M * N, device=S.device)
    return (g % M * s)[:, None] + S % d2, (g // M * s)[:, None] + S // d2


def _gather(pad, r0, c0, d):
    """Groups x K x d x d blocks of pad at the origins."""
    t = torch.arange(d, device=pad.device)
    return pad[(r0[..., None] + t)[..., :, None], (c0[..., None] + t)[..., None, :]]


def _scatter(blocks, weights, r0, c0, d, d2, m, n):
    """Sums of weighted blocks and of weights, cropped to the m x n image."""
    t = torch.arange(d, device=r0.device)
    U = torch.zeros((m + d2) * (n + d2), dtype=torch.float64, device=r0.device)
    W = torch.zeros_like(U)
    for a in range(0, r0.shape[0], 1 << 16):
        q = slice(a, a + (1 << 16))
        at = ((r0[q][..., None] + t)[..., :, None] * (n + d2) + (c0[q][..., None] + t)[..., None, :]).reshape(-1)
        w = weights[q].expand_as(blocks[q])
        U.index_add_(0, at, (blocks[q] * w).reshape(-1))
        W.index_add_(0, at, w.reshape(-1))
    h = d2 // 2
    return tuple(v.view(m + d2, n + d2)[h:h + m, h:h + n] for v in (U, W))


def _window(d, lo, hi, device):
    v = torch.sin(math.pi * torch.linspace(lo, hi, d, dtype=torch.float64, device=device))
    return v[:, None] * v[None, :]


_C = math.sqrt(0.5)
_HAAR = ([_C, _C], [-_C, _C])
_CA, _CB = 0.016572815184060, 0.121533978016438
_BIOR = {"a": ([_CA, -_CA, -_CB, _CB, _C, _C, _CB, -_CB, -_CA, _CA], [0, 0, 0, 0, -_C, _C, 0, 0, 0, 0]),
         "s": ([0, 0, 0, 0, _C, _C, 0, 0, 0, 0], [-_CA, -_CA, _CB, _CB, -_C, _C, -_CB, -_CB, _CA, _CA])}
_SYM_LO = [-0.07576571478927333, -0.02963552764599851, 0.49761866763201545, 0.8037387518059161,
           0.29785779560527736, -0.09921954357684722, -0.012603967262037833, 0.0322231006040427]
_SYM = (_SYM_LO, [(1 if k % 2 else -1) * _SYM_LO[7 - k] for k in range(8)])
_SYM = {"a": _SYM, "s": _SYM}


def _down(u, h, axis):
    out = None
    even = [slice(None)] * u.ndim
    even[axis] = slice(0, None, 2)
    for k, v in enumerate(h):
        if v:
            t = torch.roll(u, k, axis)[tuple(even)] * v
            out = t if out is None else out + t
    return out


def _up(c, g, axis):
    shape = list(c.shape)
    shape[axis] *= 2
    up = torch.zeros(shape, dtype=c.dtype, device=c.device)
    even = [slice(None)] * c.ndim
    even[axis] = slice(0, None, 2)
    up[tuple(even)] = c
    return sum(torch.roll(up, -k, axis) * v for k, v in enumerate(g) if v)


def _threshold_3d(V, bank, tau, level=0):
    """Hard threshold of the circular 3D wavelet coefficients of one level and below."""
    if level == len(tau):
        return V
    column = {1: 0, 2: 1, 4: 2, 3: 3, 5: 4, 6: 5, 7: 6}  # band code fy + 2 fx + 4 fz -> threshold column
    out = 0
    for fz in range(2):
        z = _down(V, _HAAR[fz], 2)
        for fx in range(2):
            x = _down(z, bank["a"][fx], 1)
            for fy in range(2):
                c, code = _down(x, bank["a"][fy], 0), fy + 2 * fx + 4 * fz
                c = _threshold_3d(c, bank, tau, level + 1) if code == 0 else c * (c.abs() > tau[level][column[code]])
                out = out + _up(_up(_up(c, bank["s"][fy], 0), bank["s"][fx], 1), _HAAR[fz], 2)
    return out


def _denoise_3d(V, bank, tau, cycles):
    total = 0
    for s in range(cycles):
        total = total + torch.roll(_threshold_3d(torch.roll(V, (s, s, s), (0, 1, 2)), bank, tau), (-s, -s, -s), (0, 1, 2))
    return (total / cycles).clamp(min=0)


def _tau(sigma, mode):
    rows = []
    for i in range(3):
        base = 3.3 - 0.3 * i
        rows.append([sigma * (base + (0 if mode == 1 or j < 3 else 0.5 if j < 6 else 1.0)) for j in range(7)])
    return rows


def _to_volume(B, M, N, d):
    """Groups (i + M j) x K x d x d -> (M d) x (N d) x K."""
    return B.view(N, M, K, d, d).permute(1, 3, 0, 4, 2).reshape(M * d, N * d, K)


def _to_groups(V, M, N, d):
    return V.view(M, d, N, d, K).permute(2, 0, 4, 1, 3).reshape(M * N, K, d, d)


def _variation(B):
    def diff(x, times, axis):
        return torch.diff(x, times, axis).abs().sum((1, 2, 3))
    return 0.25 * (diff(B, 3, 3) + diff(B, 3, 2)) + diff(B, 1, 1)


def _step1(img, S, M, N, o, sigma, search):
    d, d2, s = o["blockSize"], o["matchSize"], options.strides(o)[0]
    r0, c0 = _origins(S, M, N, d2, s)
    V = _denoise_3d(_to_volume(_gather(search, r0, c0, d), M, N, d), _BIOR, _tau(sigma, 1), o["cycleSpin"])
    B = _to_groups(V, M, N, d)
    w = (1 / (_variation(B) + 2.0 ** -52))[:, None, None, None] * _window(d, 0.1, 0.9, img.device)
    return _scatter(B, w, r0, c0, d, d2, img.shape[0], img.shape[1])


def _haar_slots(B, inverse=False):
    """Circular Haar along the slot axis (1), three levels: details first, approximation last."""
    if not inverse:
        parts, u = [], B
        for _ in range(3):
            parts.append(_down(u, _HAAR[1], 1))
            u = _down(u, _HAAR[0], 1)
        return torch.cat(parts + [u], 1)
    u = B[:, 14:16]
    for lo, hi in ((12, 14), (8, 12), (0, 8)):
        u = _up(B[:, lo:hi], _HAAR[1], 1) + _up(u, _HAAR[0], 1)
    return u


def _step2(pilot, img, S, M, N, o, sigma):
    d, d2, s = o["blockSizeWie"], o["matchSize"], options.strides(o)[1]
    r0, c0 = _origins(S, M, N, d2, s)
    k = torch.arange(d, dtype=torch.float64, device=img.device)
    T = math.sqrt(2 / d) * torch.cos(math.pi * (2 * k[None, :] + 1) * k[:, None] / (2 * d))
    T[0] = math.sqrt(1 / d)
    out, wt = torch.empty((M * N, K, d, d), dtype=torch.float64, device=img.device), []
    sp, sn = _search_image(pilot, d2), _search_image(img, d2)
    for a in range(0, M * N, 1 << 16):
        q = slice(a, a + (1 << 16))
        p = _haar_slots(T @ _gather(sp, r0[q], c0[q], d) @ T.T).square()
        gain = p / (p + sigma * sigma)
        gain[:, 14:, 0, 0] = 1
        v = _haar_slots(_haar_slots(T @ _gather(sn, r0[q], c0[q], d) @ T.T) * gain, inverse=True)
        out[q] = (T.T @ v @ T).clamp(min=0)
        wt.append(gain.square().sum((1, 2, 3)))
    w = _window(d, 0.2, 0.8, img.device) / torch.cat(wt)[:, None, None, None]
    return _scatter(out, w, r0, c0, d, d2, img.shape[0], img.shape[1])


def _exact_images(planes, sigmas, o):
    """Both steps on one or three planes (matching on the first), at their own
    noise levels: the estimates and the step-1 estimates, cropped."""
    m, n = planes[0].shape
    mp, np_ = _padded(m, o), _padded(n, o)
    X = [_mirror(p, mp, np_) for p in planes]
    s1, s2 = options.strides(o)
    spins, wspins = o["matchSpins"], o["matchSpinsWie"]
    back = lambda v, s: torch.roll(v, (-s, -s), (0, 1))  # noqa: E731
    U, W, stale = [0] * len(X), [0] * len(X), 0
    for ii, s in enumerate(spins):
        Y = [torch.roll(x, (s, s), (0, 1)) for x in X]
        S, M, N = _match(Y[0], o["blockSize"], o["matchSize"], s1)
        for q, y in enumerate(Y):
            u, w = _step1(y, S, M, N, o, sigmas[q], _search_image(y, o["matchSize"]))
            U[q], W[q] = U[q] + back(u, s), W[q] + back(w, s)
            if ii >= len(wspins) and o["staleWeights"] and len(X) == 1:
                stale = stale + back(w, s)
    E = [u / w for u, w in zip(U, W)]
    first = [e[:m, :n] for e in E]
    if not o["Wiener"]:
        return first, first
    U, W = [0] * len(X), [stale] * len(X)
    for s in wspins:
        Y, P = ([torch.roll(x, (s, s), (0, 1)) for x in v] for v in (X, E))
        S, M, N = _match(P[0], o["blockSizeWie"], o["matchSize"], s2)
        for q in range(len(X)):
            u, w = _step2(P[q], Y[q], S, M, N, o, sigmas[q])
            U[q], W[q] = U[q] + back(u, s), W[q] + back(w, s)
    return [(u / w)[:m, :n] for u, w in zip(U, W)], first


def _exact_rgb(planes, sigma, o):
    R, G, B = planes
    opp = [(R + G + B) / 3, (R - B) / 2 + 128, (R - 2 * G + B) / 4 + 128]
    (y, u, v), _ = _exact_images(opp, [sigma * math.sqrt(f) for f in (1 / 3, 1 / 2, 3 / 8)], o)
    u, v = u - 128, v - 128
    return [y + u + 2 * v / 3, y - 4 * v / 3, y - u + 2 * v / 3]


def _exact_video(X, sigma, d):
    """VBM3D with a 3-frame window: frames x m x n in, frames - 2 out."""
    F, m, n = X.shape
    mp, np_ = -(-m // d) * d, -(-n // d) * d
    M, N = mp // d, np_ // d
    X = torch.stack([_mirror(f, mp, np_) for f in X])
    g = torch.arange(M * N, device=X.device)
    ref = (3 * d * d) // 2 + d // 2  # the reference block's own index
    total = 0
    for s in (0, d // 2):
        Y, W = torch.zeros_like(X), torch.zeros_like(X)
        for j in range(1, F - 1):
            Z = torch.roll(X[j - 1:j + 2], (s, s), (1, 2))
            pads = torch.stack([_search_image(z, d) for z in Z])
            dist = torch.empty((M * N, 3 * d * d), dtype=torch.float64, device=X.device)
            for f in range(3):
                for b in range(d):
                    for a in range(d):
                        e = (Z[1] - pads[f, a:a + mp, b:b + np_]).square().view(M, d, N, d).sum((1, 3))
                        dist[:, a + b * d + f * d * d] = e.T.reshape(-1)
            S = _smallest(dist, K)
            S[:, 0] = ref
            a, b, f = S % d, S // d % d, S // (d * d)
            r0, c0 = (g % M * d)[:, None] + a, (g // M * d)[:, None] + b
            t = torch.arange(d, device=X.device)
            rows, cols = (r0[..., None] + t)[..., :, None], (c0[..., None] + t)[..., None, :]
            B = pads[f[..., None, None], rows, cols]
            V = _denoise_3d(_to_volume(B, M, N, d), _SYM, _tau(sigma, 2), 2).clamp(max=1)
            B = _to_groups(V, M, N, d)
            w = (1 / (_variation(B) + 2.0 ** -52))[:, None, None, None]
            r, c = rows - d // 2, cols - d // 2
            keep = ((r0 >= d // 2) & (c0 >= d // 2))[..., None, None] & (r < mp) & (c < np_)
            at = ((f[..., None, None] + j - 1) * mp + r) * np_ + c
            Y.view(-1).index_add_(0, at[keep], (w * B)[keep])
            W.view(-1).index_add_(0, at[keep], w.expand_as(B)[keep])
        total = total + torch.roll(Y / W, (-s, -s), (1, 2)) / 2
    return total[1:F - 1, :m, :n]


def exact(case, seed):
    kind, sigma = case["kind"], case["sigma"]
    m, n = case["m"], case["n"]
    x = _inputs(case, seed)
    if kind == "video":
        return _exact_video(x.transpose(1, 2), sigma / 255.0, case["patch"]).transpose(1, 2).contiguous()
    column = lambda v: v.T.contiguous()  # noqa: E731  m x n -> the column-major layout
    if kind == "batch":
        grey, rgb = _batch_items(case)
        out = []
        for img, it in zip(x[0], grey):
            out.append(column(_exact_images([img.T], [it[2]], _resolved(case, *it))[0][0]))
        for t, it in zip(x[1], rgb):
            out += [column(v) for v in _exact_rgb([p.T for p in t], it[2], _resolved(case, *it))]
        return out
    o = _resolved(case, m, n, sigma)
    if m * n > 2048 * 2048 and options.strides(o)[0] < o["blockSize"]:
        return None  # the overlapping groups of the largest dense image: over the time allowed
    if kind == "rgb":
        return [column(v) for v in _exact_rgb([p.T for p in x], sigma, o)]
    U, U1 = _exact_images([x.T], [sigma], o)
    if kind == "host":
        return [U[0].cpu().numpy(), U1[0].cpu().numpy()]
    return column(U[0]) if kind == "grey" else column(U[0]).cpu()
