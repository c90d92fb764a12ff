"""Cycle spins that share the launches of the coarse wavelet levels: any number
of them, their results and their workspace."""
import numpy as np
import pytest

from gbm3d_b200 import options
from gbm3d_b200.api import _as_set

pytestmark = pytest.mark.gpu

MIB = 1 << 20


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


def _dense(cycles):
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=8, blockSizeWie=8, matchSize=32, refStride=3, refStrideWie=3, matchSpins=[0], matchSpinsWie=[0],
             cycleSpin=cycles, Wiener=False)
    return o


def _step1(ctx, m, n, cycles, seed=1):
    """Step 1 of a random device image; the device memory in use after it."""
    import torch
    from gbm3d_b200 import api
    x = 255 * torch.rand((n, m), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
    out = torch.empty_like(x)
    torch.cuda.synchronize()
    api.GBM3D_device(x.data_ptr(), m, n, 25.0, out.data_ptr(), _dense(cycles), ctx=ctx)
    ctx.synchronize()
    res = out.cpu()
    del x, out
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free, res


def test_workspace_of_a_smaller_image_is_that_of_the_larger(gpu):
    """A smaller image after a larger one allocates nothing (a growth would stall every stream
    and drop the captured graph)."""
    from gbm3d_b200._lib import Context
    ctx = Context(0)
    used, _ = _step1(ctx, 800, 800, 2)
    for side in (700, 500, 250):
        assert _step1(ctx, side, side, 2)[0] == used
    ctx.close()


@pytest.mark.parametrize("cycles,side", [(2, 750), (8, 370)])
def test_shared_spins_memory_is_bounded(gpu, cycles, side):
    from gbm3d_b200._lib import Context
    used = {}
    for c in (1, cycles):
        ctx = Context(0)
        base = _step1(ctx, 40, 40, 1)[0]
        used[c] = _step1(ctx, side, side, c)[0] - base
        ctx.close()
    assert used[cycles] - used[1] <= 256 * MIB + 16 * MIB  # 16: pages of the few buffers


@pytest.mark.parametrize("wiener,graph", [(False, False), (True, False), (True, True)])
def test_device_without_room_for_the_shared_spins(gpu, wiener, graph):
    """With too little memory left for them (at their own allocation, or with the second step's at a
    later one) the spins run one after another, to the same result, and the context goes on working."""
    import torch
    from gbm3d_b200 import api
    from gbm3d_b200._lib import Context
    side = 600
    o = dict(_dense(3), Wiener=wiener)
    x = 255 * torch.rand((side, side), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    out = torch.empty_like(x)

    def run(ctx):
        out.zero_()
        api.GBM3D_batch([x], [25.0], o, ctx=ctx, use_graph=graph, outputs=[out])
        return ctx.launch_count(), out.cpu()

    def free():
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    start = free()
    ctx = Context(0)
    _, want = run(ctx)
    need = start - free()
    ctx.close()
    ctx = Context(0)
    hold = torch.empty(free() - (need - 128 * MIB), dtype=torch.uint8, device="cuda")
    try:
        got = [run(ctx) for _ in range(3)]
    finally:
        del hold
        torch.cuda.empty_cache()
    for launches, u in got + [run(ctx)]:
        assert torch.equal(u, want)
    assert not graph or got[2][0] == 1  # the second call at the latest was captured
    ctx.close()
