"""Launches that overlap the previous kernel's end (csrc/common.cuh, launch_next)
against the plain launches of a captured graph: the same bits on repeated calls
with changing inputs, from a single partial wave of CTAs to several."""
import numpy as np
import pytest

from gbm3d_b200 import options, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,s", [(24, 24, 8), (65, 47, 3), (128, 96, 8), (301, 203, 3), (640, 480, 3)])
def test_overlapped_launches_equal_captured(gpu, m, n, s):
    import torch
    from gbm3d_b200 import api
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=8, blockSizeWie=8, matchSize=24, refStride=s, refStrideWie=s)
    imgs = [torch.from_numpy(np.ascontiguousarray(synth.noisy_image(m, n, 25.0, seed=k)[1].T)).cuda() for k in (1, 2)]
    captured = [x.clone() for x in api.GBM3D_batch(imgs, [25.0] * 2, o, use_graph=True)]
    for _ in range(8):
        for k in (0, 1):
            plain = api.GBM3D_batch(imgs[k:k + 1], [25.0], o, use_graph=False)[0]
            assert torch.equal(plain, captured[k])


@pytest.mark.parametrize("first,between", [((96, 80), (160, 128)), ((320, 256), (304, 256))])
def test_graph_replay_after_buffers_grew(gpu, first, between):
    """A call in between that needs larger workspaces: the batch is captured again."""
    import torch
    from gbm3d_b200 import api
    from gbm3d_b200._lib import Context
    ctx = Context(0)
    o = options.resolve_opts({"profile": "default"})
    x, y = [torch.from_numpy(np.ascontiguousarray(synth.noisy_image(m, n, 25.0, seed=m)[1].T)).cuda()
            for m, n in (first, between)]
    out = [torch.empty_like(x)]
    want = api.GBM3D_batch([x], [25.0], o, ctx=ctx, use_graph=True, outputs=out)[0].clone()
    for _ in range(2):  # a replay, then the call after the workspaces grew
        out[0].zero_()
        api.GBM3D_batch([x], [25.0], o, ctx=ctx, use_graph=True, outputs=out)
        assert torch.equal(out[0], want)
        api.GBM3D_batch([y], [25.0], o, ctx=ctx, use_graph=False)


@pytest.mark.parametrize("m,n", [(24, 24), (65, 47), (301, 203)])
def test_host_arrays_shared_between_arguments(gpu, m, n):
    """The host call's copies: outputs in one array (it ends as U1), in place, and apart."""
    import ctypes as C
    from gbm3d_b200 import api
    from gbm3d_b200._lib import lib
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=8, blockSizeWie=8, matchSize=24, refStride=8, refStrideWie=8)
    x = np.asfortranarray(synth.noisy_image(m, n, 25.0, seed=3)[1])
    U, out = api.GBM3D(x, 25.0, o)
    co, ctx = api.c_opts(o), api.context()
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731

    def call(I, u, u1):
        ctx.check(lib().gbm3d_denoise(ctx.h, p(I), m, n, 25.0, C.byref(co), p(u), p(u1)))

    both = np.zeros((m, n), order="F")
    call(x, both, both)
    assert np.array_equal(both, out["U1"])
    inplace, u1 = x.copy(order="F"), np.zeros((m, n), order="F")
    call(inplace, inplace, u1)
    assert np.array_equal(inplace, U) and np.array_equal(u1, out["U1"])
    u, inplace = np.zeros((m, n), order="F"), x.copy(order="F")
    call(inplace, u, inplace)
    assert np.array_equal(u, U) and np.array_equal(inplace, out["U1"])
