"""A captured batch follows the matcher's statistics switch and wait limit: the
launch sequence depends on both, so a graph captured before one of them changed
is not replayed after it."""
import numpy as np
import pytest

from gbm3d_b200 import options, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
def test_batch_is_captured_again_when_the_matcher_changes(gpu, mixed):
    import torch
    from gbm3d_b200 import api
    from gbm3d_b200._lib import Context
    m, n = 128, 96
    refs = (m // 8) * (n // 8) * 2  # one spin per step
    ctx = Context(0)
    o = options.resolve_opts({"profile": "default"})
    o.update(blockSize=8, blockSizeWie=8, matchSize=32, refStride=8, refStrideWie=8, matchSpins=[0], matchSpinsWie=[0],
             staleWeights=False, form="tensor")
    x = torch.from_numpy(np.ascontiguousarray(synth.noisy_image(m, n, 25.0, seed=4)[1].T)).cuda()
    out = torch.empty_like(x)

    def run():
        if mixed:
            api.GBM3D_mixed([x], [25.0], opts=o, ctx=ctx, outputs=([out], [], None))
        else:
            api.GBM3D_batch([x], [25.0], o, ctx=ctx, outputs=[out])
        return ctx.launch_count(), out.clone()

    _, want = run()
    assert run()[0] == 1  # a replay
    ctx.tc_stats(True)
    assert torch.equal(run()[1], want)
    assert torch.equal(run()[1], want)
    assert sum(ctx.tc_stats(False)) == 2 * refs  # both calls counted every reference
    assert torch.equal(run()[1], want)
    assert sum(ctx.tc_stats(False)) == 0  # and none is counted once it is off
    ctx.set_tc_wait(4_000_000_000)
    launches, got = run()
    assert launches > 1 and torch.equal(got, want)
    ctx.set_tc_wait(0)
    launches, got = run()
    assert launches > 1 and torch.equal(got, want)
