"""A batch with a refused block (three channel groups, fewer than the flagger
takes) after a good one: the call fails, the streams' fork is joined and no CUDA
error stays behind, so the next batch of the context is right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [True, False])
def test_batch_after_a_refused_block(dsax, oracle, use_graph):
    import torch
    npkt, widths = 64, (16, 24)
    host = [oracle.gen_block(77 + w, npkt, 63, w, "gauss") for w in widths]
    descs = [{"blk": torch.from_numpy(b.reshape(-1)).cuda(), "nchan": w,
              "vis": torch.zeros(2 * w * 2080 * 8, dtype=torch.float32, device="cuda"),
              "chanmask": torch.zeros(64 * (w // 8), dtype=torch.uint8, device="cuda")}
             for b, w in zip(host, widths)]
    descs[0].pop("chanmask")
    torch.cuda.synchronize()
    with dsax.Context(dsax.default_config(npkt=npkt, nchan=24, nbeam=64)) as ctx:
        ctx.set_weights(*oracle.random_phase_weights(5, 3, 64))
        with pytest.raises(dsax.DsaxError):
            ctx.run_batch(descs, use_graph=use_graph)
        torch.zeros(16, device="cuda").add_(1)       # raises what a call left behind
        ctx.sync()
        for d in descs:
            d.pop("chanmask", None)
            d["vis"].zero_()
        torch.cuda.synchronize()
        for _ in range(2):
            ctx.run_batch(descs, use_graph=use_graph)
        ctx.sync()
        for b, w, d in zip(host, widths, descs):
            np.testing.assert_array_equal(d["vis"].cpu().numpy().reshape(2 * w, 2080, 4, 2),
                                          oracle.correlate(b))
