"""A captured batch submitted again after the context's scratch moved to a
larger allocation: the graph must not use the old one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _descs(oracle, npkt, widths, nbeam):
    import torch
    host = [oracle.gen_block(33 + w, npkt, 63, w, "gauss") for w in widths]
    return host, [{"blk": torch.from_numpy(b.reshape(-1)).cuda(), "nchan": w,
                   "vis": torch.zeros(2 * w * 2080 * 8, dtype=torch.float32, device="cuda"),
                   "beams": torch.zeros((npkt // 16) * nbeam * (w // 8), dtype=torch.uint8,
                                        device="cuda")} for b, w in zip(host, widths)]


def test_replay_after_growth(dsax, oracle):
    import torch
    npkt, nbeam = 256, 64
    cfg = dsax.default_config(npkt=npkt, nant_in=63, nchan=768, nbeam=nbeam, bf_scale=1e-4)
    wre, wim = oracle.random_phase_weights(5, 96, nbeam)
    small_host, small = _descs(oracle, npkt, [16, 32], nbeam)
    _, large = _descs(oracle, npkt, [768, 192], nbeam)
    with dsax.Context(dsax.default_config(npkt=npkt, nant_in=63, nchan=32, nbeam=nbeam,
                                          bf_scale=1e-4)) as ctx:
        ctx.set_weights(wre[:4], wim[:4])
        ctx.run_batch(small, use_graph=True)
        ctx.sync()
        want = [d["beams"].clone() for d in small]
    with dsax.Context(cfg) as ctx:
        ctx.set_weights(wre, wim)
        ctx.run_batch(small, use_graph=True)
        ctx.run_batch(large, use_graph=False)     # the scratch grows
        ctx.sync()
        for d in small:
            d["vis"].zero_()
            d["beams"].zero_()
        torch.cuda.synchronize()
        ctx.run_batch(small, use_graph=True)
        ctx.sync()
        for b, d, w in zip(small_host, small, want):
            np.testing.assert_array_equal(
                d["vis"].cpu().numpy().reshape(-1, 2080, 4, 2), oracle.correlate(b))
            assert torch.equal(d["beams"], w)
