"""A call whose kernel launch is refused on the host does nothing and says so:
it returns an error instead of OK, and leaves parameters and outputs alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# pixel rows of 128 samples x 64 channels (32 KB), beyond the statistics pass's 24 KB
B, T, C, TDS = 1, 256, 64, 128


def _learned(dsax):
    import torch
    p = dsax.flag_params(B, T, C, guard=1, filt=9)
    n = B * (T // TDS) * C
    x = torch.rand(B * T * C, device="cuda") + 10
    return p, x, n


def test_learned_flagger_calls(dsax):
    import torch
    p, x, n = _learned(dsax)
    F = torch.full((n * 8,), 7.0, device="cuda")
    mask = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
    logit = torch.full((n,), 7.0, device="cuda")
    torch.cuda.synchronize()
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        ctx.lf_init(3)
        with pytest.raises(dsax.DsaxError):
            ctx.lf_features(p, x, F, tds=TDS)
        with pytest.raises(dsax.DsaxError):
            ctx.flag_learned(p, x, mask, logits=logit, tds=TDS)
        ctx.sync()
    assert (F == 7.0).all() and (mask == 9).all() and (logit == 7.0).all()


def test_training_step(dsax):
    import torch
    p, x, _ = _learned(dsax)
    cm = torch.zeros(B * C, dtype=torch.uint8, device="cuda")
    tm = torch.zeros(B * T, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        ctx.lf_init(3)
        before = np.array(ctx.lf_get_params())
        with pytest.raises(dsax.DsaxError):
            ctx.lf_train_step(p, x, cm, tm, tds=TDS, lr=0.1)
        np.testing.assert_array_equal(np.array(ctx.lf_get_params()), before)


def test_batch(dsax, oracle):
    """24 channels are three channel groups, fewer than the flagger takes."""
    import torch
    blk = torch.zeros(64 * 63 * 24 * 4, dtype=torch.uint8, device="cuda")
    cm = torch.zeros(64 * 3, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with dsax.Context(dsax.default_config(npkt=64, nchan=24, nbeam=64)) as ctx:
        ctx.set_weights(*oracle.random_phase_weights(5, 3, 64))
        with pytest.raises(dsax.DsaxError):
            ctx.run_batch([{"blk": blk, "nchan": 24, "chanmask": cm}], use_graph=False)
        ctx.sync()
