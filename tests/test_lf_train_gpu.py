"""The training kernels' gradients at the edges of their tiles (rows that end
inside a CTA's four or a strip's eight or two, the narrowest and widest rows)
against the FP64 oracle: within 2e-3 of each layer's gradient scale, as the
other gradient test allows."""
import numpy as np
import pytest

import lflag_oracle as LO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,C,tds", [(1, 384, 8, 128), (2, 1152, 64, 64), (1, 640, 20, 64),
                                       (3, 1280, 36, 32)])
def test_gradients(dsax, oracle, B, T, C, tds):
    import torch
    x, _ = oracle.gen_filterbank(700 + C, nbeam=B, ntime=T, nchan=C, n_tones=B, n_bursts=B, n_drift=0)
    guard, H = 1, T // tds
    p = dsax.flag_params(B, T, C, guard=guard, filt=min(9, C - 2))
    rng = np.random.default_rng(C)
    cm = (rng.random((B, C)) < 0.1).astype(np.uint8)
    tm = (rng.random((B, T)) < 0.01).astype(np.uint8)
    params = LO.init_params(C)
    flat = np.concatenate([np.concatenate([w.reshape(-1), b]) for w, b in params]).astype(np.float32)
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        ctx.lf_set_params(flat)
        xd, cd, td = (torch.from_numpy(a).cuda() for a in (x, cm, tm))
        F = torch.zeros(B * H * C * 8, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.lf_features(p, xd, F, tds=tds)
        loss, grads = ctx.lf_train_step(p, xd, cd, td, tds=tds, update=False, pos_weight=3.0,
                                        want_grads=True)
        f = F.cpu().numpy().reshape(B, H, C, 8).astype(np.float64)
    y = LO.labels(cm, tm, tds, guard)
    valid = np.zeros((B, H, C))
    valid[:, :, guard:C - guard] = 1.0
    acts = LO.forward(params, f)
    want, dl = LO.bce_loss_grad(acts[-1], y, valid, 3.0)
    assert abs(loss - want) < 1e-4 * max(1.0, abs(want))
    o = 0
    for dw, db in LO.backward(params, acts, dl):
        for g in (dw.reshape(-1), db):
            got = grads[o:o + g.size]
            o += g.size
            assert np.abs(got - g).max() <= 2e-3 * np.abs(g).max()
