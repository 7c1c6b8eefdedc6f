"""The 64-channel layers' tiles (one run of padded rows for all nine taps) at
the narrowest and widest rows, rows that are no multiple of the swizzle's
eight, and enough tiles per CTA to go round its stages: logits against the
oracle's restatement within 5e-3 of their scale, as the other inference test."""
import numpy as np
import pytest

import lflag_oracle as LO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,C,tds", [(1, 256, 8, 32), (3, 640, 20, 64), (2, 384, 60, 32),
                                       (56, 1024, 64, 32)])
def test_logits(dsax, oracle, B, T, C, tds):
    import torch
    x, _ = oracle.gen_filterbank(900 + C, nbeam=B, ntime=T, nchan=C, n_tones=B, n_bursts=B, n_drift=0)
    p = dsax.flag_params(B, T, C, guard=1, filt=min(9, C - 2))
    rng = np.random.default_rng(C)
    params = [(w, rng.normal(scale=0.1, size=b.shape)) for w, b in LO.init_params(C)]
    flat = np.concatenate([np.concatenate([w.reshape(-1), b]) for w, b in params]).astype(np.float32)
    n = B * (T // tds) * C
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        ctx.lf_set_params(flat)
        xd = torch.from_numpy(x).cuda()
        F = torch.zeros(n * 8, dtype=torch.float32, device="cuda")
        mask = torch.zeros(n, dtype=torch.uint8, device="cuda")
        logit = torch.zeros(n, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.lf_features(p, xd, F, tds=tds)
        ctx.flag_learned(p, xd, mask, logits=logit, tds=tds)
        ctx.sync()
        got = logit.cpu().numpy().reshape(B, T // tds, C)
        f = F.cpu().numpy().reshape(B, T // tds, C, 8).astype(np.float64)
    pw = [(w.astype(np.float32).astype(np.float64), b.astype(np.float32).astype(np.float64))
          for w, b in params]
    want = LO.forward_bf16(pw, f)
    assert np.abs(got - want).max() < 5e-3 * np.abs(want).max()
