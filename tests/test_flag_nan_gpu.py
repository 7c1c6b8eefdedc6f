"""Blocks with rows of NaN: every mean of the beam is NaN, so no median of the
mean spectrum exists and that test flags nothing, while the maxima and the
peak-to-peak means (which pass over NaN) still decide as the oracle's tests do on
them; the same masks on every call, whatever the shared memory held before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,C,tbin", [(3, 640, 48, 128), (1, 8192, 48, 128), (2, 512, 256, 64),
                                        (1, 84, 76, 128)])
def test_rows_of_nan(dsax, oracle, B, T, C, tbin):
    import torch
    rng = np.random.default_rng(C + T)
    x = rng.normal(10, 1, (B, T, C)).astype(np.float32)
    x[0, :, C // 2] += 4
    other = torch.from_numpy(rng.normal(50, 20, (B, T, C)).astype(np.float32)).cuda()
    x[:, T // 3] = np.nan
    p = dsax.flag_params(B, T, C, guard=2, filt=21, tbin=tbin, ts_base=32, thresh=4.0)
    xd = torch.from_numpy(x).cuda()
    masks = []
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        for k in range(4):
            cm = torch.zeros(B * C, dtype=torch.uint8, device="cuda")
            tm = torch.zeros(B * T, dtype=torch.uint8, device="cuda")
            st = torch.zeros(4 * B * C + B * T, dtype=torch.float32, device="cuda")
            torch.cuda.synchronize()
            if k:
                ctx.flag(p, other, cm, tm)
            ctx.flag(p, xd, cm, tm, stats=st)
            ctx.sync()
            masks.append(cm.cpu().numpy().reshape(B, C))
    spec, var, mx, pp = st.cpu().numpy()[:4 * B * C].reshape(4, B, C)
    assert np.isnan(spec).all() and (var == 0).all() and np.isfinite(mx).all() and np.isfinite(pp).all()
    want, _ = oracle.chan_flags(np.zeros_like(spec), var, mx, pp, p)
    for m in masks:
        np.testing.assert_array_equal(m, want)
