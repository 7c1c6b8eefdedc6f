"""The peak-to-peak statistic where all of a channel's TBIN bins have the same
mean (one bin and a tail, or constant data) is exactly 0, as in the oracle: a
rounding residue in its place would have a median and MAD of its own and flag
channels at random."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,C,tbin", [(2, 177, 40, 151), (3, 253, 124, 187), (1, 700, 260, 512)])
def test_one_bin_fp32(dsax, oracle, B, T, C, tbin):
    import torch
    x = np.random.default_rng(C).normal(10, 1, (B, T, C)).astype(np.float32)
    p = dsax.flag_params(B, T, C, guard=2, filt=9, tbin=tbin, ts_base=64, thresh=3.0)
    xd = torch.from_numpy(x).cuda()
    cm = torch.zeros(B * C, dtype=torch.uint8, device="cuda")
    tm = torch.zeros(B * T, dtype=torch.uint8, device="cuda")
    st = torch.full((4 * B * C + B * T,), 7.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        ctx.flag(p, xd, cm, tm, stats=st)
        ctx.sync()
    spec, var, mx, pp = st.cpu().numpy()[:4 * B * C].reshape(4, B, C)
    assert (pp == 0).all()
    want, _ = oracle.chan_flags(spec, var, mx, pp, p)
    np.testing.assert_array_equal(cm.cpu().numpy().reshape(B, C), want)


def test_constant_channels_fp32(dsax):
    import torch
    B, T, C = 2, 1000, 52
    p = dsax.flag_params(B, T, C, guard=2, filt=9, tbin=100, ts_base=64)
    x = torch.rand(B, 1, C, device="cuda").add_(1).expand(B, T, C).contiguous()
    cm = torch.zeros(B * C, dtype=torch.uint8, device="cuda")
    tm = torch.zeros(B * T, dtype=torch.uint8, device="cuda")
    st = torch.zeros(4 * B * C + B * T, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        ctx.flag(p, x, cm, tm, stats=st)
        ctx.sync()
    assert (st[3 * B * C:4 * B * C] == 0).all()


@pytest.mark.parametrize("B,T,C,tbin", [(3, 160, 304, 142), (1, 3496, 496, 1811), (2, 3969, 704, 3690)])
def test_one_bin_uint8(dsax, oracle, B, T, C, tbin):
    import torch
    rng = np.random.default_rng(T)
    blocks = [np.clip(np.rint(rng.normal(48, 6, (B, T, C))), 0, 255).astype(np.uint8) for _ in range(2)]
    p = dsax.flag_params(B, T, C, guard=15, filt=9, tbin=tbin, ts_base=64, thresh=3.0, tsflag=0)
    cm = torch.zeros(B * C, dtype=torch.uint8, device="cuda")
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        with ctx.flag_state(p, dsax.flag_clean_params(naver=1, modcheck=0, scale=0), dsax.DTYPE_U8) as st:
            for x in blocks:
                xd = torch.from_numpy(x).cuda()
                torch.cuda.synchronize()
                st.clean(xd, cm)
                ctx.sync()
    spec0 = oracle.flag_stats(blocks[0], p)[0]
    s = oracle.flag_stats(blocks[1], p)
    assert (s[3] == 0).all()
    want, _ = oracle.chan_flags(*s, p, oldspec=spec0)
    np.testing.assert_array_equal(cm.cpu().numpy().reshape(B, C), want)
