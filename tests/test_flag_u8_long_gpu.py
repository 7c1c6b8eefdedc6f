"""Long bins of nearly saturated uint8 data: a lane of the statistics pass then
holds more squares than 32 bits take (66,051 of 255^2), and its sums must still
be exact.  Values alternate between 240 and 255 row by row and (one channel
out) by channel: mean 247.5 and variance 56.25, whole multiples of 1/4 that
FP64 and FP32 hold exactly, so the baseline's must equal them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,T,nbins", [(80, 393216, 9), (96, 327680, 9), (48, 688128, 9),
                                       (48, 688128, 10), (80, 393216, 11), (80, 393216, 17),
                                       (80, 393216, 3), (16, 2097152, 8), (144, 262144, 1)])
def test_variance_of_saturated_channels(dsax, C, T, nbins):
    import torch
    p = dsax.flag_params(1, T, C, guard=C // 8, filt=9, tbin=T // nbins, ts_base=64)
    row = 240 + 15 * (np.arange(C) % 2)
    x = torch.empty((T, C), dtype=torch.uint8, device="cuda")
    x[0::2] = torch.from_numpy(row.astype(np.uint8)).cuda()
    x[1::2] = torch.from_numpy((495 - row).astype(np.uint8)).cuda()
    torch.cuda.synchronize()
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        with ctx.flag_state(p, dsax.flag_clean_params(naver=1), dsax.DTYPE_U8) as st:
            st.clean(x)          # measured only: the baseline is this block's statistics
            spec, var = st.baseline()
    assert (spec == 247.5).all()
    assert (var == 56.25).all()
