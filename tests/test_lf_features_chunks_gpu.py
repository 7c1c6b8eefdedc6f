"""Learned-flagger features where the statistics pass also splits time (few
beams, many bins), at two widths and in one context after calls with other
numbers of beams, against the oracle with the tolerance of the unsplit test."""
import numpy as np
import pytest

import lflag_oracle as LO

pytestmark = pytest.mark.gpu


def test_features_of_time_chunks(dsax, oracle):
    import torch
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        for B, T, C, tds in ((2, 4096, 48, 32), (5, 2048, 64, 32), (1, 4096, 48, 16), (2, 4096, 36, 64)):
            x, _ = oracle.gen_filterbank(60 + B + C, nbeam=B, ntime=T, nchan=C, n_tones=B, n_bursts=B,
                                         n_drift=1)
            p = dsax.flag_params(B, T, C)
            F = torch.zeros(B * (T // tds) * C * 8, dtype=torch.float32, device="cuda")
            xd = torch.from_numpy(x).cuda()
            torch.cuda.synchronize()
            ctx.lf_features(p, xd, F, tds=tds)
            ctx.sync()
            got = F.cpu().numpy().reshape(B, T // tds, C, 8)
            np.testing.assert_allclose(got, LO.features(x, tds, p), rtol=2e-4, atol=2e-4)
