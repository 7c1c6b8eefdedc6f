"""The learned flagger's calls under a 1 ns wait limit: every wait, those of the
statistics pass among them, takes the context's limit and error word, so the
calls return and dsax_sync (or the training step itself) reports a timeout,
unless each wait completed at its first tries; then the results are the normal
ones.  The context with the default limit is right afterwards."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_learned_calls_with_a_1ns_wait_limit(dsax, oracle):
    import torch
    B, T, C, tds = 64, 4096, 48, 32
    x, _ = oracle.gen_filterbank(71, nbeam=B, ntime=T, nchan=C)
    p = dsax.flag_params(B, T, C)
    n = B * (T // tds) * C
    xd = torch.from_numpy(x).cuda()
    out = []
    for limit in (0, 1, 0):
        F = torch.zeros(n * 8, dtype=torch.float32, device="cuda")
        mask = torch.zeros(n, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        st = dsax.DSAX_OK
        with dsax.Context(dsax.default_config(npkt=16, nchan=8, wait_limit_ns=limit)) as ctx:
            ctx.lf_init(5)
            try:
                ctx.lf_features(p, xd, F, tds=tds)
                ctx.flag_learned(p, xd, mask, tds=tds)
                ctx.sync()
            except dsax.DsaxError as e:
                st = e.status
        assert st in (dsax.DSAX_OK, dsax.DSAX_ERR_TIMEOUT)
        assert limit or st == dsax.DSAX_OK
        out.append((st, F.cpu().numpy(), mask.cpu().numpy()))
    print("1 ns wait limit, learned flagger: status", out[1][0])
    for st, F, mask in out[1:]:
        if st == dsax.DSAX_OK:
            np.testing.assert_array_equal(F, out[0][1])
            np.testing.assert_array_equal(mask, out[0][2])
