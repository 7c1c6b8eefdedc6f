"""dsax_ct_unpack with few passes per CTA (calls of few CTAs) against numpy at every
piece width."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc,nbl,nt,nc,ch0", [(1, 1, 4097, 16, 16), (1, 2, 2049, 8, 0), (3, 1, 1023, 4, 4),
                                                (1, 1, 1025, 1, 3), (2, 300, 65, 24, 8)])
def test_few_passes(dsax, nsrc, nbl, nt, nc, ch0):
    import torch
    fil_nc, fil_nt = ch0 + nsrc * nc + ch0, nt + 3
    rng = np.random.default_rng(nt)
    recv = rng.integers(0, 256, (nsrc, nbl, nt, nc), dtype=np.uint8)
    want = np.full((nbl, fil_nt, fil_nc), 77, np.uint8)
    want[:, 2:2 + nt, ch0:ch0 + nsrc * nc] = recv.transpose(1, 2, 0, 3).reshape(nbl, nt, nsrc * nc)
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        d, fil = torch.from_numpy(recv).cuda(), torch.full(want.shape, 77, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        ctx.ct_unpack(d, nsrc, nbl, nt, nc, fil, fil_nt, fil_nc, 2, ch0)
        ctx.sync()
        np.testing.assert_array_equal(fil.cpu().numpy(), want)
