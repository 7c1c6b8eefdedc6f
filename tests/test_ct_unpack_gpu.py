"""dsax_ct_unpack against numpy at every piece width (16, 8, 4 and 1 bytes),
rows wider than a pass, row counts that end inside a pass, and offsets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc,nbl,nt,nc,ch0,extra,t0,pad", [
    (16, 3, 163, 48, 128, 128, 5, 0), (5, 2, 81, 24, 8, 0, 0, 3), (3, 1, 17, 20, 4, 12, 1, 0),
    (2, 2, 9, 7, 3, 1, 0, 2), (300, 1, 5, 1, 0, 0, 0, 0), (17, 2, 1, 256, 16, 16, 2, 1)])
def test_ct_unpack(dsax, nsrc, nbl, nt, nc, ch0, extra, t0, pad):
    import torch
    fil_nc, fil_nt = ch0 + nsrc * nc + extra, t0 + nt + pad
    rng = np.random.default_rng(nc)
    recv = rng.integers(0, 256, (nsrc, nbl, nt, nc), dtype=np.uint8)
    want = np.full((nbl, fil_nt, fil_nc), 77, np.uint8)
    want[:, t0:t0 + nt, ch0:ch0 + nsrc * nc] = recv.transpose(1, 2, 0, 3).reshape(nbl, nt, nsrc * nc)
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        d, fil = torch.from_numpy(recv).cuda(), torch.full(want.shape, 77, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        ctx.ct_unpack(d, nsrc, nbl, nt, nc, fil, fil_nt, fil_nc, t0, ch0)
        ctx.sync()
        np.testing.assert_array_equal(fil.cpu().numpy(), want)
