"""dsax_ct_unpack with as many rows as an int counts."""
import pytest

pytestmark = pytest.mark.gpu


def test_the_most_rows(dsax):
    import torch
    nt = 2**31 - 1
    recv = torch.randint(0, 256, (nt,), dtype=torch.uint8, device="cuda")
    fil = torch.zeros(nt, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with dsax.Context(dsax.default_config(npkt=16, nchan=8)) as ctx:
        ctx.ct_unpack(recv, 1, 1, nt, 1, fil, nt, 1, 0, 0)
        ctx.sync()
    assert torch.equal(recv, fil)
