"""The correlator over frequency rows at the edges of its tiles: stages of 128
packets, several frequencies per CTA, both row orders, and the largest sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vis(dsax, arr, fmt, npkt, nant, nchan, **kw):
    import torch
    with dsax.Context(dsax.default_config(npkt=npkt, nant_in=nant, nchan=nchan, **kw)) as ctx:
        d = torch.from_numpy(np.ascontiguousarray(arr).reshape(-1)).cuda()
        vis = torch.full((2 * nchan * 2080 * 8,), 1.0, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.correlate(d, vis, fmt=fmt)
        ctx.correlate(d, vis, fmt=fmt, accumulate=True)
        ctx.sync()
        return vis.cpu().numpy().reshape(2 * nchan, 2080, 4, 2)


@pytest.mark.parametrize("npkt,nant,nchan", [(1, 64, 1), (127, 63, 3), (128, 5, 75), (129, 64, 2),
                                             (300, 63, 149), (640, 64, 38)])
def test_rows_bit_exact(dsax, oracle, npkt, nant, nchan):
    blk = oracle.gen_block(4000 + npkt, npkt, nant, nchan, "uniform")
    want = 2 * oracle.correlate(blk)
    rows = np.zeros((npkt, nchan, 2, 64, 2), np.uint8)
    rows[:, :, :, :nant] = blk.reshape(npkt, nant, nchan, 2, 2).transpose(0, 2, 3, 1, 4)
    np.testing.assert_array_equal(_vis(dsax, blk, dsax.FMT_CAPTURED, npkt, nant, nchan), want)
    np.testing.assert_array_equal(_vis(dsax, rows, dsax.FMT_REORDERED, npkt, 64, nchan), want)


@pytest.mark.parametrize("corr_path", [4, 5])
def test_largest_sums(dsax, corr_path):
    """65,536 packets of -8 - 8i: every real part is 2^23, every imaginary 0."""
    npkt = 65536
    vis = _vis(dsax, np.full(npkt * 64 * 4, 0x88, np.uint8), dsax.FMT_CAPTURED, npkt, 64, 1,
               corr_path=corr_path)
    np.testing.assert_array_equal(vis[..., 0], np.float32(2 * 2.0 ** 23))
    np.testing.assert_array_equal(vis[..., 1], np.float32(0))
