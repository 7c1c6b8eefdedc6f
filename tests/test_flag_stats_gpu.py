"""The statistics and apply passes at the edges of their splits, against the
oracle: time chunks (few beams, many bins), fewer bins than warps, rows past
the last bin, full and ragged slabs, more flagged chunks than lanes."""
import numpy as np
import pytest

from test_flag_clean_gpu import _check_block, _run, _u8_blocks
from test_flag_gpu import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,C,tbin", [(2, 16384, 48, 128), (1, 5000, 104, 128), (3, 900, 48, 300),
                                        (2, 640, 1024, 128), (1, 2100, 132, 64), (1, 130, 4, 1),
                                        (1, 4096, 36, 7), (5, 100, 48, 128)])
def test_fp32_splits(dsax, oracle, B, T, C, tbin):
    x, _ = oracle.gen_filterbank(B + T + C, nbeam=B, ntime=T, nchan=C, n_tones=B, n_bursts=B, n_drift=1)
    guard = C // 8
    _compare(dsax, oracle, x, guard=guard, filt=min(21, C - 2 * guard), tbin=tbin, ts_base=min(T, 512))


@pytest.mark.parametrize("B,T,C,tbin", [(2, 8192, 256, 128), (1, 4500, 144, 128), (3, 700, 48, 350),
                                        (1, 3000, 16, 100)])
def test_uint8_splits(dsax, oracle, B, T, C, tbin):
    guard = C // 8
    p = dsax.flag_params(B, T, C, guard=guard, filt=min(21, C - 2 * guard), tbin=tbin, ts_base=128)
    res, _, _, _ = _run(dsax, oracle, _u8_blocks(B + T, 3, B, T, C), p, dsax.DTYPE_U8,
                        dsax.MEM_DEVICE, naver=1, mod_thresh=0.5)
    for r in res[1:]:
        assert r[3].flagged and not r[3].replaced
        _check_block(r)


def test_uint8_many_flagged_chunks(dsax, oracle):
    """A tone in every other 16-channel chunk: more than 32 chunks to replace."""
    B, T, C = 2, 1024, 1024
    blocks = _u8_blocks(5, 2, B, T, C)
    blocks[1][:, :, 136:888:32] = 255
    blocks[1][:, :, 152:888:48] = 0
    p = dsax.flag_params(B, T, C, guard=128, ts_base=128)
    res, _, _, _ = _run(dsax, oracle, blocks, p, dsax.DTYPE_U8, dsax.MEM_DEVICE, naver=1, mod_thresh=0.9)
    _check_block(res[1])
    assert (res[1][1].reshape(B, 64, 16).any(axis=2).sum(axis=1) > 32).any()
