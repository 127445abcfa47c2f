"""Pictures with intra blocks through every route of the superblock kernel:
level by level, and in list order where a superblock's blocks are listed
against their dependencies. Sizes: one superblock, a ragged last superblock
column and row, odd sizes (REFCPU, SPEC), block and transform sizes from 4x4
to 64x64. Tolerance: none."""
import ctypes as C

import numpy as np
import pytest

from compute_vp9_b200 import ARITH_FULL, ARITH_REFCPU, ARITH_SPEC, CVP9_OK, BlockInfo, CudaBackend, Synth, synth_config
from compute_vp9_b200.hbd import HbdEngine, hbd_frames
from oracle.oracle_py import FULL, REFCPU, SPEC, HbdOracleStream, OracleStream

pytestmark = pytest.mark.gpu

CONTENT = {
    "small": {"min_bsize": 4, "max_bsize": 16, "tx_weights": [60, 40, 0, 0]},
    "mixed": {"min_bsize": 4, "skip_prob": 0.2},
    "large": {"min_bsize": 32, "tx_weights": [40, 20, 20, 20], "density_max": 0.6},
}


def _reverse_superblocks(pf):
    """Every superblock's blocks in reverse order (their coefficients stay where they are)."""
    n = pf.contents.num_blocks
    size = C.sizeof(BlockInfo)
    a = np.ctypeslib.as_array(C.cast(pf.contents.blocks, C.POINTER(C.c_uint8)), shape=(n * size,)).reshape(n, size)
    x = a[:, 0].astype(int) | a[:, 1].astype(int) << 8
    y = a[:, 2].astype(int) | a[:, 3].astype(int) << 8
    sb = (y >> 6) * 1024 + (x >> 6)
    starts = np.flatnonzero(np.r_[True, sb[1:] != sb[:-1]])
    for s, e in zip(starts, np.r_[starts[1:], n]):
        a[s:e] = a[s:e][::-1].copy()


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("content", list(CONTENT))
@pytest.mark.parametrize("size", [(64, 64), (136, 72), (328, 200), (67, 130), (201, 251)])
@pytest.mark.parametrize("arith", [ARITH_REFCPU, ARITH_SPEC, ARITH_FULL])
def test_intra_waves(arith, size, content, reverse):
    w, h = size
    if arith == ARITH_FULL and (w % 8 or h % 8):
        pytest.skip("FULL takes multiples of 8")
    over = dict(CONTENT[content], gop=2, intra_in_inter=0.5, all_intra_modes=1)
    if arith == ARITH_SPEC:
        over["interp_filter"] = 0
    syn = Synth(synth_config(2, w, h, seed=w + h, **over))
    gpu = CudaBackend(arith=arith)
    orc = OracleStream({ARITH_REFCPU: REFCPU, ARITH_SPEC: SPEC, ARITH_FULL: FULL}[arith])
    for f in range(3):
        pf = syn.frame(f)
        if reverse:
            _reverse_superblocks(pf)
        want = orc.decode(pf)
        assert gpu.decode(pf, f) == CVP9_OK, gpu.last_error()
        rc, got, _ = gpu.get_frame_array(wait=1)
        assert rc == CVP9_OK, gpu.last_error()
        assert np.array_equal(got, want), "frame %d: %d bytes differ" % (f, int((got != want).sum()))
    gpu.close()


@pytest.mark.parametrize("step", [64, 2000])      # 2000: dequantised values past +-2^18 among smaller ones
@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("content", list(CONTENT))
@pytest.mark.parametrize("size", [(64, 64), (136, 72), (328, 200)])
def test_intra_waves_10bit(size, content, reverse, step):
    w, h = size
    eng = HbdEngine()
    sid = eng.open_stream(w, h)
    orc = HbdOracleStream()
    over = dict(CONTENT[content], gop=2, intra_in_inter=0.5, all_intra_modes=1)
    for f, (pf, c32) in enumerate(hbd_frames(2, w, h, 3, seed=w + h, step=step, **over)):
        if reverse:
            _reverse_superblocks(pf)
        want = orc.decode(pf, c32)
        assert eng.submit([sid], [(pf, c32.ctypes.data)]) == CVP9_OK
        assert eng.wait() == CVP9_OK
        got = eng.get_frame(sid)
        assert np.array_equal(got, want), "frame %d: %d samples differ" % (f, int((got != want).sum()))
    eng.close()
