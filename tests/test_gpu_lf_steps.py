"""The VP9 loop filter at the ends of its step schedule: one unit, one
superblock column or row, a last superblock of one unit (half a chroma unit),
rings of more superblocks than slots. Tolerance: none."""
import numpy as np
import pytest

from compute_vp9_b200 import ARITH_FULL, CVP9_OK, CudaBackend, Synth, synth_config
from compute_vp9_b200.hbd import HbdEngine, hbd_frames
from oracle.oracle_py import FULL, HbdOracleStream, OracleStream

pytestmark = pytest.mark.gpu

SIZES = [(8, 8), (8, 200), (264, 8), (64, 136), (72, 64), (392, 72)]
FILTERS = [{"lf_level": 1, "sharpness": 7}, {"lf_level": 63, "sharpness": 0}]
CONTENT = dict(gop=2, min_bsize=4, skip_prob=0.3, density_max=0.05)


@pytest.mark.parametrize("lf", FILTERS)
@pytest.mark.parametrize("size", SIZES)
def test_lf_steps(size, lf):
    w, h = size
    syn = Synth(synth_config(2, w, h, seed=w + h, **CONTENT, **lf))
    gpu, orc = CudaBackend(arith=ARITH_FULL), OracleStream(FULL)
    for f in range(3):
        pf = syn.frame(f)
        want = orc.decode(pf)
        assert gpu.decode(pf, f) == CVP9_OK, gpu.last_error()
        rc, got, _ = gpu.get_frame_array(wait=1)
        assert rc == CVP9_OK, gpu.last_error()
        assert np.array_equal(got, want), "frame %d: %d bytes differ" % (f, int((got != want).sum()))
    gpu.close()


@pytest.mark.parametrize("lf", FILTERS)
@pytest.mark.parametrize("size", SIZES)
def test_lf_steps_10bit(size, lf):
    w, h = size
    eng, orc = HbdEngine(), HbdOracleStream()
    sid = eng.open_stream(w, h)
    for f, (pf, c32) in enumerate(hbd_frames(2, w, h, 3, seed=w + h, step=16, **CONTENT, **lf)):
        want = orc.decode(pf, c32)
        assert eng.submit([sid], [(pf, c32.ctypes.data)]) == CVP9_OK
        assert eng.wait() == CVP9_OK
        got = eng.get_frame(sid)
        assert np.array_equal(got, want), "frame %d: %d samples differ" % (f, int((got != want).sum()))
    eng.close()
