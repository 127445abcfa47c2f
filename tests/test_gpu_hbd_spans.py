"""10-bit blocks whose coefficient spans overlap, or lie out of list order.
The block record asks for neither, so every sample must be the list-order
oracle's: blocks of a superblock at one offset, spans that share a part,
offsets exchanged between blocks of one size, gaps; DCT beside ADST, inter beside
intra, transforms of one warp and of several. Tolerance: none."""
import numpy as np
import pytest

from compute_vp9_b200 import CVP9_OK
from compute_vp9_b200.hbd import HbdEngine, hbd_frames
from oracle.oracle_py import HbdOracleStream

pytestmark = pytest.mark.gpu

CONTENT = {
    "small": {"tx_weights": [60, 40, 0, 0], "max_bsize": 16},
    "mixed": {"min_bsize": 4, "skip_prob": 0.2},
    "large": {"min_bsize": 32, "tx_weights": [0, 0, 40, 60]},
}


def _respan(pf, how):
    p = pf.contents
    sbs = {}
    for i in range(p.num_blocks):
        b = p.blocks[i]
        sbs.setdefault((b.y >> 6, b.x >> 6), []).append(b)
    for blocks in sbs.values():
        first = min(b.coeff_offset for b in blocks)
        if how == "exchanged":
            by_size = {}
            for b in blocks:
                by_size.setdefault((b.width, b.height, b.tx_size, b.skip), []).append(b)
            for same in by_size.values():
                offsets = [b.coeff_offset for b in same]
                for b, o in zip(same, offsets[::-1]):
                    b.coeff_offset = o
        elif how == "gaps":
            for b in blocks[1::3]:
                b.skip = 1
        else:
            for b in blocks:
                b.coeff_offset = first if how == "one" else first + (b.coeff_offset - first) // 8 * 4


@pytest.mark.parametrize("how", ["one", "part", "exchanged", "gaps"])
@pytest.mark.parametrize("content", list(CONTENT))
@pytest.mark.parametrize("size", [(64, 64), (136, 72), (328, 200)])
def test_spans(size, content, how):
    w, h = size
    eng, orc = HbdEngine(), HbdOracleStream()
    sid = eng.open_stream(w, h)
    over = dict(CONTENT[content], gop=2, intra_in_inter=0.5, all_intra_modes=1, density_max=0.4)
    for f, (pf, c32) in enumerate(hbd_frames(2, w, h, 3, seed=w + h, step=16, **over)):
        _respan(pf, how)
        want = orc.decode(pf, c32)
        assert eng.submit([sid], [(pf, c32.ctypes.data)]) == CVP9_OK
        assert eng.wait() == CVP9_OK
        got = eng.get_frame(sid)
        assert np.array_equal(got, want), "frame %d: %d samples differ" % (f, int((got != want).sum()))
    eng.close()
