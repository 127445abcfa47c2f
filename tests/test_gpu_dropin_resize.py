"""The drop-in backend with its ring full while the picture size changes: scratch
and device frames are replaced while earlier pictures are still on their way
down, and a device frame is taken again two pictures after its download began.
Every delivered picture must be the oracle's. Tolerance: none."""
import numpy as np
import pytest

from compute_vp9_b200 import ARITH_REFCPU, CVP9_ERR_AGAIN, CVP9_OK, CudaBackend, Synth, synth_config
from oracle.oracle_py import REFCPU, OracleStream

pytestmark = pytest.mark.gpu

# (size, pictures): references stay across a change, of their own size
PLANS = {
    "grow": [((200, 136), 4), ((640, 360), 4), ((1280, 720), 5)],
    "back_and_forth": [((640, 360), 2), ((251, 131), 3), ((640, 360), 1), ((1280, 720), 4), ((251, 131), 2), ((640, 360), 4)],
}


@pytest.mark.parametrize("plan", list(PLANS))
def test_resize_with_pictures_in_the_ring(plan):
    gpu, orc = CudaBackend(arith=ARITH_REFCPU), OracleStream(REFCPU)
    synths, waiting, delivered = {}, [], 0

    def deliver():
        rc, got, info = gpu.get_frame_array(wait=1)
        assert rc == CVP9_OK, gpu.last_error()
        pts, want = waiting.pop(0)
        assert info.pts == pts and np.array_equal(got, want), "picture %d" % pts
        return 1

    pts = 0
    for size, count in PLANS[plan]:
        if size not in synths:
            synths[size] = [Synth(synth_config(2, *size, seed=sum(size), gop=60, intra_in_inter=0.1)), 0]
        syn = synths[size]
        for _ in range(count):
            pf = syn[0].frame(syn[1])
            syn[1] += 1
            want = orc.decode(pf)
            rc = gpu.decode(pf, pts)
            if rc == CVP9_ERR_AGAIN:              # three in the ring: one leaves, two stay
                delivered += deliver()
                rc = gpu.decode(pf, pts)
            assert rc == CVP9_OK, gpu.last_error()
            waiting.append((pts, want))
            pts += 1
    while waiting:
        delivered += deliver()
    assert delivered == pts
    gpu.close()
