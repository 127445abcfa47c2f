"""Blocks off the 8x8 grid, blocks whose transforms reach past them, blocks 4
samples wide and more than 8 tall. No parser makes them, but the layout checks
take them: the first two kinds run in list order, and all samples are the
list-order oracle's. Tolerance: none.

CONTENT: "skipped" has predictions alone (edges by MI, chroma of 6 samples),
"4x4" the smallest transforms too (chroma between 4x4 cells), "any" those
that are no divisor of the block, or larger (10 bits: not larger), some across
the superblock's edge. FULL and 10 bits predict by transform and so read edges
past the superblock there: a picture of one superblock only. Blocks are
shuffled, so that transforms reach over finished ones; not in larger pictures
of "any", where the oracle's reach into superblocks that shuffled blocks would
read before their prediction. "narrow" has blocks on the 8x8 grid, many of them
cut to 4 samples in one direction."""
import ctypes as C
import random

import numpy as np
import pytest

from compute_vp9_b200 import (ARITH_FULL, ARITH_REFCPU, ARITH_SPEC, CVP9_OK, BlockInfo, CudaBackend, ParsedFrame, Synth,
                              synth_config)
from compute_vp9_b200.hbd import HbdEngine
from oracle.oracle_py import FULL, REFCPU, SPEC, HbdOracleStream, OracleStream

pytestmark = pytest.mark.gpu

HBD = 3
CONTENT = ["skipped", "4x4", "any", "narrow"]


def _split(rng, x, y, w, h, out, step):
    """Rectangles of at least 8x8 at multiples of `step`."""
    cuts = [c for c, n in (("w", w), ("h", h)) if n >= 16]
    if not cuts or (w <= 40 and h <= 40 and rng.random() < 0.3):
        out.append((x, y, w, h))
    elif rng.choice(cuts) == "w":
        k = rng.randrange(8, w - 7, step)
        _split(rng, x, y, k, h, out, step)
        _split(rng, x + k, y, w - k, h, out, step)
    else:
        k = rng.randrange(8, h - 7, step)
        _split(rng, x, y, w, k, out, step)
        _split(rng, x, y + k, w, h - k, out, step)


def _frame(rng, header, arith, w, h, key, content):
    """A picture of such blocks -> (frame, its arrays)."""
    recs, coeffs = [], 0
    for sy in range(0, h, 64):
        for sx in range(0, w, 64):
            rects = []
            _split(rng, 0, 0, 64, 64, rects, 8 if content == "narrow" else 4)
            if content != "any" or w <= 64:
                rng.shuffle(rects)
            for x, y, bw, bh in rects:
                if sx + x >= w or sy + y >= h:
                    continue
                tx = rng.randrange(4) if content == "any" else 0
                if content == "narrow" and rng.random() < 0.5:
                    bw, bh = (4, bh) if rng.random() < 0.5 else (bw, 4)
                    tx = rng.randrange(2)
                if arith == HBD:
                    tx = min(tx, 1 if min(bw, bh) < 16 else 2 if min(bw, bh) < 32 else 3)
                intra = key or rng.random() < 0.4
                b = BlockInfo(x=sx + x, y=sy + y, width=bw, height=bh, tx_size=tx, is_intra=int(intra),
                              y_mode=rng.randrange(10), uv_mode=rng.randrange(10),
                              skip=int(content == "skipped" or rng.random() < 0.2), coeff_offset=coeffs)
                b.ref_frame[0] = 0 if intra else rng.randrange(1, 4)
                for k in range(2):
                    b.mv[0][k] = 0 if intra else rng.randrange(-80, 80)
                recs.append(b)
                coeffs += 6 * 1024 * 2          # more than the largest block's transforms, these included
    blocks = (BlockInfo * len(recs))(*recs)
    gen = np.random.default_rng(rng.randrange(1 << 30))
    dtype = np.int32 if arith == HBD else np.int16
    c = np.where(gen.random(coeffs) < 0.06, gen.integers(-40, 41, coeffs), 0).astype(dtype)
    if arith == HBD:
        c *= 64
    pf = ParsedFrame()
    C.memmove(C.byref(pf), C.byref(header), C.sizeof(ParsedFrame))
    pf.hdr.filter_level = 0
    pf.blocks = C.cast(blocks, C.POINTER(BlockInfo))
    pf.num_blocks = len(recs)
    pf.coeffs = C.cast(C.c_void_p(c.ctypes.data), C.POINTER(C.c_int16))
    pf.num_coeffs = coeffs
    return pf, (blocks, c)


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("content", CONTENT)
@pytest.mark.parametrize("arith, size", [(ARITH_REFCPU, (136, 72)), (ARITH_SPEC, (64, 64)), (ARITH_SPEC, (57, 39)),
                                         (ARITH_SPEC, (136, 72)), (ARITH_SPEC, (201, 131)), (ARITH_FULL, (64, 64)),
                                         (ARITH_FULL, (136, 72)), (HBD, (64, 64)), (HBD, (136, 72))])
def test_off_grid(arith, size, content, seed):
    w, h = size
    if content == "any" and arith in (ARITH_FULL, HBD) and w > 64:
        pytest.skip("edges past the superblock")
    rng = random.Random(seed * 1000 + w)
    syn = Synth(synth_config(2, w, h, seed=seed, gop=2, **({} if arith == ARITH_REFCPU else {"interp_filter": 0})))
    if arith == HBD:
        eng, orc = HbdEngine(), HbdOracleStream()
        sid = eng.open_stream(w, h)
    else:
        gpu, orc = CudaBackend(arith=arith), OracleStream({ARITH_REFCPU: REFCPU, ARITH_SPEC: SPEC, ARITH_FULL: FULL}[arith])
    for f in range(4):
        header = syn.frame(f % 2).contents
        if arith == HBD:
            header.hdr.bit_depth, header.hdr.profile = 10, 2
        pf, keep = _frame(rng, header, arith, w, h, f % 2 == 0, content)
        if arith == HBD:
            want = orc.decode(C.pointer(pf), keep[1])
            assert eng.submit([sid], [(C.pointer(pf), keep[1].ctypes.data)]) == CVP9_OK
            assert eng.wait() == CVP9_OK
            got = eng.get_frame(sid)
        else:
            want = orc.decode(C.pointer(pf))
            assert gpu.decode(C.pointer(pf), f) == CVP9_OK, gpu.last_error()
            rc, got, _ = gpu.get_frame_array(wait=1)
            assert rc == CVP9_OK, gpu.last_error()
        assert np.array_equal(got, want), "frame %d: %d samples differ" % (f, int((got != want).sum()))
