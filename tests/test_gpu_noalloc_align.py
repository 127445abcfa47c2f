"""cuda_reconstruct_noalloc on a caller's memory at any byte: frames carved out of
a pool at odd offsets, which the next picture takes as references, and status
words, must be those at aligned addresses. Sizes: rows of whole words and odd
ones, chroma rows of whole words and not. Tolerance: none."""
import ctypes as C

import numpy as np
import pytest

from compute_vp9_b200 import CVP9_OK, BlockInfo, ParsedFrame, Synth, cuda_lib, i420_size, synth_config

pytestmark = pytest.mark.gpu

GUARD = 64


def _call():
    fn = cuda_lib().cuda_reconstruct_noalloc
    fn.argtypes = [C.POINTER(ParsedFrame), C.POINTER(C.c_void_p), C.POINTER(C.c_uint32), C.POINTER(C.c_uint32),
                   C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    fn.restype = C.c_int
    return fn


def _decode(arith, w, h, offset):
    """Three pictures, each in a pool of its own between guard bytes; their samples."""
    import torch
    fn, n = _call(), i420_size(w, h)
    syn = Synth(synth_config(2, w, h, seed=5, gop=60, intra_in_inter=0.1, interp_filter=0, mv_range_px=48))
    pools = [torch.full((n + 2 * GUARD,), 0xA5, dtype=torch.uint8, device="cuda") for _ in range(3)]
    status = torch.full((8 * 3 + 8,), 0xA5, dtype=torch.uint8, device="cuda")
    sizes = (C.c_uint32 * 8)(*([w] * 8)), (C.c_uint32 * 8)(*([h] * 8))
    keep, refs = [], (C.c_void_p * 8)()
    for f in range(3):
        src = syn.frame(f).contents
        blocks = torch.from_numpy(np.ctypeslib.as_array(C.cast(src.blocks, C.POINTER(C.c_uint8)),
                                                        shape=(src.num_blocks * 32,)).copy()).cuda()
        coeffs = torch.from_numpy(np.ctypeslib.as_array(src.coeffs, shape=(src.num_coeffs,)).copy()).cuda()
        keep += [blocks, coeffs]
        pf = ParsedFrame()
        C.memmove(C.byref(pf), C.byref(src), C.sizeof(ParsedFrame))
        pf.blocks = C.cast(C.c_void_p(blocks.data_ptr()), C.POINTER(BlockInfo))
        pf.coeffs = C.cast(C.c_void_p(coeffs.data_ptr()), C.POINTER(C.c_int16))
        torch.cuda.synchronize()
        out = pools[f].data_ptr() + GUARD + offset
        assert fn(C.byref(pf), refs, *sizes, out, arith, status.data_ptr() + 8 * f + offset, None) == CVP9_OK
        refs = (C.c_void_p * 8)(*([out] * 8))
    torch.cuda.synchronize()
    status = status.cpu().numpy()
    assert all((status[8 * f + offset:8 * f + offset + 4] == 0).all() for f in range(3))
    assert (status == 0xA5).sum() == 8 * 3 + 8 - 12
    for p in pools:
        p = p.cpu().numpy()
        assert (p[:GUARD + offset] == 0xA5).all() and (p[GUARD + offset + n:] == 0xA5).all()
    return [p.cpu().numpy()[GUARD + offset:GUARD + offset + n] for p in pools]


@pytest.mark.parametrize("size", [(64, 64), (352, 288), (353, 289), (254, 130), (200, 120)])
@pytest.mark.parametrize("arith", [0, 1])
def test_any_offset(arith, size):
    want = _decode(arith, *size, 0)
    for offset in (1, 2, 3, 4, 7):
        for f, (g, x) in enumerate(zip(_decode(arith, *size, offset), want)):
            assert np.array_equal(g, x), "offset %d, picture %d: %d bytes differ" % (offset, f, int((g != x).sum()))
