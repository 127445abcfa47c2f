"""What this framework's users have it do, as cases that can be timed.

A case is a dict of plain values:

  api      which public entry point the pass goes through:
             "noalloc"  cuda_reconstruct_noalloc, one call per picture, all
                        buffers the caller's, on a torch stream
             "stream"   the drop-in backend (cuda_decode_frame /
                        cuda_get_frame): one player, host arrays in, host
                        planes out, three pictures in flight
             "batch"    cvp9_batch_*: one picture of many streams per step
             "hbd"      cvp9_hbd_*: the same for 10-bit pictures
  arith    0 REFCPU, 1 SPEC, 2 FULL (10-bit: always FULL's rules)
  content  the synthetic generator's preset: 1 = 8x8 blocks and transforms,
           5% coefficients; 2 = blocks 8..64, transforms 4x4..32x32, 2..20%
           coefficients, three references, 5% intra blocks in inter pictures
  sizes    the streams, "WxH*count" joined by commas
  pics     "key": key pictures; "inter": inter pictures on references the
           handle already holds; "gop": a key picture and inter pictures
  steps    pictures of each stream in one pass
  inputs   "device": parsed arrays in device memory; "host": dense arrays in
           host memory; "lists": (index, value) coefficient lists
  deliver  "all": every picture comes back to the host; "last": only the
           last one (a seek, a thumbnail or a frame step decodes the
           pictures before it for their samples as references only)

Outputs are whole samples (uint8, or uint16 for 10-bit pictures): there is no
floating result.
"""
import ctypes as C
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from compute_vp9_b200 import (BlockInfo, CudaBackend, Cvp9Error, FrameInfo, ParsedFrame, Synth, cuda_lib,
                              i420_size, synth_config)
from compute_vp9_b200.batch import DEVICE_INPUTS, NO_OUTPUT, Batch, CoeffList
from compute_vp9_b200.hbd import HBD_DEVICE_INPUTS, HBD_NO_OUTPUT, HbdEngine, HbdFrameInfo, i420_samples

DISTINCT = 3          # parsed pictures of a stream: a key picture, two inter pictures taken in turn
TUNE_STEPS = 24       # a long-lived engine is past its tuner's trials, two steps per configuration
HBD_LEVEL_STEP = 288  # 10-bit levels: |level| <= 512 reaches +-2^17 dequantised
HBD_CONTENT = dict(tx_weights=(10, 15, 25, 50), density_min=0.10, density_max=0.10, mv_range_px=256,
                   interp_filter=2, nrefs=3, lf_level=-1, intra_in_inter=0.0)


def _case(api, arith, content, sizes, pics, steps, inputs, deliver, **name):
    return dict(name, api=api, arith=arith, content=content, sizes=sizes, pics=pics, steps=steps, inputs=inputs,
                deliver=deliver)


def listed():
    return [
        # a host framework that owns all device memory decodes one small picture: the smallest call
        _case("noalloc", 0, 1, "352x288*1", "inter", 1, "device", "all", name="noalloc_inter_352x288"),
        # the same caller opens a 1080p stream: a key picture and the inter pictures after it, shader arithmetic
        _case("noalloc", 1, 2, "1920x1080*1", "gop", 3, "device", "all", name="noalloc_gop_spec_1080p"),
        # a player on the drop-in backend, the reference benchmark's 720p content
        _case("stream", 0, 1, "1280x720*1", "inter", 3, "host", "all", name="player_720p"),
        # a player opening a 1080p stream with the complete VP9 arithmetic
        _case("stream", 2, 2, "1920x1080*1", "gop", 3, "host", "all", name="player_gop_full_1080p"),
        # the headline workload's step: many 1080p streams, inter pictures, inputs on the device
        _case("batch", 0, 1, "1920x1080*32", "inter", 8, "device", "last", name="batch_inter_1080p_x32"),
        # mixed block and transform sizes at a width that is not a multiple of 4
        _case("batch", 0, 2, "1366x768*24", "inter", 8, "device", "last", name="batch_mixed_1366x768_x24"),
        # streams joined at their key pictures (a GOP boundary, a channel change)
        _case("batch", 0, 1, "1920x1080*16", "key", 1, "device", "last", name="batch_key_1080p_x16"),
        # the shader arithmetic on inter pictures
        _case("batch", 1, 1, "1920x1080*16", "inter", 8, "device", "last", name="batch_spec_1080p_x16"),
        # the complete VP9 arithmetic: a key picture, then inter pictures with some intra blocks
        _case("batch", 2, 2, "1920x1080*8", "gop", 5, "device", "last", name="batch_gop_full_1080p_x8"),
        # one serving step of uneven streams, coefficient lists from the parser, every picture delivered
        _case("batch", 0, 2, "640x360*8,1280x720*6,1920x1080*4,3840x2160*2", "inter", 2, "lists", "all",
              name="serve_mix_x20"),
        # 10-bit 2160p streams, inter pictures: the largest samples and transforms
        _case("hbd", 2, 2, "3840x2160*6", "inter", 6, "device", "last", name="hbd_inter_2160p_x6"),
        # 10-bit key pictures
        _case("hbd", 2, 2, "1920x1080*8", "key", 1, "device", "last", name="hbd_key_1080p_x8"),
    ]


def _size(rng, most, multiple):
    """A picture of 64x64 up to `most` samples, spread over the logarithm; multiple 1: odd sizes too."""
    px = 64 * 64 * (most / (64.0 * 64.0)) ** rng.random()
    w = px ** 0.5 * rng.choice([1.0, 1.15, 1.333, 1.333, 0.75])
    return [max(64, int(v) // multiple * multiple) for v in (w, px / w)]


def draw(rng):
    api = rng.choice(["noalloc", "stream", "batch", "batch", "batch", "hbd"])
    arith = rng.choice([0, 1] if api == "noalloc" else [2] if api == "hbd" else [0, 0, 1, 2])
    content = 2 if api == "hbd" else rng.choice([1, 2])
    pics = rng.choice(["key", "inter", "inter", "gop"])
    multiple = 8 if arith == 2 else rng.choice([1, 2, 8])
    streams = 1 if api in ("noalloc", "stream") else int(round(24 ** rng.random()))
    most = min(1920 * 1080, 8 * 1920 * 1080 // streams)
    w, h = _size(rng, most, multiple)
    steps = rng.choice([1, 2, 3]) if api in ("noalloc", "stream") else rng.choice([1, 2, 4, 5])
    if pics == "gop":
        steps = max(steps, 2)
    inputs = "device" if api == "noalloc" else "host" if api == "stream" else rng.choice(["device", "device", "host",
                                                                                         "lists"])
    deliver = "all" if api in ("noalloc", "stream") else rng.choice(["last", "all"])
    if deliver == "all":      # every delivered picture is read when the pass ends: as many as stay valid
        steps = min(steps, 2 if api == "hbd" else max(2, 60 // streams))
    return _case(api, arith, content, "%dx%d*%d" % (w, h, streams), pics, steps, inputs, deliver)


def _streams(case):
    out = []
    for part in case["sizes"].split(","):
        size, count = part.split("*")
        w, h = size.split("x")
        out += [(int(w), int(h))] * int(count)
    return out


def _schedule(case):
    """Which of a stream's parsed pictures each step of a pass takes."""
    n = case["steps"]
    if case["pics"] == "key":
        return [0] * n
    inter = [1 + t % (DISTINCT - 1) for t in range(n)]
    return inter if case["pics"] == "inter" else [0] + inter[: n - 1]


def work(case):
    """Bytes: every sample written, a reference sample read per inter sample, 4 per nonzero coefficient that the
    arithmetic reads, 32 per block record. Operations: the interpolation filter's multiply-adds and the separable
    inverse transforms' (three per sample and pass for the blocks that carry coefficients)."""
    total = ops = 0.0
    hbd = case["api"] == "hbd"
    for w, h in _streams(case):
        samples = w * h + 2 * ((w + 1) // 2) * ((h + 1) // 2)
        coded = w * h if case["arith"] == 0 else samples   # REFCPU adds a residual to luma only
        density = 0.10 if hbd else 0.05 if case["content"] == 1 else 0.11
        blocks = w * h / (64.0 if case["content"] == 1 else 168.0)
        for f in _schedule(case):
            total += samples * (2 if hbd else 1) * (2 if f else 1) + 4 * density * coded + 32 * blocks
            ops += samples * (0 if f == 0 else 6 if case["arith"] == 0 else 32) + 12.0 * coded
    return {"bytes": total, "flops": ops}


# ── inputs ────────────────────────────────────────────────────────────────

def _generate(case, seed):
    """Parsed pictures of every stream: [stream][picture] -> (header, block bytes, coefficients)."""
    hbd = case["api"] == "hbd"
    need = sorted(set(_schedule(case)) | {0})
    extra = dict(HBD_CONTENT) if hbd else {}
    if case["arith"] == 1:
        extra["interp_filter"] = 0        # the shaders hold the regular filter only

    def one(args):
        k, (w, h) = args
        syn = Synth(synth_config(case["content"], w, h, seed=(int(seed) << 8) + k, **extra))
        pics = {}
        for f in need:
            pf = syn.frame(f).contents
            blocks = np.ctypeslib.as_array(C.cast(pf.blocks, C.POINTER(C.c_uint8)),
                                           shape=(pf.num_blocks * 32,)).copy()
            coeffs = np.ctypeslib.as_array(pf.coeffs, shape=(pf.num_coeffs,))
            coeffs = coeffs.astype(np.int32) * np.int32(HBD_LEVEL_STEP) if hbd else coeffs.copy()
            hdr = ParsedFrame()
            C.memmove(C.byref(hdr), C.byref(pf), C.sizeof(ParsedFrame))
            if hbd:
                hdr.hdr.bit_depth, hdr.hdr.profile = 10, 2
            pics[f] = (hdr, blocks, coeffs)
        syn.close()
        return pics

    jobs = list(enumerate(_streams(case)))
    with ThreadPoolExecutor(min(len(jobs), os.cpu_count() or 1)) as pool:
        return list(pool.map(one, jobs))


def _pinned(array):
    t = torch.empty(max(1, array.nbytes), dtype=torch.uint8, pin_memory=True)
    t.numpy()[: array.nbytes] = array.view(np.uint8).reshape(-1)
    return t


def _parsed(hdr, blocks, coeffs):
    pf = ParsedFrame()
    C.memmove(C.byref(pf), C.byref(hdr), C.sizeof(ParsedFrame))
    pf.blocks = C.cast(C.c_void_p(blocks), C.POINTER(BlockInfo))
    pf.coeffs = C.cast(C.c_void_p(coeffs), C.POINTER(C.c_int16))
    return pf


class _State:
    """The handle, the parsed pictures and whatever memory they live in."""

    def __init__(self, case):
        self.case = case
        self.schedule = _schedule(case)
        self.keep = []

    def view(self, pointer, count, dtype):
        """`count` samples at `pointer`, in memory of the handle that the view keeps open."""
        buf = ((C.c_uint16 if dtype == np.uint16 else C.c_uint8) * count).from_address(
            C.cast(pointer, C.c_void_p).value)
        buf.owner = self
        return np.frombuffer(buf, dtype=dtype)


def prepare(case, seed):
    pics = _generate(case, seed)
    s = _State(case)
    s.sizes = _streams(case)
    s.n = len(s.sizes)
    s.pf, s.co, s.lists = [], [], []
    hbd = case["api"] == "hbd"
    for per in pics:
        row, addr, lists = {}, {}, {}
        for f, (hdr, blocks, coeffs) in per.items():
            if case["inputs"] == "device":
                mem = [torch.from_numpy(blocks).cuda(), torch.from_numpy(coeffs).cuda()]
                b, c = (t.data_ptr() for t in mem)
            elif case["api"] == "stream":     # the parser's own arrays
                mem = [blocks, coeffs]
                b, c = (a.ctypes.data for a in mem)
            else:
                mem = [_pinned(blocks), _pinned(coeffs if case["inputs"] == "host" else coeffs[:0])]
                b, c = (t.data_ptr() for t in mem)
            if case["inputs"] == "lists":
                pos = np.flatnonzero(coeffs).astype(np.uint32)
                entries = [_pinned(pos), _pinned(coeffs[pos])]
                mem += entries
                lists[f] = (int(pos.size), entries[0].data_ptr(), entries[1].data_ptr())
                if not hbd:
                    lists[f] = CoeffList(*lists[f])
            s.keep += mem
            row[f], addr[f] = _parsed(hdr, b, None if hbd else c), c
        s.pf.append(row)
        s.co.append(addr)
        s.lists.append(lists)
    {"noalloc": _open_noalloc, "stream": _open_stream, "batch": _open_batch, "hbd": _open_hbd}[case["api"]](s)
    return s


def run(state):
    return {"noalloc": _run_noalloc, "stream": _run_stream, "batch": _run_batch,
            "hbd": _run_hbd}[state.case["api"]](state)


def _check(rc, what):
    if rc != 0:
        raise Cvp9Error(rc, what)


# ── cuda_reconstruct_noalloc ──────────────────────────────────────────────

def _open_noalloc(s):
    s.fn = cuda_lib().cuda_reconstruct_noalloc
    s.fn.argtypes = [C.POINTER(ParsedFrame), C.POINTER(C.c_void_p), C.POINTER(C.c_uint32), C.POINTER(C.c_uint32),
                     C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    s.fn.restype = C.c_int
    w, h = s.sizes[0]
    s.widths, s.heights = (C.c_uint32 * 8)(*([w] * 8)), (C.c_uint32 * 8)(*([h] * 8))
    s.out = [torch.empty(i420_size(w, h), dtype=torch.uint8, device="cuda") for _ in range(len(s.schedule) + 1)]
    s.status = torch.zeros(len(s.schedule) + 1, dtype=torch.int32, device="cuda")
    # the pool before each picture: a key picture fills it, an inter picture refreshes LAST (slot 0)
    pool, s.refs = [s.out[0]] * 8, []
    for t, f in enumerate(s.schedule):
        s.refs.append((C.c_void_p * 8)(*([0] * 8 if f == 0 else [p.data_ptr() for p in pool])))
        pool = [s.out[t + 1]] * 8 if f == 0 else [s.out[t + 1]] + pool[1:]
    s.stream = torch.cuda.current_stream().cuda_stream
    _noalloc(s, 0, (C.c_void_p * 8)(), 0)      # the reference picture that "inter" starts from


def _noalloc(s, f, refs, k):
    _check(s.fn(C.byref(s.pf[0][f]), refs, s.widths, s.heights, s.out[k].data_ptr(), s.case["arith"],
                s.status.data_ptr() + 4 * k, s.stream), "cuda_reconstruct_noalloc")


def _run_noalloc(s):
    for t, f in enumerate(s.schedule):
        _noalloc(s, f, s.refs[t], t + 1)
    return s.out[1:] + [s.status]


# ── the drop-in backend ───────────────────────────────────────────────────

def _open_stream(s):
    s.be = CudaBackend(arith=s.case["arith"])
    s.info = [FrameInfo() for _ in s.schedule]
    for t in range(TUNE_STEPS):
        _check(s.be.decode(C.pointer(s.pf[0][s.schedule[t % len(s.schedule)] if t else 0]), t), "cuda_decode_frame")
        _check(s.be.get_frame(wait=1)[0], "cuda_get_frame")
    _check(s.be.decode(C.pointer(s.pf[0][0]), 0), "cuda_decode_frame")
    _check(s.be.get_frame(wait=1)[0], "cuda_get_frame")


def _run_stream(s):
    for t, f in enumerate(s.schedule):
        _check(s.be.decode(C.pointer(s.pf[0][f]), t), "cuda_decode_frame")
    out = []
    for _ in s.schedule:
        rc, info = s.be.get_frame(wait=1)
        _check(rc, "cuda_get_frame")
        out.append(s.view(info.plane_y, i420_size(info.width, info.height), np.uint8))
    return out


# ── the batch engine ──────────────────────────────────────────────────────

def _flags(case, t, device, no_output):
    last = t == case["steps"] - 1
    return (device if case["inputs"] == "device" else 0) | (0 if case["deliver"] == "all" or last else no_output)


def _batch_step(s, f, flags):
    pfs = [C.pointer(s.pf[k][f]) for k in range(s.n)]
    if s.case["inputs"] == "lists":
        s.eng.submit_sparse(s.sids, pfs, [s.lists[k][f] for k in range(s.n)], flags=flags)
    else:
        s.eng.submit(s.sids, pfs, flags=flags)


def _open_batch(s):
    s.eng = Batch(arith=s.case["arith"], hbm_budget=16 << 30)
    for size in sorted(set(s.sizes)):
        s.eng.reserve(size[0], size[1], s.sizes.count(size))
    s.sids = [s.eng.open_stream(w, h) for w, h in s.sizes]
    quiet = _flags(s.case, -1, DEVICE_INPUTS, 0) | NO_OUTPUT
    for t in range(TUNE_STEPS):
        _batch_step(s, s.schedule[t % len(s.schedule)] if t else 0, quiet)
        _check(s.eng.wait(), "cvp9_batch_wait")
    _batch_step(s, 0, quiet)
    _check(s.eng.wait(), "cvp9_batch_wait")


def _run_batch(s):
    seqs = []
    for t, f in enumerate(s.schedule):
        flags = _flags(s.case, t, DEVICE_INPUTS, NO_OUTPUT)
        _batch_step(s, f, flags)
        if not flags & NO_OUTPUT:
            seqs.append(s.eng.last_seq())
    _check(s.eng.wait(), "cvp9_batch_wait")
    out = []
    for seq in seqs:
        for sid in s.sids:
            rc, info = s.eng.get_frame_at(sid, seq)
            _check(rc, "cvp9_batch_get_frame_at")
            out.append(s.view(info.plane_y, i420_size(info.width, info.height), np.uint8))
    return out


# ── the 10-bit engine ─────────────────────────────────────────────────────

def _hbd_step(s, f, flags):
    pfs = [C.pointer(s.pf[k][f]) for k in range(s.n)]
    if s.case["inputs"] == "lists":
        rc = s.eng.submit_sparse(s.sids, pfs, [s.lists[k][f] for k in range(s.n)], flags=flags)
    else:
        rc = s.eng.submit(s.sids, [(pfs[k], s.co[k][f]) for k in range(s.n)], flags=flags)
    _check(rc, "cvp9_hbd_submit")


def _open_hbd(s):
    s.eng = HbdEngine()
    s.get = cuda_lib().cvp9_hbd_get_frame
    s.sids = [s.eng.open_stream(w, h) for w, h in s.sizes]
    device = HBD_DEVICE_INPUTS if s.case["inputs"] == "device" else 0
    for f in (0, s.schedule[-1], 0):
        _hbd_step(s, f, device)
    _check(s.eng.wait(), "cvp9_hbd_wait")


def _run_hbd(s):
    out = []
    for t, f in enumerate(s.schedule):
        flags = _flags(s.case, t, HBD_DEVICE_INPUTS, HBD_NO_OUTPUT)
        _hbd_step(s, f, flags)
        if flags & HBD_NO_OUTPUT:
            continue
        _check(s.eng.wait(), "cvp9_hbd_wait")
        for sid in s.sids:
            info = HbdFrameInfo()
            _check(s.get(s.eng._h, sid, C.byref(info)), "cvp9_hbd_get_frame")
            out.append(s.view(info.plane_y, i420_samples(info.width, info.height), np.uint16))
    return out
