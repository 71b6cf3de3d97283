"""Workloads that the performance of this package is measured on.

Each case is one call (or the few calls that belong together) that an encoder built on the library
makes, through the public entry points of uavs3e_gb300, on seeded synthetic pictures.  Device
buffers are used where the encoder keeps its pictures on the GPU, host buffers where it hands them
over from the host.  All results but the pruning network's are integers and have to stay the same.
"""
import math

import numpy as np
import torch

import uavs3e_gb300 as u
from uavs3e_gb300 import cnn
from uavs3e_gb300.synth import intra_frame, lambda_mv_for_qp, motion_sequence

PAD = 144            # luma padding of reference pictures
PAD_C = 72           # chroma padding
QPS = (27, 32, 37, 42)
SHORTLIST = 5        # modes per CU that the candidate search keeps


def listed():
    return [
        # one small frame handed over from the host (416x240, the low-delay test configuration):
        # upload, one graph replay, download -- latency and launches count
        dict(name="me_240p_host", kind="me", w=416, h=240, refs=2, range=64, host=True),
        # the headline: every block of a 1080p frame against 2 references, pictures on the device
        dict(name="me_1080p", kind="me", w=1920, h=1080, refs=2, range=64, host=False),
        # the whole intra lattice of a 1080p I-frame at the four test QPs (the largest call)
        dict(name="lattice_1080p", kind="lattice", w=1920, h=1080, n_qp=4, ipf=False),
        # the same of a small frame at one QP with the prediction filter, as one slice asks for it
        dict(name="lattice_240p", kind="lattice", w=416, h=240, n_qp=1, ipf=True),
        # the intra decision in the encoder's order (SATD of all modes, candidate list, transform
        # records of the listed modes) on a 720p frame whose sides are not multiples of the CTU
        dict(name="decision_720p", kind="decision", w=1272, h=716, n_qp=4),
        # the encoder's own per-block searches of a 1080p frame as one call list
        dict(name="tz_1080p", kind="tz", w=1920, h=1080, rows=17),
        # predictions of the inter candidates of a 1080p frame: translational and affine CUs
        dict(name="mc_1080p", kind="mc", w=1920, h=1080, rows=17),
        # the affine searches of a 1080p frame
        dict(name="affine_1080p", kind="affine", w=1920, h=1080, rows=17),
        # RDOQ of a frame's transform blocks, and the rate of coded blocks
        dict(name="rdoq_rate_60k", kind="rdoq", n=60000),
        # picture-level estimate of a random-access B picture (both lists, padded references)
        dict(name="lookahead_1080p", kind="lookahead", w=1920, h=1080, l0=1, l1=1, padding=True, range=384),
        # one gradient step of the pruning network at the training batch (forward, loss, backward)
        dict(name="cnn_train_1024", kind="train", batch=1024),
        # the network's split flags and mode logits for all CTUs of a 1080p picture
        dict(name="cnn_infer_1080p", kind="infer", w=1920, h=1080, qp=32),
    ]


def _log(rng, lo, hi, step=1):
    """a size between lo and hi, spread over its logarithm, on a grid of `step`"""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["me", "lattice", "decision", "tz", "mc", "affine", "rdoq", "lookahead", "train", "infer"])
    if kind == "me":
        return dict(kind=kind, w=_log(rng, 200, 1920), h=_log(rng, 120, 1080), refs=rng.randint(1, 3),
                    range=_log(rng, 8, 64), host=rng.random() < 0.5)
    if kind == "lattice":
        return dict(kind=kind, w=_log(rng, 128, 1280, 4), h=_log(rng, 128, 720, 4), n_qp=rng.randint(1, 4),
                    ipf=rng.random() < 0.5)
    if kind == "decision":
        return dict(kind=kind, w=_log(rng, 128, 1280, 4), h=_log(rng, 128, 720, 4), n_qp=rng.randint(1, 4))
    if kind in ("tz", "mc", "affine"):
        w, h = _log(rng, 256, 1920, 2), _log(rng, 128, 1080, 2)
        return dict(kind=kind, w=w, h=h, rows=rng.randint(1, (h + 63) // 64))
    if kind == "rdoq":
        return dict(kind=kind, n=_log(rng, 500, 60000))
    if kind == "lookahead":
        return dict(kind=kind, w=_log(rng, 200, 1920, 2), h=_log(rng, 120, 1080, 2), l0=rng.randint(1, 2),
                    l1=rng.randint(0, 2), padding=rng.random() < 0.5, range=rng.choice([64, 128, 384]))
    if kind == "train":
        return dict(kind=kind, batch=_log(rng, 16, 1024))
    return dict(kind=kind, w=_log(rng, 200, 1920), h=_log(rng, 120, 1080), qp=rng.randint(22, 45))


def _dev(a):
    """a numpy array's bytes on the device"""
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()


def _motion(w, h, n, seed, speed=1.0):
    """n frames of a panned texture with moving objects, `speed` frames of motion apart"""
    rng = np.random.default_rng(seed)
    vel = [tuple(speed * rng.uniform(-3, 3, 2)) for _ in range(12)]
    return motion_sequence(w, h, n, seed=seed, pan=(3.25 * speed, -1.5 * speed), rect_vel=vel)


def _chroma(y):
    """chroma planes of a luma picture: 2x-downsampled, offset by +16 / -16"""
    h, w = y.shape[0] // 2 * 2, y.shape[1] // 2 * 2
    c = y[:h, :w].reshape(h // 2, 2, w // 2, 2).astype(np.int32).mean((1, 3)).astype(np.int32)
    return (np.ascontiguousarray(np.clip(c + d, 0, 255).astype(np.uint8)) for d in (16, -16))


def _blocks(w, h, rows, least=8):
    """(x, y, w, h) of the blocks of the first `rows` CTU rows that lie inside the picture"""
    b = u.me_blocks(w, h)
    b = b[(b[:, 0] + b[:, 2] <= w) & (b[:, 1] + b[:, 3] <= h) & (b[:, 1] < 64 * rows)]
    return b[(b[:, 2] >= least) & (b[:, 3] >= least)]


def _lambda_mv(qp):
    return np.floor(65536.0 * np.sqrt(1.43631 * 2.0 ** ((qp - 16) / 4.0))).astype(np.uint32)


class _Refs:
    """a session that holds two reference pictures (and their chroma), and the next picture"""

    def __init__(self, c, seed, chroma=False):
        w, h = c["w"], c["h"]
        seq = _motion(w, h, 3, seed)
        self.ms = u.MotionSearch(w, h, n_refs=2, search_range=64, pad=PAD)
        for s in range(2):
            self.ms.set_ref(s, seq[1 - s])
            if chroma:
                self.ms.set_ref_chroma(s, *_chroma(seq[1 - s]))
        self.org = torch.from_numpy(seq[2]).cuda()
        self.planes = [self.ms.plane_ptr(s, p) for s in range(2) for p in range(16)]
        self.chroma = [self.ms.chroma_plane_ptr(s, p) for s in range(2) for p in range(2)] if chroma else []


def _prepare_me(c, seed):
    w, h = c["w"], c["h"]
    seq = _motion(w, h, c["refs"] + 1, seed)
    ms = u.MotionSearch(w, h, n_refs=c["refs"], search_range=c["range"], pad=PAD)
    for s in range(1, c["refs"]):
        ms.set_ref(s, seq[c["refs"] - 1 - s])
    ref, org = torch.from_numpy(seq[-2]), torch.from_numpy(seq[-1])
    n = ms.n_results * u.ME_RESULT.itemsize
    if c["host"]:
        return dict(ms=ms, ref=ref.pin_memory(), org=org.pin_memory(), out=torch.empty(n, dtype=torch.uint8).pin_memory())
    return dict(ms=ms, ref=ref.cuda(), org=org.cuda(), out=torch.empty(n, dtype=torch.uint8, device="cuda"))


def _run_me(c, s):
    # the newest picture becomes reference 0, then the frame is searched
    args = (0, s["ref"].data_ptr(), c["w"], s["org"].data_ptr(), c["w"], lambda_mv_for_qp(32), s["out"].data_ptr())
    if c["host"]:
        s["ms"].frame_ptr(*args)
    else:
        s["ms"].frame_graph(*args, stream=torch.cuda.current_stream().cuda_stream)
    return s["out"]


def _intra_pictures(c, seed):
    org = intra_frame(c["w"], c["h"], seed=seed)
    noise = np.random.default_rng(seed).integers(-5, 6, org.shape)
    rec = np.clip(org.astype(int) + noise, 0, 255).astype(np.uint8)
    cus = u.lattice_cus(c["w"], c["h"])
    return dict(org=torch.from_numpy(org).cuda(), rec=torch.from_numpy(rec).cuda(), cus=cus, d_cus=_dev(cus), n=len(cus),
                qps=np.array(QPS[:c["n_qp"]], np.int32))


def _prepare_lattice(c, seed):
    s = _intra_pictures(c, seed)
    s["satd"] = torch.zeros(s["n"] * 33, dtype=torch.int32, device="cuda")
    s["q"] = torch.zeros(s["n"] * 33 * c["n_qp"] * 4, dtype=torch.int32, device="cuda")
    return s


def _lattice(c, s, modes, n_modes, ipf, qps, satd, q):
    u.check(u.lib().uavs3e_cuda_intra_lattice_modes_device(
        s["org"].data_ptr(), c["w"], s["rec"].data_ptr(), c["w"], c["w"], c["h"], s["d_cus"].data_ptr(), s["n"], modes,
        n_modes, ipf, qps.ctypes.data if qps is not None else None, len(qps) if qps is not None else 0, 1,
        satd.data_ptr(), q.data_ptr() if q is not None else None, torch.cuda.current_stream().cuda_stream), "intra_lattice")


def _run_lattice(c, s):
    _lattice(c, s, None, 33, int(c["ipf"]), s["qps"], s["satd"], s["q"])
    return s["satd"], s["q"]


def _prepare_decision(c, seed):
    s = _prepare_lattice(c, seed)
    rng, n, cus = np.random.default_rng(seed + 1), s["n"], s["cus"]
    r = np.zeros(n, dtype=u.RMD_REQ)
    r["satd_row"] = np.arange(n)
    r["pb_w"], r["pb_h"] = cus["w"], cus["h"]
    r["mpm"] = np.sort(rng.integers(0, 33, (n, 2)), axis=1)
    r["fast"] = 1
    r["range"] = rng.integers(256, 512, n)
    r["ctx"] = (rng.integers(8, 1016, (n, 7)) << 1) | rng.integers(0, 2, (n, 7))
    r["sqrt_lambda"] = 30.0
    r["inter_satd"] = np.iinfo(np.uint64).max
    s["reqs"] = _dev(r)
    s["all_satd"] = torch.zeros(n * 33, dtype=torch.int32, device="cuda")
    s["lists"] = torch.zeros(n * u.RMD_OUT.itemsize, dtype=torch.uint8, device="cuda")
    return s


def _run_decision(c, s):
    n = s["n"]
    _lattice(c, s, None, 33, 1, None, s["all_satd"], None)
    u.intra_rmd_device(s["all_satd"].data_ptr(), n, s["reqs"].data_ptr(), n, s["lists"].data_ptr())
    lists = s["lists"].view(torch.int8).view(n, u.RMD_OUT.itemsize)[:, :SHORTLIST]
    modes = torch.where(lists < 0, lists[:, :1], lists).contiguous()      # lists of 4 repeat their first mode
    _lattice(c, s, modes.data_ptr(), SHORTLIST, 1, s["qps"], s["satd"], s["q"])
    return s["all_satd"], s["lists"], s["satd"], s["q"]


def _prepare_tz(c, seed):
    s = _Refs(c, seed)
    rng = np.random.default_rng(seed + 1)
    b = _blocks(c["w"], c["h"], c["rows"])
    n = 2 * len(b)
    r = np.zeros(n, dtype=u.TZ_REQ)
    for i, f in enumerate(("x", "y", "w", "h")):
        r[f] = np.repeat(b[:, i], 2)
    r["ref_slot"] = np.tile([0, 1], len(b))
    r["other_slot"] = 1 - r["ref_slot"]
    r["dist"] = r["ref_slot"] + 1
    r["num_refp"] = rng.integers(1, 5, n)
    r["refi"] = rng.integers(0, r["num_refp"])
    r["mvr"] = rng.integers(0, 5, n)
    r["bi"] = rng.random(n) < 0.3
    r["flags"] = rng.integers(0, 4, n)
    unit = (1 << r["mvr"].astype(int))[:, None]
    r["mvp"] = rng.integers(-200, 201, (n, 2)) // unit * unit
    r["mv"] = (r["mvp"] + rng.integers(-48, 49, (n, 2))) // unit * unit
    r["mv_ipel"] = rng.integers(-40, 41, (n, 2))
    r["other_mv"] = rng.integers(-120, 121, (n, 2))
    r["mot_bits_other"] = rng.integers(2, 24, n)
    r["lambda_mv"] = _lambda_mv(rng.integers(22, 46, n))
    return dict(refs=s, n=n, reqs=_dev(r), out=torch.zeros(n * 2, dtype=torch.int64, device="cuda"))


def _run_tz(c, s):
    f = s["refs"]
    u.me_tz_device((c["w"], c["h"], 1, 384, 16), f.org.data_ptr(), c["w"], f.planes, f.ms.stride, PAD,
                   s["reqs"].data_ptr(), s["n"], s["out"].data_ptr())
    return s["out"]


def _prepare_mc(c, seed):
    s = _Refs(c, seed, chroma=True)
    rng = np.random.default_rng(seed + 1)
    b = _blocks(c["w"], c["h"], c["rows"])
    n = 2 * len(b)
    r = np.zeros(n, dtype=u.MC_REQ)
    for i, f in enumerate(("x", "y", "w", "h")):
        r[f] = np.repeat(b[:, i], 2)
    slot = np.tile([0, 1], len(b)).astype(np.int8)
    r["slot"][:, 0] = slot
    r["slot"][:, 1] = np.where(rng.random(n) < 0.3, 1 - slot, -1)
    r["mv"] = rng.integers(-160, 161, (n, 2, 2))
    size = r["w"].astype(np.int64) * r["h"] * 3 // 2
    r["out_offset"] = np.cumsum(size) - size
    big = _blocks(c["w"], c["h"], c["rows"], 16)
    m = len(big)
    a = np.zeros(m, dtype=u.AFFINE_REQ)
    for i, f in enumerate(("x", "y", "w", "h")):
        a[f] = big[:, i]
    use = rng.integers(1, 4, m)
    for l in range(2):
        a["slot"][:, l] = np.where(use >> l & 1, rng.integers(0, 2, m), -1)
        t = rng.integers(-1200, 1201, (m, 2))                   # translation in 1/16 samples
        k = rng.uniform(-0.25, 0.25, (m, 4))                    # zoom and rotation
        a["cpmv"][:, l, 0] = t
        a["cpmv"][:, l, 1] = t + np.rint(16 * big[:, 2:3] * k[:, :2]).astype(int)
        a["cpmv"][:, l, 2] = t + np.rint(16 * big[:, 3:4] * k[:, 2:]).astype(int)
    a["cp_num"] = rng.integers(2, 4, m)
    a["sub8"] = rng.integers(0, 2, m)
    asize = a["w"].astype(np.int64) * a["h"] * 3 // 2
    a["out_offset"] = np.cumsum(asize) - asize
    return dict(refs=s, n=n, m=m, reqs=_dev(r), areqs=_dev(a),
                out=torch.zeros(int(size.sum()), dtype=torch.uint8, device="cuda"),
                aout=torch.zeros(max(1, int(asize.sum())), dtype=torch.uint8, device="cuda"))


def _run_mc(c, s):
    f = s["refs"]
    cu = (c["w"], c["h"], f.planes, f.ms.stride, PAD, f.chroma, f.ms.chroma_stride(), PAD_C)
    u.mc_cu_device(*cu, s["reqs"].data_ptr(), s["n"], s["out"].data_ptr(), s["out"].numel())
    u.mc_affine_device(*cu, s["areqs"].data_ptr(), s["m"], s["aout"].data_ptr(), s["aout"].numel())
    return s["out"], s["aout"]


def _prepare_affine(c, seed):
    s = _Refs(c, seed)
    rng = np.random.default_rng(seed + 1)
    b = _blocks(c["w"], c["h"], c["rows"], 16)
    n = 2 * len(b)
    r = np.zeros(n, dtype=u.AFFME_REQ)
    for i, f in enumerate(("x", "y", "w", "h")):
        r[f] = np.repeat(b[:, i], 2)
    r["ref_slot"] = np.tile([0, 1], len(b))
    r["other_slot"] = 1 - r["ref_slot"]
    r["num_refp"] = rng.integers(1, 5, n)
    r["refi"] = rng.integers(0, r["num_refp"])
    r["mvr"] = rng.integers(0, 3, n)
    unit = np.array([4, 16, 1])[r["mvr"]][:, None, None]
    bi = rng.random(n) < 0.3
    start = ~bi & (rng.random(n) < 0.6)
    r["flags"] = np.where(bi, u.AFFME_BI, 0) | np.where(start, u.AFFME_UNI_START, 0) | \
        np.where(rng.random(n) < 0.3, u.AFFME_SUB8, 0)
    r["lambda_mv"] = _lambda_mv(rng.integers(22, 46, n))
    r["mot_bits_other"] = rng.integers(2, 24, n)
    t = rng.integers(-700, 701, (n, 2))
    k = np.rint(16 * r["w"][:, None] * rng.uniform(-0.06, 0.06, (n, 2))).astype(int)
    r["mvp"] = np.stack([t, t + k], 1) // unit * unit
    mv = r["mvp"] + rng.integers(-64, 65, (n, 2, 2)) // unit * unit
    mv[start] = 0
    mv[start, 0] = rng.integers(-300, 301, (int(start.sum()), 2))
    r["mv"] = mv
    o = rng.integers(-500, 501, (n, 2))
    r["other_mv"] = np.stack([o, o + rng.integers(-40, 41, (n, 2))], 1)
    return dict(refs=s, n=n, reqs=_dev(r), out=torch.zeros(max(1, n) * 4, dtype=torch.int64, device="cuda"))


def _run_affine(c, s):
    f = s["refs"]
    u.me_affine_device(c["w"], c["h"], f.org.data_ptr(), c["w"], f.planes, f.ms.stride, PAD, s["reqs"].data_ptr(),
                       s["n"], s["out"].data_ptr())
    return s["out"]


def _bin_costs(rng, shape):
    """costs of the two values of a bin, in 1/32768 bits, for models of any skew"""
    p = rng.uniform(0.03, 0.97, shape)
    return np.rint(-32768.0 * np.log2(np.stack([p, 1 - p], -1))).astype(np.int32)


def _prepare_rdoq(c, seed):
    rng, n = np.random.default_rng(seed), c["n"]
    # transform blocks of the 23 shapes 4x4 .. 64x64, as many of each, in any order
    shapes = np.array([(a, b) for a in range(2, 7) for b in range(2, 7) if abs(a - b) <= 3])
    lw, lh = shapes[rng.permutation(n) % len(shapes)].T
    size = 1 << (lw + lh)
    off = np.cumsum(size) - size
    r = np.zeros(n, dtype=u.RDOQ_REQ)
    r["coef_offset"], r["log2w"], r["log2h"] = off, lw, lh
    r["qp"] = rng.integers(22, 46, n)
    r["is_intra"] = rng.integers(0, 2, n)
    r["ch_type"] = np.where((lw > 5) | (lh > 5), 0, rng.integers(0, 3, n))
    r["slice_type"] = rng.integers(1, 4, n)
    r["est"] = rng.integers(0, 8, n)
    r["lambda_"] = np.rint(1.43631 * 2.0 ** ((r["qp"].astype(float) - 16) / 4.0) * 32768).astype(np.int64)
    e = np.zeros(8, dtype=u.RDOQ_EST)
    for i in range(8):
        e[i]["ctp"] = _bin_costs(rng, ())
        for f, shape in (("cbf", (3,)), ("run", (24,)), ("lvl", (24,)), ("lst", (2, 6, 12))):
            e[i][f] = _bin_costs(rng, shape)
    # coefficients: Laplacian, their scale falling with the frequency, residual energies 2 .. 60
    g = torch.Generator("cuda").manual_seed(seed)
    scale = rng.choice([2.0, 6.0, 20.0, 60.0], n) * 2.0 ** (7 - (lw + lh) / 2)
    blk = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.from_numpy(size).cuda())
    at = torch.arange(len(blk), device="cuda") - torch.from_numpy(off).cuda()[blk]
    lwd = torch.from_numpy(lw).cuda()[blk]
    x, y = at & ((1 << lwd) - 1), at >> lwd
    b = torch.rand(len(blk), device="cuda", generator=g) - 0.5
    sc = torch.from_numpy(scale.astype(np.float32)).cuda()[blk] * 2.0 / (1.0 + 0.15 * (x + y))
    v = -torch.sign(b) * torch.log1p(-2.0 * b.abs().clamp(max=0.499999)) * sc
    coefs = v.round().clamp(-32000, 32000).to(torch.int16)
    # levels of coded blocks of the same shapes: plainly quantised at their QP, zero past 32 columns and
    # rows, the first one not zero
    step = torch.from_numpy((2.0 ** (r["qp"] / 8.0 + 7 - (lw + lh) / 2)).astype(np.float32)).cuda()[blk]
    lev = torch.where((x < 32) & (y < 32), torch.sign(v) * torch.floor(v.abs() / step + 0.4), 0.0).to(torch.int16)
    lev = torch.where((at == 0) & (lev == 0), torch.ones_like(lev), lev)
    cum = torch.cumsum((lev != 0).to(torch.int64), 0).cpu().numpy()
    nz = np.diff(np.concatenate([[0], cum[off + size - 1]]))
    q = np.zeros(n, dtype=u.COEF_RATE_REQ)
    q["coef_offset"], q["log2w"], q["log2h"], q["num_sig"] = off, lw, lh, nz
    q["ch_type"] = r["ch_type"] != 0
    q["range"] = rng.integers(256, 512, n)
    for f, m in (("run", 12), ("run_rdoq", 12), ("level", 12), ("last1", 6), ("last2", 12)):
        q[f] = (rng.integers(0, 4, (n, m)) << 11) | (rng.integers(4, 1024, (n, m)) << 1) | rng.integers(0, 2, (n, m))
    return dict(n=n, reqs=_dev(r), ests=_dev(e), src=coefs, coefs=torch.empty_like(coefs), rreqs=_dev(q), levels=lev,
                nz=torch.zeros(n, dtype=torch.int32, device="cuda"),
                rate=torch.zeros(n * u.COEF_RATE_OUT.itemsize, dtype=torch.uint8, device="cuda"))


def _run_rdoq(c, s):
    s["coefs"].copy_(s["src"])          # the call quantises in place: fresh transform output for each pass
    u.rdoq_device(s["reqs"].data_ptr(), s["n"], s["ests"].data_ptr(), 8, s["coefs"].data_ptr(), s["coefs"].numel(),
                  s["nz"].data_ptr())
    u.coef_rate_device(s["rreqs"].data_ptr(), s["n"], s["levels"].data_ptr(), s["levels"].numel(), s["rate"].data_ptr())
    return s["coefs"], s["nz"], s["rate"]


def _prepare_lookahead(c, seed):
    w, h = c["w"], c["h"]
    # POC 0, 8, 16, ...: the picture is POC 8, list 0 holds earlier ones, list 1 later ones
    seq = _motion(w, h, 1 + c["l0"] + c["l1"], seed, 8.0)
    cur = c["l0"]
    uu, vv = _chroma(seq[cur])
    l0, l1 = [cur - 1 - i for i in range(c["l0"])], [cur + 1 + i for i in range(c["l1"])]
    stride = (w + 2 * PAD + 15) // 16 * 16
    ref = {}
    for t in l0 + l1:
        p = np.zeros((h + 2 * PAD, stride), np.uint8)
        p[:, :w + 2 * PAD] = np.pad(seq[t], PAD, mode="edge")
        ref[t] = torch.from_numpy(p).cuda()
    n = (w // 16) * (h // 16)
    cfg = u.loka_cfg(w, h, int(c["padding"]), c["range"], 16, 8 * cur, [8 * t for t in l0], [8 * t for t in l1])
    return dict(cfg=cfg, y=torch.from_numpy(seq[cur]).cuda(), u=torch.from_numpy(uu).cuda(), v=torch.from_numpy(vv).cuda(),
                ref=ref, l0=l0, l1=l1, stride=stride, units=torch.zeros(n * u.LOKA_UNIT.itemsize, dtype=torch.uint8, device="cuda"),
                energy=torch.zeros(n, dtype=torch.int64, device="cuda"), totals=torch.zeros(5, dtype=torch.int64, device="cuda"))


def _run_lookahead(c, s):
    at = PAD * s["stride"] + PAD
    u.loka_units_device(s["cfg"], s["y"].data_ptr(), c["w"], s["u"].data_ptr(), s["v"].data_ptr(), c["w"] // 2,
                        [s["ref"][t].data_ptr() + at for t in s["l0"]], [s["ref"][t].data_ptr() + at for t in s["l1"]],
                        s["stride"], PAD, s["units"].data_ptr(), s["energy"].data_ptr(), s["totals"].data_ptr())
    return s["units"], s["energy"], s["totals"]


def _labels(rng, b):
    lab = np.zeros((b, 40), np.uint8)
    lab[:, :21] = rng.random((b, 21)) < 0.6
    lab[:, 21:37] = np.minimum(rng.geometric(0.12, (b, 16)) - 1, 32)
    return lab


def _ctu_batch(b, seed):
    """b CTUs of textures at random QPs, as the network sees them: [b][64][64][2], bf16"""
    g = torch.Generator("cuda").manual_seed(seed)
    rnd = lambda *s: torch.rand(*s, device="cuda", generator=g)  # noqa: E731
    x = torch.arange(64, device="cuda", dtype=torch.float32)
    ang, per, amp = (2 * math.pi * rnd(b, 1, 1), 6 + 34 * rnd(b, 1, 1), 8 + 60 * rnd(b, 1, 1))
    phase = (x[None, None, :] * torch.cos(ang) + x[None, :, None] * torch.sin(ang)) * (2 * math.pi) / per
    luma = 64 + 128 * rnd(b, 1, 1) + amp * torch.sin(phase) + 12 * (rnd(b, 64, 64) + rnd(b, 64, 64) - 1)
    qp = torch.tensor(QPS, device="cuda", dtype=torch.float32)[(rnd(b) * 4).long().clamp(max=3)]
    out = torch.empty(b, 64, 64, 2, device="cuda")
    out[..., 0] = (luma.round().clamp(0, 255) - 128.0) / 64.0
    out[..., 1] = ((qp - 32.0) / 8.0)[:, None, None]
    return out.to(torch.bfloat16)


def _prepare_train(c, seed):
    net = cnn.PruneNet(c["batch"], seed=seed)
    net.acts[0].copy_(_ctu_batch(c["batch"], seed))
    return dict(net=net, labels=torch.from_numpy(_labels(np.random.default_rng(seed), c["batch"])).cuda())


def _run_train(c, s):
    # no weight update, so that every pass is a step from the same weights
    net = s["net"]
    logits = net.forward()
    loss = net.backward(s["labels"])
    return logits, loss, net.flat_g


def _ctus(c):
    return [(x, y) for y in range(0, c["h"], 64) for x in range(0, c["w"], 64)]


def _prepare_infer(c, seed):
    xy = np.array(_ctus(c), np.int32)
    return dict(net=cnn.PruneNet(len(xy), seed=seed), pic=torch.from_numpy(intra_frame(c["w"], c["h"], seed=seed)).cuda(),
                xy=torch.from_numpy(xy).cuda())


def _run_infer(c, s):
    net = s["net"]
    net.load_input(s["pic"].data_ptr(), c["w"], c["w"], c["h"], s["xy"].data_ptr(), net.B, c["qp"])
    return net.forward()


_PREPARE = dict(me=_prepare_me, lattice=_prepare_lattice, decision=_prepare_decision, tz=_prepare_tz, mc=_prepare_mc,
                affine=_prepare_affine, rdoq=_prepare_rdoq, lookahead=_prepare_lookahead, train=_prepare_train,
                infer=_prepare_infer)
_RUN = dict(me=_run_me, lattice=_run_lattice, decision=_run_decision, tz=_run_tz, mc=_run_mc, affine=_run_affine,
            rdoq=_run_rdoq, lookahead=_run_lookahead, train=_run_train, infer=_run_infer)


def prepare(case, seed):
    u.init(0)
    return case, _PREPARE[case["kind"]](case, seed)


def run(state):
    case, s = state
    return _RUN[case["kind"]](case, s)


def _network(params, x):
    """logits of the network in 64 bits: params [(w [Cout][Kp], b)], x [b][64][64][2]"""
    a = x.permute(0, 3, 1, 2)
    layers = cnn.LAYERS + [cnn.HEAD]
    for i, ((cin, cout, ks, st), (w, b)) in enumerate(zip(layers, params)):
        ho = (a.shape[2] + 2 * (ks // 2) - ks) // st + 1
        col = torch.nn.functional.unfold(a, ks, padding=ks // 2, stride=st)          # [b][cin ks ks][ho ho]
        m = w[:, :ks * ks * cin].reshape(cout, ks * ks, cin).transpose(1, 2).reshape(cout, -1)
        a = (m @ col + b[:, None]).reshape(len(x), cout, ho, ho)
        if i < len(layers) - 1:
            a = torch.relu(a)
    return a.permute(0, 2, 3, 1).reshape(len(x), 16, cnn.HEAD[1])


def _losses(logits, lab):
    """the four loss parts: split64, split32, split16 (binary cross-entropy), modes (softmax)"""
    bce = torch.nn.functional.binary_cross_entropy_with_logits
    y = lab.to(torch.float64)
    cell = logits.reshape(-1, 2, 2, 2, 2, logits.shape[-1])       # [b][qy][cy][qx][cx][channel]
    s64 = logits[:, :, 2].mean(1)
    s32 = cell[..., 1].mean((2, 4)).reshape(-1, 4)
    modes = torch.nn.functional.cross_entropy(logits[:, :, 3:36].reshape(-1, 33), lab[:, 21:37].reshape(-1).long())
    return torch.stack([bce(s64, y[:, 0]), bce(s32, y[:, 1:5]), bce(logits[:, :, 0], y[:, 5:21]), modes])


def exact(case, seed):
    """the pruning network in 64 bits; every other result is an integer"""
    if case["kind"] == "train":
        x = _ctu_batch(case["batch"], seed).double()
        lab = torch.from_numpy(_labels(np.random.default_rng(seed), case["batch"])).cuda()
    elif case["kind"] == "infer":
        pic = torch.from_numpy(intra_frame(case["w"], case["h"], seed=seed)).cuda()
        i = torch.arange(64, device="cuda")
        ctus = torch.stack([pic[(y0 + i).clamp(max=case["h"] - 1)][:, (x0 + i).clamp(max=case["w"] - 1)]
                            for x0, y0 in _ctus(case)]).double()
        x = torch.stack([(ctus - 128.0) / 64.0, torch.full_like(ctus, (case["qp"] - 32.0) / 8.0)], -1)
    else:
        return None
    params = []
    for w, b in cnn.init_params(seed):
        wd = torch.from_numpy(w).cuda().to(torch.bfloat16).double()
        params.append((wd.requires_grad_(), torch.from_numpy(b).cuda().double().requires_grad_()))
    logits = _network(params, x)
    if case["kind"] == "infer":
        return logits.detach()
    loss = _losses(logits, lab)
    loss.sum().backward()
    return logits.detach(), loss.detach(), torch.cat([t.grad.reshape(-1) for p in params for t in p])


def _samples(case, least=8):
    b = _blocks(case["w"], case["h"], case["rows"], least).astype(np.int64)
    return int((b[:, 2] * b[:, 3]).sum()), len(b)


def _lattice_work(w, h, modes, n_qp, satd_only=False):
    c = u.lattice_cus(w, h)
    cw, ch, n = c["w"].astype(np.int64), c["h"].astype(np.int64), len(c)
    kw, kh = np.minimum(cw, 32), np.minimum(ch, 32)
    macs = 0 if satd_only else kw * ch * cw + kh * kw * ch + n_qp * (kh * kw * ch + cw * ch * kw)
    ops = 12 * cw * ch                       # prediction and SATD
    return 2 * w * h + 8 * n + n * modes * (4 + 16 * n_qp), int(modes * (ops + 2 * macs).sum())


def work(case):
    """bytes: inputs read once and results written once; flops: multiplies and adds (absolute
    differences and their sums, butterflies, filter taps, transform products)"""
    k = case["kind"]
    if k == "me":
        n, ctus = case["w"] * case["h"], len(_ctus(case))
        cand = (2 * case["range"] + 1) ** 2
        # the search sums every sample's difference once per candidate; 17 SATDs of ten shapes
        return dict(bytes=n * (1 + case["refs"]) + 32 * 169 * ctus * case["refs"],
                    flops=case["refs"] * n * (2 * cand + 17 * 10 * 8) + n * 15 * 16)
    if k == "lattice":
        b, f = _lattice_work(case["w"], case["h"], 33, case["n_qp"])
        return dict(bytes=b, flops=f)
    if k == "decision":
        b, f = _lattice_work(case["w"], case["h"], 33, 0, True)
        b5, f5 = _lattice_work(case["w"], case["h"], SHORTLIST, case["n_qp"])
        return dict(bytes=b + b5 + len(u.lattice_cus(case["w"], case["h"])) * (u.RMD_REQ.itemsize + 8), flops=f + f5)
    if k == "tz":
        s, n = _samples(case)
        # about 100 candidates of each search and 17 refinement points
        return dict(bytes=3 * case["w"] * case["h"] + 2 * n * (u.TZ_REQ.itemsize + 16), flops=2 * s * (100 * 2 + 17 * 8))
    if k == "mc":
        s, n = _samples(case)
        a, m = _samples(case, 16)
        return dict(bytes=3 * case["w"] * case["h"] + 3 * s + 3 * a // 2 + 2 * n * u.MC_REQ.itemsize + m * u.AFFINE_REQ.itemsize,
                    flops=(3 * s + 3 * a // 2) * 16)
    if k == "affine":
        s, n = _samples(case, 16)
        # about five steps: filters, gradients, 14 sums and a SATD of each sample
        return dict(bytes=3 * case["w"] * case["h"] + 2 * n * (u.AFFME_REQ.itemsize + 32), flops=2 * s * 5 * (32 + 16 + 28 + 8))
    if k == "rdoq":
        # 646 coefficients a block on average over the 23 shapes; both lists of blocks
        return dict(bytes=case["n"] * (646 * 2 * 3 + u.RDOQ_REQ.itemsize + 4 + u.COEF_RATE_REQ.itemsize + u.COEF_RATE_OUT.itemsize),
                    flops=case["n"] * 646 * 2 * 4)
    if k == "lookahead":
        n = (case["w"] // 16) * (case["h"] // 16)
        refs = case["l0"] + case["l1"]
        # some 60 candidates of each search and 13 predictions with their SATDs
        return dict(bytes=case["w"] * case["h"] * (3 + 2 * refs) // 2 + n * (u.LOKA_UNIT.itemsize + 8),
                    flops=n * 256 * (refs * 60 * 2 + 13 * 16))
    b = case["batch"] if k == "train" else len(_ctus(case))
    acts = 64 * 64 * 2 + 32 * 32 * 16 + 16 * 16 * 32 + 8 * 8 * 32 + 4 * 4 * 64
    fwd, h = 0, 64
    for cin, cout, ks, st in cnn.LAYERS + [cnn.HEAD]:
        h = (h + 2 * (ks // 2) - ks) // st + 1
        fwd += 2 * b * h * h * cout * ks * ks * cin
    if k == "infer":
        return dict(bytes=case["w"] * case["h"] + b * (acts * 2 * 2 + 16 * 48 * 4), flops=fwd)
    return dict(bytes=b * (acts * 2 * 4 + 16 * 48 * (4 * 2 + 2 * 2) + 40), flops=int(cnn.step_flops(b)))
