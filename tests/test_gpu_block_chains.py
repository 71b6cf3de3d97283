"""GPU: the grouped block chains of RDOQ and the coefficient rate at the sizes where the grouping
and the listing can go wrong (block counts around a warp and a bucket table, blocks that start off
the 16-byte grid, chains of every length up to a full 64x64 block, calls in flight on two streams)
bit-exact against the oracle."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))
import cases  # noqa: E402

COUNTS = (1, 31, 33, 256, 257)


def _shift(reqs, coefs, by):
    """the same blocks `by` samples further into the array"""
    r = reqs.copy()
    r["coef_offset"] += by
    return r, np.concatenate([np.full(by, 77, np.int16), coefs])


@pytest.mark.gpu
@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("by", (0, 3))
def test_rdoq_block_counts_and_alignment(gpu, oracle, n, by):
    reqs, ests, coefs = cases.rdoq_inputs(oracle, dict(n=n, k=3), 4000 + n)
    reqs, coefs = _shift(reqs, coefs, by)
    want_c, got_c = coefs.copy(), coefs.copy()
    want = oracle.rdoq(reqs, ests, want_c)
    assert np.array_equal(gpu.rdoq(reqs, ests, got_c), want)
    assert np.array_equal(got_c, want_c)


def _rate_device(gpu, levels, reqs, stream=None):
    import torch
    d = [torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).copy()).cuda() for a in (levels, reqs)]
    out = torch.zeros(len(reqs) * gpu.COEF_RATE_OUT.itemsize, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    gpu.coef_rate_device(d[1].data_ptr(), len(reqs), d[0].data_ptr(), levels.size, out.data_ptr(), stream)
    return d, out


@pytest.mark.gpu
@pytest.mark.parametrize("n", COUNTS)
def test_coef_rate_block_counts(gpu, oracle, n):
    import torch
    levels, reqs = cases.coef_rate_inputs(np.random.default_rng(600 + n), n)
    keep, out = _rate_device(gpu, levels, reqs)
    torch.cuda.synchronize()
    assert out.cpu().numpy().tobytes() == oracle.coef_rate(levels, reqs).tobytes()


def _chains(gpu, rng):
    """64x64 blocks with 1, 2, ... 4096 levels: magnitudes up to the escapes, dense and sparse"""
    counts = [1, 2, 15, 16, 17, 100, 1000, 2047, 4095, 4096]
    levels = np.zeros((len(counts), 4096), np.int16)
    for k, c in enumerate(counts):
        at = rng.permutation(4096)[:c]
        levels[k, at] = rng.integers(1, 14, c) * rng.choice([-1, 1], c)
    levels[-1, :8] = (-32768, 32767, 9, 10, -1, 1, 8, -9)
    r = np.zeros(len(counts), dtype=gpu.COEF_RATE_REQ)
    r["coef_offset"] = np.arange(len(counts)) * 4096
    r["log2w"] = r["log2h"] = 6
    r["num_sig"] = (levels != 0).sum(1)
    r["range"] = rng.integers(256, 512, len(counts))
    for f, m in (("run", 12), ("run_rdoq", 12), ("level", 12), ("last1", 6), ("last2", 12)):
        r[f] = cases.coef_models(rng, m * len(counts)).reshape(-1, m)
    return levels.ravel(), r


@pytest.mark.gpu
def test_coef_rate_chain_lengths_on_two_streams(gpu, oracle):
    import torch
    sets = [_chains(gpu, np.random.default_rng(s)) for s in (1, 2, 3, 4)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [_rate_device(gpu, lv, rq, streams[k % 2].cuda_stream) for k, (lv, rq) in enumerate(sets)]
    torch.cuda.synchronize()
    for (lv, rq), (keep, out) in zip(sets, got):
        assert out.cpu().numpy().tobytes() == oracle.coef_rate(lv, rq).tobytes()


def _rdoq_device(gpu, reqs, ests, coefs, stream=None, est_shift=0):
    """the call on device copies; the estimates start est_shift bytes off a 256-byte boundary"""
    import torch
    e = np.ascontiguousarray(ests).view(np.uint8).reshape(-1)
    d_e = torch.zeros(len(e) + 256, dtype=torch.uint8, device="cuda")
    d_e[est_shift:est_shift + len(e)] = torch.from_numpy(e.copy()).cuda()
    d_r = torch.from_numpy(np.ascontiguousarray(reqs).view(np.uint8).reshape(-1).copy()).cuda()
    d_c = torch.from_numpy(coefs.copy()).cuda()
    nz = torch.zeros(len(reqs), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    gpu.rdoq_device(d_r.data_ptr(), len(reqs), d_e.data_ptr() + est_shift, len(ests), d_c.data_ptr(), coefs.size,
                    nz.data_ptr(), stream)
    return d_c, nz, (d_e, d_r)


def _check_rdoq(oracle, reqs, ests, coefs, d_c, nz):
    want_c = coefs.copy()
    want = oracle.rdoq(reqs, ests, want_c)
    assert np.array_equal(nz.cpu().numpy(), want)
    assert np.array_equal(d_c.cpu().numpy(), want_c)


@pytest.mark.gpu
@pytest.mark.parametrize("est_shift,n", ((0, 70), (4, 70), (4, 900), (8, 70), (8, 900)))
def test_rdoq_estimates_off_16_bytes(gpu, oracle, est_shift, n):
    import torch
    reqs, ests, coefs = cases.rdoq_inputs(oracle, dict(n=n, k=3), 4400 + n)
    d_c, nz, keep = _rdoq_device(gpu, reqs, ests, coefs, est_shift=est_shift)
    torch.cuda.synchronize()
    _check_rdoq(oracle, reqs, ests, coefs, d_c, nz)


@pytest.mark.gpu
def test_rdoq_lists_on_two_streams(gpu, oracle):
    import torch
    sets = [cases.rdoq_inputs(oracle, dict(n=n, k=2), 4500 + n) for n in (900, 3, 90, 801)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [_rdoq_device(gpu, *s, stream=streams[k % 2].cuda_stream) for k, s in enumerate(sets)]
    torch.cuda.synchronize()
    for s, (d_c, nz, keep) in zip(sets, got):
        _check_rdoq(oracle, *s, d_c, nz)


class _Graph:
    """what a capture of `calls` on a stream gives, by the driver's own interface"""

    def __init__(self, stream, calls):
        import ctypes
        self.c, self.L, self.execs = ctypes, ctypes.CDLL("libcuda.so.1"), []
        self.handle = ctypes.c_void_p()
        self.ok(self.L.cuStreamBeginCapture_v2(ctypes.c_void_p(stream), 0))
        calls()
        self.ok(self.L.cuStreamEndCapture(ctypes.c_void_p(stream), ctypes.byref(self.handle)))

    def ok(self, rc):
        assert rc == 0, f"CUDA driver error {rc}"

    def instantiate(self, graph=None):
        e = self.c.c_void_p()
        self.ok(self.L.cuGraphInstantiateWithFlags(self.c.byref(e), graph or self.handle, self.c.c_ulonglong(0)))
        self.execs.append(e)
        return e

    def launch(self, e, stream):
        self.ok(self.L.cuGraphLaunch(e, self.c.c_void_p(stream)))

    def parent(self):
        """a graph with this one as its only, child, node"""
        g, node = self.c.c_void_p(), self.c.c_void_p()
        self.ok(self.L.cuGraphCreate(self.c.byref(g), 0))
        self.ok(self.L.cuGraphAddChildGraphNode(self.c.byref(node), g, None, self.c.c_size_t(0), self.handle))
        return g

    def destroy(self, *graphs):
        for e in self.execs:
            self.ok(self.L.cuGraphExecDestroy(e))
        for g in graphs:
            self.ok(self.L.cuGraphDestroy(g))


@pytest.mark.gpu
@pytest.mark.parametrize("n", (3, 1000))
def test_captured_block_lists(gpu, oracle, n):
    # one capture of both calls, replayed on new blocks by two executables of the graph and as a child of
    # another graph, after the captured one itself is gone
    import torch
    rd = [cases.rdoq_inputs(oracle, dict(n=n, k=2), 4600 + n)]
    for k in range(3):
        r, e, c = rd[0]
        rng = np.random.default_rng(k)
        rd.append((r, e, np.clip(c.astype(int) * rng.choice([-1, 1], c.size) + rng.integers(-3, 4, c.size), -32768, 32767).astype(np.int16)))
    levels, rreqs = cases.coef_rate_inputs(np.random.default_rng(700 + n), n)
    d_c, nz, keep = _rdoq_device(gpu, *rd[0])                          # tables and pools exist from here on
    d_e, d_r = keep
    rate_keep, rate = _rate_device(gpu, levels, rreqs)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    st = s.cuda_stream

    def calls():
        gpu.rdoq_device(d_r.data_ptr(), n, d_e.data_ptr(), 2, d_c.data_ptr(), rd[0][2].size, nz.data_ptr(), st)
        gpu.coef_rate_device(rate_keep[1].data_ptr(), n, rate_keep[0].data_ptr(), levels.size, rate.data_ptr(), st)

    g = _Graph(st, calls)
    want_rate = oracle.coef_rate(levels, rreqs).tobytes()
    parent = g.parent()
    runs = [g.instantiate(), g.instantiate(), g.instantiate(parent)]
    g.ok(g.L.cuGraphDestroy(g.handle))
    for (r, e, c), x in zip(rd[1:], runs):
        d_c.copy_(torch.from_numpy(c))
        nz.fill_(-5)
        rate.zero_()
        torch.cuda.synchronize()
        g.launch(x, st)
        # a call outside the graph while it runs
        other, onz, okeep = _rdoq_device(gpu, *rd[0])
        torch.cuda.synchronize()
        _check_rdoq(oracle, r, e, c, d_c, nz)
        _check_rdoq(oracle, *rd[0], other, onz)
        assert rate.cpu().numpy().tobytes() == want_rate
    g.destroy(parent)


@pytest.mark.gpu
def test_captured_workspaces_are_given_back(gpu, oracle):
    import torch
    reqs, ests, coefs = cases.rdoq_inputs(oracle, dict(n=8, k=1), 4700)
    coefs = np.concatenate([coefs, np.zeros((8 << 20) - coefs.size, np.int16)])     # 32 MB of workspace a call
    d_c, nz, (d_e, d_r) = _rdoq_device(gpu, reqs, ests, coefs)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    free = []
    for k in range(48):
        g = _Graph(s.cuda_stream, lambda: gpu.rdoq_device(d_r.data_ptr(), 8, d_e.data_ptr(), 1, d_c.data_ptr(), coefs.size,
                                                          nz.data_ptr(), s.cuda_stream))
        x = g.instantiate()
        g.launch(x, s.cuda_stream)
        torch.cuda.synchronize()
        g.destroy(g.handle)
        free.append(torch.cuda.mem_get_info()[0])
    assert free[7] - free[-1] < 512 << 20, (free[7], free[-1])           # 40 calls' blocks would be 1.3 GB


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.gpu
@pytest.mark.parametrize("extra", (-1, 0, 1, 33))
@pytest.mark.parametrize("by", (0, 3))
def test_rdoq_list_lengths(gpu, oracle, extra, by):
    # around the length from which blocks are grouped by their chains (5 per SM); some outside the domain
    n = 5 * _sms() + extra
    reqs, ests, coefs = cases.rdoq_inputs(oracle, dict(n=n, k=3), 4800 + extra)
    reqs, coefs = _shift(reqs, coefs, by)
    bad = np.arange(n) % 97 == 5
    want_c, got_c = coefs.copy(), coefs.copy()
    want = np.full(n, -1, np.int32)
    want[~bad] = oracle.rdoq(reqs[~bad], ests, want_c)
    reqs["qp"][bad] = 80
    assert np.array_equal(gpu.rdoq(reqs, ests, got_c), want)
    assert np.array_equal(got_c, want_c)


@pytest.mark.gpu
@pytest.mark.parametrize("extra", (-1, 0, 1, 33))
def test_coef_rate_list_lengths(gpu, oracle, extra):
    # around the length from which blocks are grouped by their chains (6 per SM); each block from two coder
    # states, some requests outside the domain
    n = 6 * _sms() + extra
    levels, reqs = cases.coef_rate_inputs(np.random.default_rng(800 + extra), (n + 1) // 2)
    other = reqs.copy()
    other["range"] = 256 + (reqs["range"] + 100) % 256
    reqs = np.concatenate([reqs, other])[:n]
    reqs["range"][::89] = 512
    reqs["num_sig"][7::101] = 4096
    bad = np.arange(n) % 89 == 0
    bad[7::101] = True
    want = np.zeros(n, dtype=gpu.COEF_RATE_OUT)
    want[~bad] = oracle.coef_rate(levels, reqs[~bad])
    want["bits"][bad] = 0xFFFFFFFF                       # and the state as it was
    for f in ("range", "run", "run_rdoq", "level", "last1", "last2"):
        want[f][bad] = reqs[f][bad]
    assert gpu.coef_rate(levels, reqs).tobytes() == want.tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("call", ("rdoq", "rate"))
def test_large_workspace_is_kept_between_calls(gpu, oracle, call):
    # a workspace of 384 MB (a word per coefficient, of which only a few blocks are named) stays with the
    # library when the device is waited for: given back, it would be mapped anew by every call of a frame loop
    import torch
    n = 96 << 20
    data = torch.zeros(n, dtype=torch.int16, device="cuda")
    if call == "rdoq":
        reqs, ests, coefs = cases.rdoq_inputs(oracle, dict(n=9, k=2), 77)
        d = [torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).copy()).cuda() for a in (reqs, ests)]
        out = torch.zeros(len(reqs), dtype=torch.int32, device="cuda")
    else:
        coefs, reqs = cases.coef_rate_inputs(np.random.default_rng(77), 9)
        d = [torch.from_numpy(np.ascontiguousarray(reqs).view(np.uint8).copy()).cuda()]
        out = torch.zeros(len(reqs) * gpu.COEF_RATE_OUT.itemsize, dtype=torch.uint8, device="cuda")
    data[:coefs.size] = torch.from_numpy(coefs).cuda()
    torch.cuda.synchronize()
    if call == "rdoq":
        gpu.rdoq_device(d[0].data_ptr(), len(reqs), d[1].data_ptr(), len(ests), data.data_ptr(), n, out.data_ptr())
    else:
        gpu.coef_rate_device(d[0].data_ptr(), len(reqs), data.data_ptr(), n, out.data_ptr())
    held = torch.cuda.mem_get_info()[0]
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] - held < 32 << 20
    if call == "rdoq":
        assert np.array_equal(out.cpu().numpy(), oracle.rdoq(reqs, ests, coefs.copy()))
    else:
        assert out.cpu().numpy().tobytes() == oracle.coef_rate(coefs, reqs).tobytes()
