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
