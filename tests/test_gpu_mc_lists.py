"""CU motion compensation of lists around the length from which small CUs are grouped, mixed and sorted by
size, at aligned and unaligned output offsets, against the oracle."""
import numpy as np
import pytest

from test_gpu_mc import _gpu_affine, _gpu_mc, cases

pytestmark = pytest.mark.gpu

LONG = 4 * 64 * 152


@pytest.mark.parametrize("n,sort,shift", [(LONG - 1, True, 0), (LONG, False, 1), (LONG + 2, True, 0), (3, True, 2), (1, False, 3)])
def test_mc_list_lengths(gpu, oracle, n, sort, shift):
    p = cases.MC_CASES[0]
    luma, chroma, reqs, nbytes = cases.mc_inputs(oracle, dict(p, n=n), 77)
    reqs["out_offset"] += shift
    nbytes += shift
    if sort:
        reqs = reqs[np.argsort(reqs["w"].astype(int) * reqs["h"], kind="stable")]
    want = oracle.mc_cu(p["w"], p["h"], luma[1], luma[2], chroma[1], chroma[2], reqs, nbytes)
    assert np.array_equal(want, _gpu_mc(gpu, p, luma, chroma, reqs, nbytes))


@pytest.mark.parametrize("channel", [0, 1])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_mc_unaligned_luma(gpu, oracle, shift, channel):
    # every size with its luma off the 4-byte grid, one and two lists
    p = cases.MC_CASES[0]
    luma, chroma, reqs, _ = cases.mc_inputs(oracle, dict(p, n=400), 80 + shift)
    reqs["channel"] = channel
    size = reqs["w"].astype(int) * reqs["h"] * (2 if channel else 3) // 2
    reqs["out_offset"] = np.cumsum(size) - size + shift
    nbytes = int(size.sum()) + shift
    assert len({(r["w"], r["h"]) for r in reqs}) >= 10 and (reqs["slot"] >= 0).all(1).any()
    want = oracle.mc_cu(p["w"], p["h"], luma[1], luma[2], chroma[1], chroma[2], reqs, nbytes)
    assert np.array_equal(want, _gpu_mc(gpu, p, luma, chroma, reqs, nbytes))


@pytest.mark.parametrize("shift", [0, 1, 2])
def test_affine_output_alignment(gpu, oracle, shift):
    p = cases.MC_CASES[0]
    luma, chroma, _, _ = cases.mc_inputs(oracle, dict(p, n=1), 78)
    reqs, nbytes = cases.affine_requests(np.random.default_rng(78), p["w"], p["h"], 200)
    reqs["out_offset"] += shift
    nbytes += shift
    want = oracle.mc_affine(p["w"], p["h"], luma[1], luma[2], chroma[1], chroma[2], reqs, nbytes)
    assert np.array_equal(want, _gpu_affine(gpu, p, luma, chroma, reqs, nbytes))


@pytest.mark.parametrize("extra,big_at", [(-1, ()), (0, ()), (0, (0, 31, 32, 95, 1000)), (33, (70,)), (7, "last")])
def test_mc_small_cus_in_long_lists(gpu, oracle, extra, big_at):
    # CUs of at most 256 samples, grouped by 32 from the device's list length on: lists one short of it, at
    # it and not a multiple of 32 past it, groups broken by one larger CU or by a request that is skipped
    import torch
    p = cases.MC_CASES[0]
    n = 256 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    luma, chroma, reqs, _ = cases.mc_inputs(oracle, dict(p, n=6000), 79)
    area = reqs["w"].astype(int) * reqs["h"]
    small, big = reqs[(area <= 256) & (area > 0)], reqs[area > 256]
    reqs = small[np.random.default_rng(n).integers(0, len(small), n)].copy()
    for k in (n - 1,) if big_at == "last" else big_at:
        reqs[k] = big[k % len(big)]
    size = np.where(reqs["channel"] == 0, 3, np.where(reqs["channel"] == 1, 2, 1)) * reqs["w"].astype(int) * reqs["h"] // 2
    reqs["out_offset"] = np.cumsum(size) - size
    nbytes = int(size.sum())
    keep = np.ones(n, bool)
    if big_at:
        reqs["x"][200], keep[200] = -8, False            # outside the domain: nothing written
    want = oracle.mc_cu(p["w"], p["h"], luma[1], luma[2], chroma[1], chroma[2], reqs[keep], nbytes)
    assert np.array_equal(want, _gpu_mc(gpu, p, luma, chroma, reqs, nbytes))
