"""CU motion compensation of lists around the length from which a warp takes four CUs, mixed and sorted by
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


@pytest.mark.parametrize("shift", [0, 1, 2])
def test_affine_output_alignment(gpu, oracle, shift):
    p = cases.MC_CASES[0]
    luma, chroma, _, _ = cases.mc_inputs(oracle, dict(p, n=1), 78)
    reqs, nbytes = cases.affine_requests(np.random.default_rng(78), p["w"], p["h"], 200)
    reqs["out_offset"] += shift
    nbytes += shift
    want = oracle.mc_affine(p["w"], p["h"], luma[1], luma[2], chroma[1], chroma[2], reqs, nbytes)
    assert np.array_equal(want, _gpu_affine(gpu, p, luma, chroma, reqs, nbytes))
