"""QP counts and mode lists of the intra lattice against the oracle: the QPs of a tile run one after the
other, a job that a QP codes nothing of keeps the prediction's SSD, and a tile holds a bounded number of
jobs."""
import numpy as np
import pytest

from test_gpu_intra import oracle_lattice
from uavs3e_gb300.synth import intra_frame

pytestmark = pytest.mark.gpu

FIELDS = ("ssd", "coef_hash", "num_nz", "last_nz", "sum_abs")


def _frames(W, H, seed, noise):
    org = intra_frame(W, H, seed=seed)
    rng = np.random.default_rng(seed)
    rec = np.clip(org.astype(int) + rng.integers(-noise, noise + 1, org.shape), 0, 255).astype(np.uint8)
    return org, rec


@pytest.mark.parametrize("qps", [[37], [63, 0], [51, 22, 63], [30, 63, 4, 45]])
@pytest.mark.parametrize("ipf", [0, 1])
def test_lattice_qp_counts(gpu, oracle, qps, ipf):
    # unsorted QPs, from all jobs coded to none, one to four of them
    W, H = 128, 72
    org, rec = _frames(W, H, len(qps) + 10 * ipf, 4)
    cus = gpu.lattice_cus(W, H)
    satd, q = gpu.intra_lattice(org, rec, cus, qps, ipf=ipf)
    satd_o, q_o = oracle_lattice(oracle, org, rec, cus, ipf, qps)
    assert np.array_equal(satd, satd_o)
    for f in FIELDS:
        assert np.array_equal(q[f], q_o[f]), f


@pytest.mark.parametrize("n_modes,n_qp", [(1, 2), (4, 1), (17, 3), (20, 2), (32, 1)])
def test_lattice_mode_list_sizes(gpu, oracle, n_modes, n_qp):
    import torch
    W, H, qps = 128, 72, np.array([24, 41, 34][:n_qp], np.int32)
    org, rec = _frames(W, H, 40 + n_modes, 8)
    cus = gpu.lattice_cus(W, H)
    n = len(cus)
    satd_o, q_o = oracle_lattice(oracle, org, rec, cus, 1, list(qps))
    rng = np.random.default_rng(n_modes)
    modes = np.stack([rng.permutation(33)[:n_modes] for _ in range(n)]).astype(np.uint8)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (org, rec, cus.view(np.uint8), modes)]
    d_satd = torch.zeros(n * 33, dtype=torch.int32, device="cuda")
    d_q = torch.zeros(n * 33 * n_qp * gpu.LAT_Q.itemsize, dtype=torch.uint8, device="cuda")
    gpu.check(gpu.lib().uavs3e_cuda_intra_lattice_modes_device(
        d[0].data_ptr(), W, d[1].data_ptr(), W, W, H, d[2].data_ptr(), n, d[3].data_ptr(), n_modes, 1, qps.ctypes.data,
        n_qp, 1, d_satd.data_ptr(), d_q.data_ptr(), torch.cuda.current_stream().cuda_stream), "intra_lattice")
    torch.cuda.synchronize()
    at = (np.arange(n)[:, None] * 33 + modes).ravel()
    assert np.array_equal(d_satd.cpu().numpy().view(np.uint32)[at], satd_o.ravel()[at])
    got, want = d_q.cpu().numpy().view(gpu.LAT_Q).reshape(n * 33, n_qp)[at], q_o.reshape(n * 33, n_qp)[at]
    for f in FIELDS:
        assert np.array_equal(got[f], want[f]), f


@pytest.mark.parametrize("n_modes", [33, 20, 5])
def test_lattice_satd_only(gpu, oracle, n_modes):
    # no QP: the tiles hold predictions alone, so more CUs or modes of one
    import torch
    W, H = 136, 72
    org, rec = _frames(W, H, 60 + n_modes, 6)
    cus = gpu.lattice_cus(W, H)
    n = len(cus)
    satd_o, _ = oracle_lattice(oracle, org, rec, cus, 0, [32])
    rng = np.random.default_rng(n_modes)
    modes = np.stack([rng.permutation(33)[:n_modes] if n_modes < 33 else np.arange(33) for _ in range(n)]).astype(np.uint8)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (org, rec, cus.view(np.uint8), modes)]
    d_satd = torch.full((n * 33,), -1, dtype=torch.int32, device="cuda")
    gpu.check(gpu.lib().uavs3e_cuda_intra_lattice_modes_device(
        d[0].data_ptr(), W, d[1].data_ptr(), W, W, H, d[2].data_ptr(), n, d[3].data_ptr() if n_modes < 33 else None,
        n_modes, 0, None, 0, 1, d_satd.data_ptr(), None, torch.cuda.current_stream().cuda_stream), "intra_lattice")
    torch.cuda.synchronize()
    want = np.full(n * 33, 0xFFFFFFFF, np.uint32)
    at = (np.arange(n)[:, None] * 33 + modes).ravel()
    want[at] = satd_o.ravel()[at]
    assert np.array_equal(d_satd.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("n_qp", [0, 1, 3])
def test_lattice_list_entries_that_are_no_modes(gpu, oracle, n_qp):
    # empty slots (255) and IPCM (33) of candidate lists write no record: every record of a listed mode is
    # right, every other word of the buffers, and the words behind them, keep what they held
    import torch
    W, H, n_modes, guard, qps = 72, 64, 5, 2048, np.array([24, 41, 34][:n_qp], np.int32)
    org, rec = _frames(W, H, 90 + n_qp, 6)
    cus = gpu.lattice_cus(W, H)
    n = len(cus)
    satd_o, q_o = oracle_lattice(oracle, org, rec, cus, 1, list(qps) if n_qp else [32])
    rng = np.random.default_rng(90 + n_qp)
    modes = np.stack([rng.permutation(33)[:n_modes] for _ in range(n)]).astype(np.uint8)
    drop = rng.random(modes.shape) < 0.3
    drop[-1], drop[-2] = True, [True, False, True, True, False]        # the last CU has no mode at all
    modes[drop] = rng.choice(np.array([33, 34, 128, 255], np.uint8), int(drop.sum()))
    modes[-1, :2] = 255, 33
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (org, rec, cus.view(np.uint8), modes)]
    words = gpu.LAT_Q.itemsize // 4
    d_satd = torch.full((n * 33 + guard,), -7, dtype=torch.int32, device="cuda")
    d_q = torch.full(((n * 33 * n_qp + guard) * words,), -7, dtype=torch.int32, device="cuda")
    gpu.check(gpu.lib().uavs3e_cuda_intra_lattice_modes_device(
        d[0].data_ptr(), W, d[1].data_ptr(), W, W, H, d[2].data_ptr(), n, d[3].data_ptr(), n_modes, 1,
        qps.ctypes.data if n_qp else None, n_qp, 1, d_satd.data_ptr(), d_q.data_ptr() if n_qp else None,
        torch.cuda.current_stream().cuda_stream), "intra_lattice")
    torch.cuda.synchronize()
    cu, slot = np.nonzero(~drop)
    at = cu * 33 + modes[cu, slot]
    want = np.full(n * 33 + guard, -7, np.int32)
    want[at] = satd_o.ravel().astype(np.uint32).view(np.int32)[at]
    assert np.array_equal(d_satd.cpu().numpy(), want)
    if n_qp:
        want_q = np.full((n * 33 + guard, n_qp * words), -7, np.int32)[:n * 33]
        got = d_q.cpu().numpy()
        assert (got[n * 33 * n_qp * words:] == -7).all()
        got = got[:n * 33 * n_qp * words].reshape(n * 33, n_qp * words)
        keep = np.zeros(n * 33, bool)
        keep[at] = True
        assert np.array_equal(got[~keep], want_q[~keep])
        rec_g, rec_o = np.ascontiguousarray(got[keep]).view(gpu.LAT_Q), q_o.reshape(n * 33, n_qp)[keep]
        for f in FIELDS:
            assert np.array_equal(rec_g[f], rec_o[f]), f


@pytest.mark.parametrize("n_modes,first", [(29, 1), (30, 2)])
def test_lattice_layouts_are_tuned_per_kind(gpu, n_modes, first):
    # calls of one QP and of several have different tile layouts: each kind tunes with its own first call
    # (told by the launches it takes: 4 of a tuned call), and a captured call tunes nothing
    import torch
    W, H = 136, 104
    org, rec = _frames(W, H, n_modes, 5)
    cus = gpu.lattice_cus(W, H)
    n = len(cus)
    modes = np.stack([np.random.default_rng(k).permutation(33)[:n_modes] for k in range(n)]).astype(np.uint8)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (org, rec, cus.view(np.uint8), modes)]
    stream = torch.cuda.Stream()

    def buffers():
        return (torch.zeros(n * 33, dtype=torch.int32, device="cuda"),
                torch.zeros(n * 33 * 2 * gpu.LAT_Q.itemsize, dtype=torch.uint8, device="cuda"))

    def call(n_qp, out):
        before = gpu.lib().uavs3e_cuda_launch_count()
        qps = np.array([27, 36][:n_qp], np.int32)
        gpu.check(gpu.lib().uavs3e_cuda_intra_lattice_modes_device(
            d[0].data_ptr(), W, d[1].data_ptr(), W, W, H, d[2].data_ptr(), n, d[3].data_ptr(), n_modes, 1, qps.ctypes.data,
            n_qp, 1, out[0].data_ptr(), out[1].data_ptr(), stream.cuda_stream), "intra_lattice")
        return gpu.lib().uavs3e_cuda_launch_count() - before

    second = 3 - first
    plain, cap = {k: buffers() for k in (1, 2)}, buffers()
    torch.cuda.synchronize()
    assert call(first, plain[first]) > 4 and call(first, plain[first]) == 4
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=stream):
        assert call(second, cap) == 4
    g.replay()
    torch.cuda.synchronize()
    assert call(second, plain[second]) > 4 and call(second, plain[second]) == 4
    assert call(first, plain[first]) == 4
    torch.cuda.synchronize()
    assert any(gpu.lattice_budgets(n_modes))
    assert torch.equal(cap[0], plain[second][0]) and torch.equal(cap[1], plain[second][1])


@pytest.mark.parametrize("W,H", [(16, 8), (256, 128), (256, 136)])
def test_lattice_satd_only_call_sizes(gpu, oracle, W, H):
    # the tile layout of a SATD-only call follows from its size: the smallest, and both sides of the line
    # (on 152 SMs)
    import torch
    org, rec = _frames(W, H, W + H, 6)
    cus = gpu.lattice_cus(W, H)
    n = len(cus)
    satd_o, _ = oracle_lattice(oracle, org, rec, cus, 1, [32])
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (org, rec, cus.view(np.uint8))]
    d_satd = torch.full((n * 33,), -1, dtype=torch.int32, device="cuda")
    gpu.check(gpu.lib().uavs3e_cuda_intra_lattice_device(
        d[0].data_ptr(), W, d[1].data_ptr(), W, W, H, d[2].data_ptr(), n, 1, None, 0, 1, d_satd.data_ptr(), None,
        torch.cuda.current_stream().cuda_stream), "intra_lattice")
    torch.cuda.synchronize()
    assert np.array_equal(d_satd.cpu().numpy().view(np.uint32), satd_o.ravel())


@pytest.mark.parametrize("n_modes,W,H", [(1, 64, 64), (2, 136, 72), (3, 128, 128), (33, 64, 32)])
def test_lattice_four_qps_of_few_jobs(gpu, oracle, n_modes, W, H):
    # the lists of the jobs that each QP codes, from none of them to all, in tiles of few and of many jobs
    import torch
    qps = np.array([63, 37, 0, 51], np.int32)
    org, rec = _frames(W, H, 70 + n_modes, 7)
    cus = gpu.lattice_cus(W, H)
    n = len(cus)
    satd_o, q_o = oracle_lattice(oracle, org, rec, cus, 0, list(qps))
    modes = np.stack([np.random.default_rng(k).permutation(33)[:n_modes] for k in range(n)]).astype(np.uint8)
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (org, rec, cus.view(np.uint8), modes)]
    d_satd = torch.zeros(n * 33, dtype=torch.int32, device="cuda")
    d_q = torch.zeros(n * 33 * 4 * gpu.LAT_Q.itemsize, dtype=torch.uint8, device="cuda")
    gpu.check(gpu.lib().uavs3e_cuda_intra_lattice_modes_device(
        d[0].data_ptr(), W, d[1].data_ptr(), W, W, H, d[2].data_ptr(), n, d[3].data_ptr(), n_modes, 0, qps.ctypes.data,
        4, 1, d_satd.data_ptr(), d_q.data_ptr(), torch.cuda.current_stream().cuda_stream), "intra_lattice")
    torch.cuda.synchronize()
    at = (np.arange(n)[:, None] * 33 + modes).ravel()
    assert np.array_equal(d_satd.cpu().numpy().view(np.uint32)[at], satd_o.ravel()[at])
    got, want = d_q.cpu().numpy().view(gpu.LAT_Q).reshape(n * 33, 4)[at], q_o.reshape(n * 33, 4)[at]
    for f in FIELDS:
        assert np.array_equal(got[f], want[f]), f


@pytest.mark.parametrize("n_qp,jobs_per_cta,extra", [(4, 2, -1), (4, 2, 1), (1, 2, -1), (0, 6, -1), (0, 6, 1)])
def test_lattice_of_few_cus(gpu, oracle, n_qp, jobs_per_cta, extra):
    # CUs of any shape in lists on both sides of the lengths where the tile layouts change (four CTAs an SM)
    import torch
    W, H, qps = 192, 128, np.array([27, 45, 33, 38][:n_qp], np.int32)
    n = jobs_per_cta * 4 * torch.cuda.get_device_properties(0).multi_processor_count // 33 + extra
    org, rec = _frames(W, H, 50 + n_qp, 6)
    cus = gpu.lattice_cus(W, H)
    big = cus[(cus["w"].astype(int) * cus["h"] >= 1024)]
    rng = np.random.default_rng(n)
    cus = np.concatenate([big[rng.permutation(len(big))[:n // 3]], cus[rng.permutation(len(cus))[:n - n // 3]]])
    satd_o, q_o = oracle_lattice(oracle, org, rec, cus, 1, list(qps) if n_qp else [32])
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (org, rec, cus.view(np.uint8))]
    d_satd = torch.zeros(n * 33, dtype=torch.int32, device="cuda")
    d_q = torch.zeros(max(1, n * 33 * n_qp * gpu.LAT_Q.itemsize), dtype=torch.uint8, device="cuda")
    gpu.check(gpu.lib().uavs3e_cuda_intra_lattice_device(
        d[0].data_ptr(), W, d[1].data_ptr(), W, W, H, d[2].data_ptr(), n, 1, qps.ctypes.data if n_qp else None, n_qp, 1,
        d_satd.data_ptr(), d_q.data_ptr() if n_qp else None, torch.cuda.current_stream().cuda_stream), "intra_lattice")
    torch.cuda.synchronize()
    assert np.array_equal(d_satd.cpu().numpy().view(np.uint32), satd_o.ravel())
    if n_qp:
        got = d_q.cpu().numpy().view(gpu.LAT_Q).ravel()
        for f in FIELDS:
            assert np.array_equal(got[f], q_o.ravel()[f]), f
