"""GPU: the TZ search's wide row loads on plane strides that are a multiple of 4 but not of 8 (the
alignment of a candidate's rows alternates) and on org pictures of any alignment and pitch, bit-exact
against the oracle."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))
import cases  # noqa: E402


@pytest.mark.gpu
@pytest.mark.parametrize("extra,org_at", [(0, 0), (4, 0), (4, 1), (12, 3)])
def test_tz_plane_strides_and_org_alignment(gpu, oracle, extra, org_at):
    import torch
    p = dict(cases.TZ_CASES[0], n=300)
    pic, org, keep, addrs, stride, reqs = cases.tz_inputs(oracle, p, 77 + extra + org_at)
    want = oracle.me_tz(pic, org, p["w"], addrs, stride, reqs)
    s2 = stride + extra
    planes = []
    for a in keep:
        rows = a.reshape(-1, stride)
        planes.append(torch.from_numpy(np.pad(rows, ((0, 0), (0, extra)))).contiguous().cuda())
    i_org = p["w"] + org_at
    flat = np.zeros(org_at + p["h"] * i_org, np.uint8)
    flat[org_at:].reshape(p["h"], i_org)[:, :p["w"]] = org
    d_org = torch.from_numpy(flat).cuda()
    d_req = torch.from_numpy(np.ascontiguousarray(reqs).view(np.uint8).copy()).cuda()
    d_out = torch.zeros(len(reqs) * gpu.TZ_OUT.itemsize, dtype=torch.uint8, device="cuda")
    base = cases.TZ_PAD * s2 + cases.TZ_PAD
    gpu.me_tz_device(pic, d_org.data_ptr() + org_at, i_org, [t.data_ptr() + base for t in planes], s2, cases.TZ_PAD,
                     d_req.data_ptr(), len(reqs), d_out.data_ptr())
    torch.cuda.synchronize()
    assert d_out.cpu().numpy().tobytes() == np.ascontiguousarray(want).tobytes()
