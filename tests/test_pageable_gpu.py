"""gmle_fit on pageable buffers over several chunks (64 MiB of pixels each; two
full ones and a remainder): inputs and outputs that the copy engine reads and
writes in the caller's memory, the same bits as the device-resident fit."""
import numpy as np
import pytest

import gaussmle_gb300 as G
from gaussmle_gb300.fitter import make_desc
from parity_cases import make_case
from test_edge_gpu import host_fit

pytestmark = pytest.mark.gpu


def test_several_pageable_chunks_equal_the_device_fit(ctx):
    torch = pytest.importorskip("torch")
    w = make_case("xynb-7-poisson", 0, 7, 0, 1000, seed=3)
    n = 2 * ((64 << 20) // (4 * 49)) + 1001
    rois = np.ascontiguousarray(w.data.transpose(2, 1, 0)).reshape(1000, -1)
    data = np.resize(rois, (n, 49))  # the 1000 ROIs over and over
    desc = make_desc(w.psf, 7, 20, w.constraints, 0)
    st, got = host_fit(ctx, desc, data.reshape(n, 7, 7).transpose(2, 1, 0))
    ctx.check(st)
    dev = torch.device("cuda", 0)
    out = [torch.empty((n, 4), device=dev), torch.empty((n, 4), device=dev),
           torch.empty(n, device=dev), torch.empty(n, dtype=torch.uint8, device=dev)]
    G.fit_device(ctx, desc, torch.from_numpy(data).to(dev), None, None, *out)
    torch.cuda.synchronize()
    for a, b in zip(got, out):
        assert np.array_equal(a, b.cpu().numpy())
