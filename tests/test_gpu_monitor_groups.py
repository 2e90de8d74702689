"""dugks_cell_macros_noalloc where its groups of four DVs and blocks of cells
leave remainders, against plain torch FP64 sums.  Tolerance 1e-13: at most 70
positive terms, each sum off by at most 70 x 2^-53 = 8e-15 of itself, and a few
operations after it; U against the largest node."""
import ctypes as C

import numpy as np
import pytest

from dugks_b200 import lib as dl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [2, 3])
@pytest.mark.parametrize("nv", [1, 2, 3, 4, 5, 7, 9, 33, 70])
@pytest.mark.parametrize("n", [1, 33, 128, 257])
def test_group_remainders(D, nv, n):
    import torch
    lib = dl.load()
    gen = torch.Generator().manual_seed(100 * nv + n)
    dev = torch.device("cuda:0")
    xi = 400.0 * torch.randn(nv, 3, dtype=torch.float64, generator=gen)
    if D == 2:
        xi[:, 2] = 0.0
    w = torch.rand(nv, dtype=torch.float64, generator=gen) + 0.5
    g = torch.rand(nv, n, dtype=torch.float64, generator=gen) + 0.5
    h = 1e6 * (torch.rand(nv, n, dtype=torch.float64, generator=gen) + 0.5)
    rho = (w[:, None] * g).sum(0)
    U = torch.einsum("dc,dk->ck", w[:, None] * g, xi) / rho[:, None]
    gas = dl.Gas(208.0, 0.81, 273.0, 2.1e-5, 2.0 / 3.0, 0)
    x, ww, gg, hh = (a.to(dev).contiguous() for a in (xi, w, g, h))
    r = torch.full((n,), float("nan"), dtype=torch.float64, device=dev)
    u = torch.full((n, 3), float("nan"), dtype=torch.float64, device=dev)
    msg = C.create_string_buffer(256)
    st = lib.dugks_cell_macros_noalloc(D, nv, x.data_ptr(), ww.data_ptr(), n, gg.data_ptr(), hh.data_ptr(), C.byref(gas),
                                       1e-6, r.data_ptr(), u.data_ptr(), None, None,
                                       torch.cuda.current_stream(dev).cuda_stream, msg, len(msg))
    assert st == 0, msg.value.decode()
    torch.cuda.synchronize()
    assert np.abs(r.cpu().numpy() / rho.numpy() - 1).max() <= 1e-13
    assert np.abs(u.cpu().numpy() - U.numpy()).max() <= 1e-13 * max(1.0, float(xi.abs().max()))
