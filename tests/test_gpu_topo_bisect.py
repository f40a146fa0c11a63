"""The device bisection of the segmented guess against the same bisection driven from the host with
single residual evaluations.

The first steps decide on residuals far from zero and must take the same branches, so c is equal bit
for bit; after 60 steps the interval is below 1e-15 m and c may move by the residual's rounding over the
ocean area, far below the 1e-9 m bar of the guess.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlat,nlon", [(2, 8), (10, 16), (64, 128), (300, 512), (512, 1024)])
def test_device_bisection_matches_host_bisection(nlat, nlon):
    import torch

    from slevolve_b200 import _lib
    from slevolve_b200.init_topo import _Grids

    rng = np.random.default_rng(nlat)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()   # noqa: E731
    topo = rng.normal(-2500.0, 2000.0, (nlat, nlon))
    I0 = np.where(rng.random((nlat, nlon)) < 0.2, 2000.0 * rng.random((nlat, nlon)), 0.0)
    gr = _Grids(dev(topo), dev(I0), dev(0.5 * I0), 920.0, 1000.0, 6.371e6, torch)
    S = dev(rng.normal(0.0, 20.0, (nlat, nlon)))

    def host(lo, hi, steps):
        for _ in range(steps):
            mid = 0.5 * (lo + hi)
            lo, hi = (mid, hi) if gr.residual(S, mid) > 0 else (lo, mid)
        return 0.5 * (lo + hi)

    def device(lo, hi, steps):
        out, L = C.c_double(), _lib.lib()
        scratch = torch.zeros(int(L.sle_topo_bisect_scratch_bytes()), dtype=torch.uint8, device="cuda")
        for _ in range(2):   # the second call finds the scratch as the first left it
            _lib.check(L.sle_topo_bisect(*[C.c_void_p(t.data_ptr()) for t in (gr.Tp, S)], lo, hi, steps,
                                         *[C.c_void_p(t.data_ptr()) for t in (gr.I0, gr.Ip, gr.gp_u8, gr.wrow)], nlat,
                                         nlon, gr.rhoi, gr.rhow, gr.Vp, C.c_void_p(scratch.data_ptr()), C.byref(out),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return out.value

    for steps in (1, 3, 4, 5, 13):
        assert device(-300.0, 260.0, steps) == host(-300.0, 260.0, steps)
    assert abs(gr.solve_c(S, 62.0, 160.0) - host(-98.0, 222.0, 60)) <= 1e-9
