"""Mixed-precision launches at the edges of their field blocks: 1, 8, 9, 16, 17, 31, 32 and 33 fields
(eight fields per column block, 32 per launch), a grid of one 64-latitude chunk pair and one of
several, the largest degree and a truncated one.

A field's result must not depend on the fields beside it (bit for bit, the launch's own contract), and
its degree-0 coefficient is formed in FP64: within 1e-13 of the FP64 transform's.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nlon,L", [(64, 128, 63), (192, 512, 170), (256, 512, 255)])
def test_fields_of_a_launch_are_independent(n, nlon, L):
    import torch

    from slevolve_b200 import _lib, make_sht

    s, s64 = make_sht("cuda", n, nlon, L, precision="mixed"), make_sht("cuda", n, nlon, L)
    gen = torch.Generator(device="cuda").manual_seed(n)
    g = [torch.randn((n, nlon), dtype=torch.float64, device="cuda", generator=gen) + 3.0 for _ in range(33)]
    one_c = [torch.empty(s.ncoef, dtype=torch.complex128, device="cuda") for _ in g]
    one_g = [torch.empty_like(x) for x in g]
    for f in range(33):
        s.analysis_device([g[f]], [one_c[f]], layout=_lib.LAYOUT_PACKED)
        s.synthesis_device([one_c[f]], [one_g[f]], layout=_lib.LAYOUT_PACKED)
    ref = torch.empty_like(one_c[0])
    s64.analysis_device([g[0]], [ref], layout=_lib.LAYOUT_PACKED)
    assert abs(one_c[0][0].item() - ref[0].item()) <= 1e-13 * abs(ref[0].item())
    for nf in (8, 9, 16, 17, 31, 32, 33):
        c = [torch.full_like(x, float("nan")) for x in one_c[:nf]]
        back = [torch.full_like(x, float("nan")) for x in g[:nf]]
        s.analysis_device(g[:nf], c, layout=_lib.LAYOUT_PACKED)
        s.synthesis_device(c, back, layout=_lib.LAYOUT_PACKED)
        for f in range(nf):
            assert torch.equal(torch.view_as_real(c[f]), torch.view_as_real(one_c[f])), (nf, f)
            assert torch.equal(back[f], one_g[f]), (nf, f)
