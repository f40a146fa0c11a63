"""The FP64 transform kernels at the edges of their tiles, against the CPU oracle: every number of
32-latitude groups a pass or block takes (one to eight, more than eight), latitudes and degrees that
fill neither a group nor a segment, the smallest grids, one to four fields, both layouts.

Tolerance: 1e-12 of the largest value, the bar of the transforms' other tests (sums of at most a few
thousand products, each rounded to 1.1e-16).  Fields taken in pairs, and the dense and the packed
layout, use the same arithmetic and must agree bit for bit.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REL = 1e-12

GRIDS = [(2, 8, 1), (4, 8, 0), (8, 16, 7), (64, 128, 63), (66, 128, 64), (100, 128, 50), (128, 256, 127), (192, 256, 100),
         (250, 256, 65), (300, 512, 143), (384, 512, 190), (446, 512, 129), (1090, 2048, 70)]


def _spectrum(rng, L):
    c = np.tril(rng.standard_normal((L + 1, L + 1)) + 1j * rng.standard_normal((L + 1, L + 1)))
    c[:, 0] = c[:, 0].real
    return c


@pytest.mark.parametrize("n,nlon,L", GRIDS)
def test_fp64_kernels_at_tile_edges(n, nlon, L):
    import torch

    from oracle.sht import OracleSHT
    from slevolve_b200 import _lib, make_sht

    rng = np.random.default_rng(100 * n + L)
    s, o = make_sht("cuda", n, nlon, L), OracleSHT(n, nlon, L)
    m, l = np.triu_indices(L + 1)
    grids = rng.standard_normal((3, n, nlon))
    specs = np.stack([_spectrum(rng, L) for _ in range(3)])
    gd = [torch.tensor(g, device="cuda") for g in grids]
    dense = [torch.full((L + 1, L + 1), float("nan"), dtype=torch.complex128, device="cuda") for _ in gd]
    packed = [torch.empty(s.ncoef, dtype=torch.complex128, device="cuda") for _ in gd]
    s.analysis_device(gd, dense)
    s.analysis_device(gd, packed, layout=_lib.LAYOUT_PACKED)
    for f in range(3):
        ref = o.analysis(grids[f])
        got = dense[f].cpu().numpy()
        assert np.abs(got - ref).max() <= REL * np.abs(ref).max()
        assert np.array_equal(got[l, m], packed[f].cpu().numpy())
    cd = [torch.tensor(c, device="cuda") for c in specs]
    cp = [torch.tensor(np.ascontiguousarray(c[l, m]), device="cuda") for c in specs]
    out, outp = [torch.empty_like(g) for g in gd], [torch.empty_like(g) for g in gd]
    s.synthesis_device(cd, out)
    s.synthesis_device(cp, outp, layout=_lib.LAYOUT_PACKED)
    for f in range(3):
        ref = o.synthesis(specs[f])
        assert np.abs(out[f].cpu().numpy() - ref).max() <= REL * np.abs(ref).max()
        assert torch.equal(out[f], outp[f])


@pytest.mark.parametrize("n,nlon,L", [(512, 1024, 511), (1024, 2048, 400)])
@pytest.mark.parametrize("nf", [2, 3, 4])
def test_paired_fields_equal_single_fields(n, nlon, L, nf):
    """Enough warps for the paired form (one recurrence for two fields): the same bits as alone."""
    import torch

    from slevolve_b200 import _lib, make_sht

    s = make_sht("cuda", n, nlon, L)
    gen = torch.Generator(device="cuda").manual_seed(n + nf)
    g = [torch.randn((n, nlon), dtype=torch.float64, device="cuda", generator=gen) for _ in range(nf)]
    c = [torch.empty(s.ncoef, dtype=torch.complex128, device="cuda") for _ in g]
    back = [torch.empty_like(x) for x in g]
    s.analysis_device(g, c, layout=_lib.LAYOUT_PACKED)
    s.synthesis_device(c, back, layout=_lib.LAYOUT_PACKED)
    one, gone = torch.empty_like(c[0]), torch.empty_like(g[0])
    for f in range(nf):
        s.analysis_device([g[f]], [one], layout=_lib.LAYOUT_PACKED)
        assert torch.equal(one, c[f])
        s.synthesis_device([one], [gone], layout=_lib.LAYOUT_PACKED)
        assert torch.equal(gone, back[f])


@pytest.mark.parametrize("n,nlon,L,nf", [(64, 128, 63, 33), (64, 128, 63, 32), (180, 512, 170, 21), (512, 1024, 511, 16)])
def test_long_lists_equal_single_fields(n, nlon, L, nf):
    """Lists of a whole launch, one field more, and beyond the plan's limit: the same bits as alone."""
    import torch

    from slevolve_b200 import _lib, make_sht

    s = make_sht("cuda", n, nlon, L)
    gen = torch.Generator(device="cuda").manual_seed(nf)
    g = [torch.randn((n, nlon), dtype=torch.float64, device="cuda", generator=gen) for _ in range(nf)]
    c = [torch.full((s.ncoef,), float("nan"), dtype=torch.complex128, device="cuda") for _ in g]
    back = [torch.full_like(x, float("nan")) for x in g]
    s.analysis_device(g, c, layout=_lib.LAYOUT_PACKED)
    s.synthesis_device(c, back, layout=_lib.LAYOUT_PACKED)
    one, gone = torch.empty_like(c[0]), torch.empty_like(g[0])
    for f in range(nf):
        s.analysis_device([g[f]], [one], layout=_lib.LAYOUT_PACKED)
        assert torch.equal(one, c[f]), f
        s.synthesis_device([one], [gone], layout=_lib.LAYOUT_PACKED)
        assert torch.equal(gone, back[f]), f
    with pytest.raises(ValueError):   # the dense layout's limit is unchanged
        s.analysis_device(g[:5], [torch.empty((L + 1, L + 1), dtype=torch.complex128, device="cuda") for _ in range(5)])
