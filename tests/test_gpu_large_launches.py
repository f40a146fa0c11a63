"""Forms that only large launches take: spectral passes in runs of four blocks' worth of coefficients (from
8192 runs of 256 coefficients over all slots on), the analysis contraction with more landing than work
slots (more than two work units per CTA), and the Nyquist order of the mixed unfold.

A member's or field's result must not depend on what else is in the launch: bit for bit the one of a
small launch, which takes the other form of the passes.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# runs per slot: 9 with 32 coefficients in the last at L = 63 (B18 into the spectrum), 513 at L = 511
# (mixed: B18 into the B operand); in both the last block of four holds a single run
@pytest.mark.parametrize("nlat,nlon,L,members,precision", [(64, 128, 63, 911, "fp64"), (512, 1024, 511, 16, "mixed")])
def test_members_of_a_large_batch_equal_those_of_a_small_one(nlat, nlon, L, members, precision):
    import torch

    from slevolve_b200 import SyntheticEarth
    from slevolve_b200.batch import SolverBatch

    runs = -(-((L + 1) * (L + 2) // 2) // 256)
    assert runs * members >= 8192 > runs * 3 and runs % 4 == 1
    love = SyntheticEarth(L, 4, 7)
    j, i = np.meshgrid(np.arange(nlat), np.arange(nlon), indexing="ij")
    wave = 64.0 / nlat
    topo = np.round((1500.0 * np.sin(0.05 * wave * i + 0.4) * np.cos(0.07 * wave * j) - 1800.0) * 1000.0) / 1000.0
    topo[-nlat // 8:] = -400.0   # a marine cap, whose margin the step ungrounds
    shape = np.where(j >= nlat - nlat // 8, 1.0, 0.0)

    def ice(b, k):
        return torch.tensor(np.round(shape * (450.0 + (b % 7) - 40.0 * k) * 1000.0) / 1000.0, device="cuda")

    def run(slots):
        bt = SolverBatch(nlat, nlon, L, len(slots), max_modes=4, precision=precision)
        for s, b in enumerate(slots):
            bt.load(s, love, topo, ice(b, 0), 10.0)
        for k in (1, 2):
            infos = bt.step({s: ice(b, k) for s, b in enumerate(slots)})
        return {b: (infos[s]["numiter"], infos[s]["xi"], infos[s]["gr_reguess"], bt.get(s, "tgrid").copy(),
                    bt.get(s, "deltasl").copy()) for s, b in enumerate(slots)}

    keep = [0, 3, members - 1]
    big, small = run(list(range(members))), run(keep)
    assert any(v[2] > 0 for v in small.values())
    for b in keep:
        assert big[b][:3] == small[b][:3]
        assert np.array_equal(big[b][3], small[b][3]) and np.array_equal(big[b][4], small[b][4])


@pytest.mark.parametrize("nf", [8, 9, 31, 33])
def test_many_fields_equal_single_fields_with_many_units_per_cta(nf):
    import torch

    from slevolve_b200 import _lib, make_sht

    s = make_sht("cuda", 512, 1024, 511, precision="mixed")
    gen = torch.Generator(device="cuda").manual_seed(nf)
    g = [torch.randn((512, 1024), dtype=torch.float64, device="cuda", generator=gen) + 3.0 for _ in range(nf)]
    c = [torch.full((s.ncoef,), float("nan"), dtype=torch.complex128, device="cuda") for _ in g]
    back = [torch.full_like(x, float("nan")) for x in g]
    s.analysis_device(g, c, layout=_lib.LAYOUT_PACKED)
    s.synthesis_device(c, back, layout=_lib.LAYOUT_PACKED)
    one, gone = torch.empty_like(c[0]), torch.empty_like(g[0])
    for f in range(nf):
        s.analysis_device([g[f]], [one], layout=_lib.LAYOUT_PACKED)
        assert torch.equal(torch.view_as_real(one), torch.view_as_real(c[f])), f
        s.synthesis_device([one], [gone], layout=_lib.LAYOUT_PACKED)
        assert torch.equal(gone, back[f]), f


@pytest.mark.parametrize("nlat,nlon", [(64, 128), (128, 256)])
def test_mixed_transforms_with_the_nyquist_order(nlat, nlon):
    """lmax = nlon / 2: the mixed transforms against the FP64 ones, at the bar of their other tests."""
    from slevolve_b200 import make_sht

    L = nlon // 2
    f64, mx = make_sht("cuda", nlat, nlon, L), make_sht("cuda", nlat, nlon, L, precision="mixed")
    rng = np.random.default_rng(nlat)
    c = np.tril(rng.standard_normal((L + 1, L + 1)) + 1j * rng.standard_normal((L + 1, L + 1)))
    c[:, 0] = c[:, 0].real
    want, got = f64.synthesis(c).copy(), mx.synthesis(c).copy()
    assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()
    g = rng.standard_normal((nlat, nlon))
    want, got = f64.analysis(g).copy(), mx.analysis(g).copy()
    assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()
