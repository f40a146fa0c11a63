"""The ocean-function refresh with several chunks of cells per block (large batches) against the same
members in small batches (one chunk per block): the last chunk of a grid partly filled, blocks with and
without ice, every slot's result bit for bit the one it gets in a small batch."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlat,nlon,L,members", [(64, 128, 63, 520), (330, 512, 40, 64)])
def test_chunked_refresh_equals_single_chunks(nlat, nlon, L, members):
    import torch

    from slevolve_b200 import SyntheticEarth
    from slevolve_b200.batch import SolverBatch

    love = SyntheticEarth(L, 4, 7)
    j, i = np.meshgrid(np.arange(nlat), np.arange(nlon), indexing="ij")
    topo = np.round((1500.0 * np.sin(0.05 * i + 0.4) * np.cos(0.07 * j) - 1800.0) * 1000.0) / 1000.0
    topo[-nlat // 8:] = -400.0   # a marine cap, whose margin the step ungrounds
    shape = np.where(j >= nlat - nlat // 8, 1.0, 0.0)

    def ice(b, k):
        return torch.tensor(np.round(shape * (450.0 + (b % 7) - 40.0 * k) * 1000.0) / 1000.0, device="cuda")

    def run(slots):
        bt = SolverBatch(nlat, nlon, L, len(slots), max_modes=4, precision="fp64")
        for s, b in enumerate(slots):
            bt.load(s, love, topo, ice(b, 0), 10.0)
        out = {}
        for k in (1, 2):
            infos = bt.step({s: ice(b, k) for s, b in enumerate(slots)})
        for s, b in enumerate(slots):
            out[b] = (infos[s]["numiter"], infos[s]["gr_reguess"], bt.get(s, "tgrid"), bt.get(s, "beta"))
        return out

    big, small = run(list(range(members))), run([0, 3, members - 1])
    assert any(v[1] > 0 for v in small.values())
    for b, v in small.items():
        assert big[b][:2] == v[:2]
        assert np.array_equal(big[b][2], v[2]) and np.array_equal(big[b][3], v[3])
