"""Contents of a saved image: every library that reads this image version finds the topography of the
last step at the place of the previous topography (the second grid section, after the initial
topography), whatever the step itself keeps."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [0, 1, 4])
def test_image_holds_the_last_topography_as_the_previous_one(steps):
    from oracle.sht import OracleSHT
    from slevolve_b200.batch import SolverBatch
    from slevolve_b200.synthetic import case_c0

    case = case_c0(OracleSHT(64, 128, 63), nsteps=6)
    bt = SolverBatch(64, 128, 63, 2, precision="mixed")
    bt.load(1, case.love, case.topo, case.ice(0), 1.0)
    for k in range(1, steps + 1):
        bt.step({1: case.ice(k)})
    topo = np.ascontiguousarray(case.topo, dtype=np.float64)
    img = bt.snapshot(1).tobytes()
    first = img.find(topo.tobytes())   # the first section: the initial topography
    assert first > 0
    prev = np.frombuffer(img, np.float64, topo.size, first + topo.nbytes).reshape(topo.shape)
    assert np.array_equal(prev, bt.get(1, "tgrid"))
    assert np.array_equal(prev, topo) == (steps == 0)
