"""The segmented guess with a transform of the caller's own: only its analysis and synthesis are used,
whatever else it calls its weights (another normalisation, a device tensor, plain ones, none)."""

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "init_topo.npz")


class Wrapped:
    def __init__(self, sht):
        self.analysis, self.synthesis = sht.analysis, sht.synthesis


@pytest.mark.parametrize("weights", ["none", "to one", "device", "equal"])
def test_guess_takes_only_the_transforms_of_a_foreign_object(weights):
    import torch

    from slevolve_b200 import make_sht
    from slevolve_b200.init_topo import segmented_guess
    from slevolve_b200.love import SyntheticEarth

    g = np.load(GOLD)
    own = make_sht("cuda", 64, 128, 63)
    sht = Wrapped(own)
    if weights != "none":
        sht.weights = {"to one": own.weights / 2, "device": torch.tensor(own.weights, device="cuda"),
                       "equal": np.ones(64)}[weights]
    T0, info = segmented_guess(g["topo"], list(g["ice"]), SyntheticEarth(63, 8, 20261203 + 5), 63, 10.0, sht=sht)
    # the bar of the guess against the reference's output
    assert info["iters"] == int(g["uniform_iters"])
    assert abs(info["c"] - float(g["uniform_c"])) <= 1e-9
    assert np.abs(T0 - g["uniform_T0"]).max() <= 1e-9
