"""The tiled kernels at the edges of their tiles and on both sides of their dispatch rules, bit for bit against a
kernel of this library that knows no tiles."""
import numpy as np
import pytest

from _gpu import bits, cuda_moe
from apus_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [33, 513, 2100])
def test_grouping_of_many_routings(T):
    """n = T * topk routings: a few per warp, several steps per warp, more than 4,096 in all."""
    W = synth.MoeWeights(seed=5, E=9, topk=2)
    x = synth.activations(np.random.default_rng(T), T, W.dim)
    whole = cuda_moe(W, x)
    for lo in (0, T // 2, T - 7):
        part = cuda_moe(W, x[lo:lo + 7])
        assert np.array_equal(whole["idx"][lo:lo + 7], part["idx"])
        assert np.array_equal(bits(whole["out"][lo:lo + 7]), bits(part["out"]))
