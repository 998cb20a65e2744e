"""The FP64 path of the network potential uploads the weights of the whole population before its kernels: the first evaluation
of a fresh engine is the same as the second."""
import numpy as np
import pytest

from gpuga_b200 import PATH_PLAIN64, Fitness, synth
from tests.test_gpu_pair_expansion import _set

pytestmark = pytest.mark.gpu


def test_first_evaluation():
    data, kw = _set("nn", [8, 3, 2, 8], 2, neurons=32)
    pop = synth.population(data, 64, seed=2)
    for _ in range(25):
        with Fitness(arrays=data, **kw) as e:
            first = e.compute(64, pop, path=PATH_PLAIN64)
            assert np.array_equal(e.compute(64, pop, path=PATH_PLAIN64), first)
