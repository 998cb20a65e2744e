"""Per-atom forces of a set with a pair expansion come from a launch set of their own, in which every pair is evaluated
directly: they, the fitness and the per-configuration results do not depend on what was called before, and the
expansion does not run beside it."""
import ctypes as C

import numpy as np
import pytest

from gpuga_b200 import Fitness, _lib, synth
from tests.test_gpu_pair_expansion import _set

pytestmark = pytest.mark.gpu


def _launch_ms(e, P):
    n = C.c_int()
    rows = np.zeros((8, 8))
    _lib.check(_lib.load().gpuga_plan_info(e.handle, P, C.byref(n), C.c_void_p(rows.ctypes.data), 8))
    return rows[:n.value]


@pytest.mark.parametrize("fold", [0, 1])
@pytest.mark.parametrize("kind", ["ri", "nn"])
def test_forces_among_generations(kind, fold):
    data, kw = _set(kind, [64, 62, 64, 30, 64, 64], 3)
    P = 35
    pop, other = synth.population(data, P, seed=2), synth.population(data, P, seed=3)
    with Fitness(arrays=data, fitness_fold=fold, **kw) as e:
        first = e.batched_forces(pop)
        after_forces = e.config_results(P)
        fit = e.compute(P, other)
        results = e.config_results(P)
        assert np.array_equal(e.batched_forces(pop), first)
        for a, b in zip(e.config_results(P), after_forces):
            assert np.array_equal(a, b)
        assert np.array_equal(e.compute(P, other), fit)
        for a, b in zip(e.config_results(P), results):
            assert np.array_equal(a, b)
        rows = _launch_ms(e, P)
        assert np.any(rows[:, 1] == 0)  # the generations use the expansion
        _lib.check(_lib.load().gpuga_kernel_timing(e.handle, P, 1))
        e.batched_forces(pop)
        assert not _launch_ms(e, P)[:, 7].any()  # its launches did not run
        _lib.check(_lib.load().gpuga_kernel_timing(e.handle, P, 0))
    with Fitness(arrays=data, fitness_fold=fold, **kw) as e:
        assert np.array_equal(e.compute(P, other), fit)
