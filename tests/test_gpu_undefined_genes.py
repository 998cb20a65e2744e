"""Individuals with an undefined or infinite gene: their fitness says so whichever kernels a set takes, as the direct
evaluation of every pair does, and every other individual keeps its bits."""
import numpy as np
import pytest

from gpuga_b200 import Fitness, synth
from tests.test_gpu_pair_expansion import _set
from tests.test_gpu_tersoff_pairs import _cells, _targets

pytestmark = pytest.mark.gpu


def _fitness(data, kw, P, gene, value):
    pop = synth.population(data, P, seed=4)
    odd = pop.copy()
    odd[3, gene] = value
    with Fitness(arrays=data, **kw) as e:
        fit, got = np.asarray(e.compute(P, pop)), np.asarray(e.compute(P, odd))
    rest = np.arange(P) != 3
    assert np.array_equal(fit[rest], got[rest])
    return got[3]


def test_infinite_dispersion():
    """C01 = inf, finite elsewhere: an infinite energy error, not an undefined one."""
    data, kw = _set("ri", [64] * 8, 4)
    assert _fitness(data, kw, 40, 6, np.inf) == np.inf
    assert np.isnan(_fitness(data, kw, 40, 6, np.nan))
    assert np.isnan(_fitness(data, kw, 40, 0, np.nan))


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("nf,nc", [(4, 6), (1, 8)])
def test_fixed_inner_radius(nf, nc, value):
    """R1 is fixed by its bounds and belongs to the geometry of the packed force and pair-by-pair items."""
    data = _targets(dict(_cells([64] * nc), Nc_force=nf))
    for gene in (6, 7):
        assert np.isnan(_fitness(data, {}, 40, gene, value)), gene
