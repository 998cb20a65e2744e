"""Packed Tersoff force items (csrc/tersoff_force.cu) against the FP64 path: configurations around the sizes where the
individuals per item change (32 to 2; one beyond shared memory stays on the items by atom), odd populations, atoms with
fewer than four bonds, bonds between R1 and R2, two elements, S fitted.

Tolerances: per-atom forces 2e-5 of scale, the batched path's bar; an individual gives the same bits alone, and whatever
tile option is asked for."""
import numpy as np
import pytest

from gpuga_b200 import Fitness, synth
from tests.test_gpu_tersoff_pairs import _cells, _targets

pytestmark = pytest.mark.gpu


def _check(data, pop):
    P = len(pop)
    with Fitness(arrays=data) as e:
        forces = e.batched_forces(pop)
        fit = e.compute(P, pop)
        _, _, F2 = e.config_results(P)
        one = np.array([e.compute(1, pop[p:p + 1])[0] for p in (0, P - 1)])
        Nf, N = e.N_force, e.N
        starts = np.concatenate([[0], np.cumsum(data["Na"])])
        for p in {0, P // 2, P - 1}:
            F, _, _ = e.find_force64(e.decode(pop[p]).astype(np.float64))
            F = F.reshape(3, N)[:, :Nf]
            scale = np.abs(F).max()
            assert np.abs(forces[p] - F).max() <= 2e-5 * scale
            d2 = ((F - data["force_ref"].reshape(3, N)[:, :Nf]) ** 2).sum(0)
            for c in range(data["Nc_force"]):
                a, b = starts[c], starts[c + 1]
                # |F - Fref| to 2e-5 of scale per component
                assert abs(np.sqrt(F2[p, c]) - np.sqrt(d2[a:b].sum())) <= 2e-5 * scale * np.sqrt(3 * (b - a))
    assert np.array_equal(one, fit[[0, P - 1]])
    with Fitness(arrays=data, tiles=3) as e:
        assert np.array_equal(e.compute(P, pop), fit)


@pytest.mark.parametrize("P", [1, 3, 31, 34])
@pytest.mark.parametrize("na", [[2, 7, 8, 63, 64, 65, 66], [128, 130, 260, 261], [512, 522, 1000], [64, 2197, 64]])
def test_sizes_and_populations(na, P):
    data = _cells(na + [64, 64])
    data["Nc_force"] = len(na)
    _check(_targets(data), synth.population(data, P, seed=P))


@pytest.mark.parametrize("sigma", [0.02, 0.25])
@pytest.mark.parametrize("cutoff", [3.0, 3.9])
def test_cutoff_shell(sigma, cutoff):
    """Most atoms with four bonds inside R1, or most without; a list that is longer than what lies inside R2."""
    data = _cells([64, 216, 60, 64, 64], sigma=sigma, cutoff=cutoff)
    data["Nc_force"] = 3
    with Fitness(arrays=data) as e0:
        if e0.max_neighbors > 16:
            pytest.skip("more neighbors than the batched path takes")
    _check(_targets(data), synth.population(data, 37, seed=2))


@pytest.mark.parametrize("S_free", [False, True])
def test_two_elements(S_free):
    data = synth.make(2, Nc=8, seed=21)
    data["potential_type"] = 2
    rng = np.random.default_rng(1)
    data["type"] = rng.integers(0, 2, len(data["type"])).astype(np.int32)
    lo = [2.7, 1.0, 2.2, 2, 2.8, 1.0, 2.2, 2, 0.5, 0.1, -1, 2.8, 3.2]
    hi = [3.3, 1.5, 2.4, 2, 3.3, 1.5, 2.4, 2, 1.5, 0.5, -0.5, 2.8, 3.2]
    data["pmin"], data["pmax"] = np.array(lo, np.float32), np.array(hi, np.float32)
    if S_free:
        data["pmin"][[3, 7]], data["pmax"][[3, 7]] = 1.5, 2.5
    data["teacher01"] = rng.uniform(0, 1, 13).astype(np.float32)
    _check(_targets(data), synth.population(data, 21, seed=4))


@pytest.mark.parametrize("P", [1, 5])
def test_cta_sizes(P):
    """525 atoms are the last in a CTA of 128 threads; the two kinds of CTA in one set, and a set of the larger alone."""
    for na in ([525, 526, 64], [526, 800]):
        data = _cells(na + [64, 64])
        data["Nc_force"] = len(na)
        _check(_targets(data), synth.population(data, P, seed=10 + P))
