"""Pair-by-pair energy/virial items of the Tersoff potential (csrc/tersoff_ev.cu) against the FP64 path, at the edges
of their blocking (segments of 240 pairs, batches of 2, groups of 32 individuals), with neighbors between R1 and R2, up
to 14 neighbors per atom, two elements with S fitted, and where the bond-order table does not reach: n too sharp for
its polynomials, h beyond its bounds, beta = 0.

Tolerances: per-configuration energies and virials 2e-6 of scale, the batched path's own bar; for n up to 12, where
b'(s) varies by its size within an eighth of an octave and s is rounded to FP32 (6e-8), ten times that."""
import numpy as np
import pytest

from gpuga_b200 import PATH_PLAIN64, Fitness, synth

pytestmark = pytest.mark.gpu


def _cells(na, sigma=0.1, a=5.43, frac=synth.DIAMOND, cutoff=3.0, seed=3):
    """Diamond (or `frac`) cells of which the first na[c] atoms are kept; the first configuration is a force one."""
    rng = np.random.default_rng(seed)
    configs = []
    for n in na:
        reps = 1
        while len(frac) * reps ** 3 < n or reps < 2:
            reps += 1
        f, cell = synth._structure(np.asarray(frac, float), np.eye(3) * a, (reps, reps, reps))
        pos, cell, t = synth._config(rng, f, cell, np.zeros(len(f)), 0.02, sigma)
        configs.append((pos[:n], cell, t[:n]))
    b = synth.SI_TERSOFF_BOUNDS
    spec = dict(potential_type=1, num_neurons=0, cutoff=cutoff, w_force=0.05, w_energy=0.15, w_stress=0.8,
                pmin=b[:, 0].copy(), pmax=b[:, 1].copy(), ga={})
    data = synth._assemble(configs, 1, spec)
    data["teacher01"] = rng.uniform(0.2, 0.8, 9).astype(np.float32)
    return data


def _targets(data):
    with Fitness(arrays=data) as e0:
        return synth.fill_targets(data, lambda _d, p: e0.find_force64(p))


def _check(data, pop, wtol=2e-6):
    P = len(pop)
    with Fitness(arrays=data) as e:
        fit, comps = e.compute(P, pop, components=True)
        E, W, _ = e.config_results(P)
        assert np.isfinite(comps).all()
        starts = np.concatenate([[0], np.cumsum(data["Na"])])
        N = e.N
        for p in (0, P // 2, P - 1):
            _, w, pe = e.find_force64(e.decode(pop[p]).astype(np.float64))
            w = w.reshape(6, N)
            for c in range(1, len(data["Na"])):
                a, b = starts[c], starts[c + 1]
                assert abs(E[p, c] - pe[a:b].sum()) <= wtol * np.abs(pe[a:b]).sum()
                assert np.abs(W[p, c] - w[:, a:b].sum(1)).max() <= wtol * np.abs(w[:, a:b]).sum()
        one = np.array([e.compute(1, pop[p:p + 1])[0] for p in (0, P - 1)])
    assert np.array_equal(one, fit[[0, P - 1]])  # the same bits alone
    return fit


@pytest.mark.parametrize("P", [1, 31, 33])
@pytest.mark.parametrize("na", [[64, 64, 63, 61], [64, 120, 121, 122, 216], [8, 512, 8, 64], [40, 240, 2, 241, 255, 5]])
def test_segments_and_groups(na, P):
    data = _targets(_cells(na))
    _check(data, synth.population(data, P, seed=P))


@pytest.mark.parametrize("sigma", [0.05, 0.25])
@pytest.mark.parametrize("frac,a", [(synth.DIAMOND, 5.43), ([[0, 0, 0]], 2.53), (synth.FLUORITE_CATION, 3.9),
                                    ([[0, 0, 0], [.5, .5, .5]], 3.08)])
def test_neighbors_and_cutoff_shell(frac, a, sigma):
    """4, 6, 12 and 14 neighbors; at sigma 0.25 many lie between R1 and R2."""
    if sigma == 0.25 and len(frac) == 2:
        sigma = 0.1  # 14 neighbors: more would pass the 16 that the force items take
    data = _targets(_cells([54, 64, 54, 128], sigma=sigma, a=a, frac=frac, cutoff=3.2))
    _check(data, synth.population(data, 40, seed=9))


def test_two_elements_and_fitted_S():
    data = synth.make(2, Nc=8, seed=12)
    data["potential_type"] = 2
    rng = np.random.default_rng(0)
    data["type"] = rng.integers(0, 2, len(data["type"])).astype(np.int32)
    lo = [2.7, 1.0, 2.2, 1.5, 2.8, 1.0, 2.2, 1.5, 0.5, 0.1, -1, 2.9, 3.2]
    hi = [3.3, 1.5, 2.4, 2.5, 3.3, 1.5, 2.4, 2.5, 1.5, 0.5, -0.5, 2.9, 3.2]
    data["pmin"], data["pmax"] = np.array(lo, np.float32), np.array(hi, np.float32)
    data["teacher01"] = rng.uniform(0, 1, 13).astype(np.float32)
    data = _targets(data)
    with Fitness(arrays=data) as e:
        pop = synth.population(data, 45, seed=4)
        fit, f64 = e.compute(45, pop), e.compute(45, pop, path=PATH_PLAIN64)
    assert np.abs(fit / f64 - 1).max() <= 1e-6


def test_outside_the_table():
    data = _cells([64, 64, 216])
    data["pmin"][4], data["pmax"][4] = 0.5, 12.0  # n
    data = _targets(data)
    pop = synth.population(data, 64, seed=6)
    pop[1, 5] = 0.0             # beta = 0
    pop[2, 6], pop[3, 6] = 4.0, -3.0  # h beyond its bounds
    pop[4, 4] = 0.0
    _check(data, pop, wtol=2e-5)
