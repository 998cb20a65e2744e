"""A cell of thousands of atoms in the pair expansion: its triangle is factored in dozens of levels (808 columns against
tiles of 1024 rows), whose work space is given back level by level."""
import threading

import numpy as np
import pytest
import torch

from gpuga_b200 import PATH_PLAIN64, Fitness, synth

pytestmark = pytest.mark.gpu


def test_levels_of_a_large_cell():
    data = synth.make(4, Nc=2, neurons=32, seed=3)
    frac, cell = synth._structure(synth.DIAMOND, np.eye(3) * 5.43, (8, 8, 8))
    rng = np.random.default_rng(0)
    configs = [synth._config(rng, frac, cell, np.zeros(len(frac)), 0.0, 0.15)]
    frac, cell = synth._structure(synth.DIAMOND, np.eye(3) * 5.43, (3, 3, 3))
    configs += [synth._config(rng, frac, cell, np.zeros(len(frac)), 0.0, 0.15) for _ in range(2)]
    spec = {k: data[k] for k in ("potential_type", "num_neurons", "w_force", "w_energy", "w_stress", "pmin", "pmax", "ga")}
    teacher, kw = data["teacher01"], dict(nn2b_r1=7.0, nn2b_r2=8.0)
    data = dict(synth._assemble(configs, 1, dict(spec, cutoff=8.0)), teacher01=teacher)
    torch.zeros(1, device="cuda")
    with Fitness(arrays=data, **kw) as e0:
        data = synth.fill_targets(data, lambda _d, p: e0.find_force64(p))
    free, done = [], threading.Event()

    def watch():
        while not done.wait(0.0005):
            free.append(torch.cuda.mem_get_info()[0])

    t = threading.Thread(target=watch)
    pop = synth.population(data, 6, seed=1)
    with Fitness(arrays=data, **kw) as e0:
        e0.compute(6, pop)  # the kernels' code and stacks
    t.start()
    try:
        e = Fitness(arrays=data, **kw)
        _, comps = e.compute(6, pop, components=True)  # the first plan builds the expansion
    finally:
        done.set()
        t.join()
    with e:
        after = torch.cuda.mem_get_info()[0]
        level = 24 * 4096 * 1024  # the first, of at most 1024 columns
        assert after - min(free) <= 2 * level + (64 << 20)  # two levels at a time, and the lists' scratch
        _, exact = e.compute(6, pop, path=PATH_PLAIN64, components=True)
    assert np.abs(comps / exact - 1).max() <= 1e-7
