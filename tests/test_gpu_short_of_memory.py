"""Where the device has no room for the tables and buffers of an evaluation that another can stand in for, the other
takes its place: a population whose Tersoff tables (40 kB and more per 32 individuals) do not fit."""
import numpy as np
import pytest
import torch

from gpuga_b200 import PATH_PLAIN64, Fitness, synth
from tests.test_gpu_tersoff_pairs import _cells, _targets

pytestmark = pytest.mark.gpu


def test_population_without_room_for_its_tables():
    data = _targets(_cells([8, 64, 64]))
    P, some = 600_000, [0, 31, 299_999, 599_999]
    pop = np.random.default_rng(0).uniform(0, 1, (P, 9)).astype(np.float32)
    with Fitness(arrays=data) as e:
        e.compute(4, pop[some])
        exact = e.compute(4, pop[some], path=PATH_PLAIN64)
        torch.zeros(1, device="cuda")
        hold = []
        spare = 700_000_000  # results, constants and populations take 0.25 GB, the tables 0.75 GB and more
        while torch.cuda.mem_get_info()[0] > spare + (64 << 20):
            hold.append(torch.empty(min(torch.cuda.mem_get_info()[0] - spare, 8 << 30) & ~((2 << 20) - 1),
                                    dtype=torch.uint8, device="cuda"))
        fit = e.compute(P, pop)
        del hold
        torch.cuda.empty_cache()
        assert np.abs(fit[some] / exact - 1).max() <= 1e-6
        fit4 = e.compute(4, pop[some])  # its own plan has room
        assert np.abs(fit4 / exact - 1).max() <= 1e-6
