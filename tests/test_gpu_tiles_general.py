"""Tiles of the Tersoff force items by atom (gpuga_options.tiles, csrc/batched.cu) on sets that run them: configurations with
fixed R1 and R2 and at most four bonds per atom have items of their own, whose one tile every option names, so here R1 is
fitted, or atoms have 6 to 14 neighbors; S fixed and fitted, one and two elements, the autotuner's choice.  Every tile gives
the same bits (atoms are summed in a canonical order)."""
import ctypes as C

import numpy as np
import pytest

from gpuga_b200 import Fitness, _lib, synth
from tests.test_gpu_tersoff_pairs import _cells, _targets

pytestmark = pytest.mark.gpu

P = 45  # a partial group of individuals in most tiles


def _data(kind):
    if kind == "polytypes":
        out = _cells([54, 54, 64, 128, 32], sigma=0.05, a=2.53, frac=[[0, 0, 0]], cutoff=3.2)
        other = _cells([54, 128, 64, 108, 54], sigma=0.05, a=3.08, frac=[[0, 0, 0], [.5, .5, .5]], cutoff=3.2)
        sets = []
        for d in (out, other):
            sets.append(_targets(dict(d, Nc_force=4)))
        return sets
    data = _cells([8, 64, 216, 512, 60, 64, 64], sigma=0.1, cutoff=3.2)
    data["Nc_force"] = 5
    if "two" in kind:
        rng = np.random.default_rng(1)
        data["potential_type"] = 2
        data["type"] = rng.integers(0, 2, len(data["type"])).astype(np.int32)
        lo = [2.7, 1.0, 2.2, 2, 2.8, 1.0, 2.2, 2, 0.5, 0.1, -1, 2.8, 3.2]
        hi = [3.3, 1.5, 2.4, 2, 3.3, 1.5, 2.4, 2, 1.5, 0.5, -0.5, 2.8, 3.2]
        data["pmin"], data["pmax"] = np.array(lo, np.float32), np.array(hi, np.float32)
        data["teacher01"] = rng.uniform(0, 1, 13).astype(np.float32)
    off = 4 if "two" in kind else 0
    data["pmin"][7 + off], data["pmax"][7 + off] = 2.5, 2.9
    if "S fitted" in kind:
        for k in (3, 7) if off else (3,):
            data["pmin"][k], data["pmax"][k] = 1.5, 2.5
    return [_targets(data)]


def _run(data, tiles, pop):
    with Fitness(arrays=data, tiles=tiles) as e:
        fit, comps = e.compute(P, pop, components=True)
        out = [fit, comps, *e.config_results(P)]
        n = C.c_int()
        rows = np.zeros((16, 8))
        _lib.check(_lib.load().gpuga_plan_info(e.handle, P, C.byref(n), C.c_void_p(rows.ctypes.data), 16))
        rows = rows[:n.value]
        forces = rows[rows[:, 2] > 0]
        assert len(forces) and np.all(forces[:, 1] >= 4)  # by atom, 4, 8 or 16 slots
        codes, _ = e.plan_tiles(P)
        alone = e.compute(1, pop[17:18])
        assert alone[0] == fit[17]
        return out, codes[:e.Nc_force]


@pytest.mark.parametrize("kind", ["R1 fitted", "R1 and S fitted", "two elements, R1 fitted", "two elements, R1 and S fitted",
                                  "polytypes"])
def test_every_tile_gives_the_same_bits(kind):
    for data in _data(kind):
        pop = synth.population(data, P, seed=5)
        ref, _ = _run(data, 1, pop)
        for tiles in (2, 3, 4, 5, 0):
            got, codes = _run(data, tiles, pop)
            for a, b in zip(got, ref):
                assert np.array_equal(a, b), f"tiles={tiles}"
            assert np.all(codes == tiles) if tiles else np.all((codes >= 1) & (codes <= 5))
