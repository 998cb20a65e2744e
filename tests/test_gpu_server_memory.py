"""The server's admission estimate covers what an admitted job takes on the device: engine, plan, launch set and GA state,
for sets that use each of the evaluations with memory of their own."""
import time

import numpy as np
import pytest
import torch

from gpuga_b200 import Server, synth

pytestmark = pytest.mark.gpu


def _sets():
    yield "Tersoff, cells of 1000 atoms, population 1000", synth.diamond_set([5] * 40, 4, P=1000)
    yield "Tersoff, packed forces", synth.diamond_set([4] * 60, 58, P=200)
    two = synth.diamond_set([5] * 30, 3, P=640)
    two["potential_type"] = 2
    lo = [2.7, 1.0, 2.2, 1.5, 2.8, 1.0, 2.2, 1.5, 0.5, 0.1, -1, 2.9, 3.2]
    hi = [3.3, 1.5, 2.4, 2.5, 3.3, 1.5, 2.4, 2.5, 1.5, 0.5, -0.5, 2.9, 3.2]
    two["pmin"], two["pmax"] = np.array(lo, np.float32), np.array(hi, np.float32)
    two["type"] = np.random.default_rng(0).integers(0, 2, len(two["type"])).astype(np.int32)
    yield "two elements, S fitted", two
    yield "rigid ion", synth.make(3, Nc=60)
    yield "network", synth.make(4, Nc=60)


def _dir(data, path):
    rng = np.random.default_rng(1)
    data = dict(data)
    for k in ("pe_ref", "virial_ref", "force_ref"):
        data[k] = rng.normal(size=len(data[k])).astype(np.float32)
    if data["potential_type"] == 2:
        names = synth.write_dir(dict(data, potential_type=1, pmin=data["pmin"][:9], pmax=data["pmax"][:9]), path)
        rows = "".join(f"p{k} {a:.9g} {b:.9g}\n" for k, (a, b) in enumerate(zip(data["pmin"], data["pmax"])))
        with open(f"{names}/potential.in", "w") as f:
            f.write("potential_type 2\ncutoff 3.2\nweight_force 0.3\nweight_energy 0.3\nweight_virial 0.4\n" + rows)
        return names
    return synth.write_dir(data, path)


def test_estimate_covers_the_footprint(tmp_path):
    torch.zeros(1, device="cuda")
    for turn in range(2):  # the first round brings the kernels' code and stacks
        for k, (name, data) in enumerate(_sets()):
            d = _dir(data, str(tmp_path / f"{turn}{k}"))
            with Server(device=0, max_jobs=2) as srv:
                srv.hold(True)
                before = torch.cuda.mem_get_info()[0]
                job = srv.submit(d, seed=3, generations=2)
                deadline = time.time() + 60
                while srv.poll(job)[3] == Server.QUEUED and time.time() < deadline:
                    time.sleep(0.01)
                taken, estimate = before - torch.cuda.mem_get_info()[0], srv.stats()["device_bytes"]
                srv.hold(False)
                assert srv.drain(120) == 0
                assert srv.poll(job)[0] == 0
            if turn:
                assert estimate >= taken, f"{name}: {taken / 1e6:.1f} MB taken, estimated {estimate / 1e6:.1f}"
