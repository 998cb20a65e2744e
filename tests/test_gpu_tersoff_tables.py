"""The tables of the pair-by-pair Tersoff energy/virial items (csrc/tersoff_ev.cu) result by result: clusters of three
atoms, closed (six bond orders from the table) and open (the end atoms' s = 0 lies outside it: the exact form), whose
energy and virial hold so few bonds that no error averages out, beside cells that put the set on those items.  Bond
orders and exponentials, within what the tables represent and beyond.

Tolerances, from the sizes of the terms: b 7e-8 and b' 2e-7 of their size (tests/test_bond_table_cpu.py), the
argument s rounded to FP32 (6e-8, which b' takes up to (n + 1)-fold and b by half), the FP32 products and sums of
the virial six roundings of its terms, ds/d(strain) = X0 + (h - h0) X1 four of those two."""
import ctypes as C

import numpy as np
import pytest

from gpuga_b200 import Fitness, _lib, synth

pytestmark = pytest.mark.gpu

R = 2.0 ** -24
SMALL = 40


def _trimers(bounds, closed, seed=0):
    """A force cell, a 512-atom cell for every 12 trimers (64 pairs per configuration and more) and the trimers."""
    rng = np.random.default_rng(seed)
    configs = []
    for reps in [2] + [4] * (SMALL // 12 + 1):
        frac, cell = synth._structure(synth.DIAMOND, np.eye(3) * 5.43, (reps,) * 3)
        configs.append(synth._config(rng, frac, cell, np.zeros(len(frac)), 0.02, 0.1))
    for k in range(SMALL):
        a, b = rng.uniform(2.2, 2.75, 2)
        angle = rng.uniform(0.95, 1.05) if closed else rng.uniform(1.75, 2.6)
        pos = np.array([[0, 0, 0], [a, 0, 0], [b * np.cos(angle), b * np.sin(angle), 0]])
        turn, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        configs.append((pos @ turn.T + 10, np.eye(3) * 20.0, np.zeros(3, np.int32)))
    lo_hi = synth.SI_TERSOFF_BOUNDS.astype(np.float64)
    for k, v in bounds.items():
        lo_hi[k] = v
    spec = dict(potential_type=1, num_neurons=0, cutoff=3.2, w_force=0.05, w_energy=0.15, w_stress=0.8,
                pmin=lo_hi[:, 0].astype(np.float32), pmax=lo_hi[:, 1].astype(np.float32), ga={})
    data = synth._assemble(configs, 1, spec)
    data["teacher01"] = rng.uniform(0.2, 0.8, 9).astype(np.float32)
    with Fitness(arrays=data) as e0:
        return synth.fill_targets(data, lambda _d, p: e0.find_force64(p))


def _launches(e, P):
    n = C.c_int()
    rows = np.zeros((16, 8))
    _lib.check(_lib.load().gpuga_plan_info(e.handle, P, C.byref(n), C.c_void_p(rows.ctypes.data), 16))
    return rows[:n.value]


def _terms(par, pos, h0):
    """Sizes of the terms of three atoms: of the energy, of the virial without b', of its b' part, and of that part as a
    polynomial in h - h0."""
    D0, al, r0, S, n, beta, h = par[:7]
    la, lr = np.sqrt(2 / S) * al, np.sqrt(2 * S) * al
    energy = force = bent = poly = 0.0
    for i in range(3):
        for j in range(3):
            r = np.linalg.norm(pos[j] - pos[i])
            if j == i or r > 2.8:
                continue
            s, b, turn, terms = 0.0, 1.0, 0.0, 0.0
            for k in range(3):
                q = np.linalg.norm(pos[k] - pos[i])
                if k not in (i, j) and q < 2.8:
                    y = (pos[j] - pos[i]) @ (pos[k] - pos[i]) / (r * q) - h
                    s, turn = s + y * y, turn + 4 * abs(y)  # |ds/d(strain)| <= 4 |y|
                    terms += 4 * (abs(y + h - h0) + abs(h - h0))
            fr, fa = D0 / (S - 1) * np.exp(-lr * (r - r0)), S * D0 / (S - 1) * np.exp(-la * (r - r0))
            if s > 0:
                z = n * np.log(beta * s)
                b = np.exp(-np.logaddexp(0, z) / (2 * n))
                slope = 0.5 * fa * 0.5 * b / s * np.exp(z - np.logaddexp(0, z))
                bent, poly = bent + slope * turn, poly + slope * terms
            energy += 0.5 * (fr + b * fa)
            force += 0.5 * r * (lr * fr + b * la * fa)
    return energy, force, bent, poly


def _check(data, pop):
    P, N = len(pop), int(data["Na"].sum())
    starts = np.concatenate([[0], np.cumsum(data["Na"])])
    xyz = data["r"].reshape(3, N).T.astype(np.float64)
    h0 = (float(data["pmin"][6]) + float(data["pmax"][6])) / 2
    with Fitness(arrays=data) as e:
        e.compute(P, pop)
        E, W, _ = e.config_results(P)
        rows = _launches(e, P)
        assert np.any((rows[:, 0] == 0) & (rows[:, 1] == 0) & (rows[:, 2] == 0))  # the items by pairs
        for p in range(P):
            par = e.decode(pop[p]).astype(np.float64)
            _, w, pe = e.find_force64(par)
            w = w.reshape(6, N)
            for c in np.flatnonzero(data["Na"] == 3):
                a, b = starts[c], starts[c + 1]
                energy, force, bent, poly = _terms(par, xyz[a:b], h0)
                assert abs(E[p, c] - pe[a:b].sum()) <= (7e-8 + R / 2 + 1e-9) * energy
                tol = (7e-8 + R / 2 + 6 * R) * force + (2e-7 + (par[4] + 1) * R + 6 * R) * bent + 4 * R * poly
                assert np.abs(W[p, c] - w[:, a:b].sum(1)).max() <= tol


@pytest.mark.parametrize("closed", [True, False])
@pytest.mark.parametrize("n", [0.787, 3, 6, 12, 22.956, 50])
def test_bond_orders_one_by_one(n, closed):
    """beta s from below to above 1, where b bends."""
    data = _trimers({4: (0.97 * n, 1.03 * n), 5: (0.2, 2) if closed else (2, 20)}, closed)
    _check(data, np.random.default_rng(1).uniform(0, 1, (40, 9)).astype(np.float32))


@pytest.mark.parametrize("closed", [True, False])
@pytest.mark.parametrize("alpha,S", [(1.5, (2, 2)), (5, (1.5, 10)), (10, (2, 2)), (12, (1.5, 2)), (24, (2, 2)), (10, (1.5, 10)),
                                     (20, (1.5, 10))])
def test_exponentials_one_by_one(alpha, S, closed):
    """Decay constants l up to 25 / A, the steepest that the tables take; sets whose bounds allow more stay with the
    items by atom; and individuals outside their bounds.  r0 lies at the bonds, so that the terms are of one size
    whatever l is."""
    data = _trimers({1: (0.9 * alpha, alpha), 2: (2.4, 2.5), 3: S}, closed)
    steepest = alpha * max(np.sqrt(2 / S[0]), np.sqrt(2 * S[1]) if S != (2, 2) else 0)
    pop = np.random.default_rng(2).uniform(0, 1, (40, 9)).astype(np.float32)
    pop[5, 1] = (30 - 0.9 * alpha) / (0.1 * alpha)
    pop[6, 1] = -(0.9 * alpha) / (0.1 * alpha)  # alpha = 0
    if steepest <= 25:
        _check(data, pop)
    else:
        with Fitness(arrays=data) as e:
            e.compute(40, pop)
            rows = _launches(e, 40)
            assert not np.any((rows[:, 0] == 0) & (rows[:, 1] == 0) & (rows[:, 2] == 0))
