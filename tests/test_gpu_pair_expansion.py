"""The pair expansion (csrc/spectral.cu) against the FP64 path, at the edges of its blocking: row
blocks of 8 and chunks of 192 rows (2 to 72 atoms per configuration), groups of 8 and 32 individuals,
sets without force or energy/virial configurations next to ones with both, every width class of the
network; and the individuals that it leaves to the direct items.

Tolerances.  Coefficients and sums are FP64 and a dropped coefficient is below 1e-9 of the function's
scale, so fitness components agree with the FP64 path to 1e-7 (two decades for fitness values a
hundredth of the targets); per-atom forces come back in FP32 (6e-8 of their size, 1e-6 of scale)."""
import numpy as np
import pytest

from gpuga_b200 import PATH_PLAIN64, Fitness, synth

pytestmark = pytest.mark.gpu


def _cut(data, na, Ncf):
    """The first na[c] atoms of configuration c, the first Ncf of them force configurations."""
    starts = np.concatenate([[0], np.cumsum(data["Na"])[:-1]])
    keep = np.concatenate([np.arange(starts[c], starts[c] + n) for c, n in enumerate(na)])
    N = int(data["Na"].sum())
    out = dict(data)
    pick = lambda a: np.concatenate([a[k * N:(k + 1) * N][keep] for k in range(3)])  # noqa: E731
    out.update(Na=np.array(na, np.int32), Nc_force=Ncf, type=data["type"][keep], r=pick(data["r"]),
               box9=data["box9"][:9 * len(na)], force_ref=np.zeros(3 * len(keep), np.float32),
               pe_ref=np.zeros(len(na), np.float32), virial_ref=np.zeros(6 * len(na), np.float32))
    return out


def _set(kind, na, Ncf, neurons=16, neutral=False):
    data = synth.make(3 if kind == "ri" else 4, Nc=len(na), neurons=neurons, seed=17)
    kw = {} if kind == "ri" else dict(nn2b_r1=data["nn2b_r1"], nn2b_r2=data["nn2b_r2"])
    data = _cut(data, na, Ncf)
    if neutral:
        data["potential_type"] = 4
    with Fitness(arrays=data, **kw) as e0:
        data = synth.fill_targets(data, lambda _d, p: e0.find_force64(p))
    return data, kw


def _check(data, kw, P, pop, rtol):
    with Fitness(arrays=data, **kw) as e:
        fit, comps = e.compute(P, pop, components=True)
        f64, c64 = e.compute(P, pop, path=PATH_PLAIN64, components=True)
    ok = np.isfinite(c64)
    assert np.array_equal(ok, np.isfinite(comps))
    assert np.abs(comps[ok] / c64[ok] - 1).max() <= rtol
    return fit


@pytest.mark.parametrize("P", [1, 8, 31, 33, 65])
@pytest.mark.parametrize("na,Ncf", [([64] * 24 + [64] * 25, 24), ([63, 64, 61, 62, 64, 60], 3),
                                    ([64, 8, 48, 3, 2, 64, 64, 24], 5)])
def test_rigid_ion_blocks(na, Ncf, P):
    data, kw = _set("ri", na, Ncf, neutral=P == 33)
    _check(data, kw, P, synth.population(data, P, seed=P), 1e-7)


@pytest.mark.parametrize("consistent", [False, True])
@pytest.mark.parametrize("neurons,P", [(4, 40), (8, 33), (9, 7), (10, 64), (16, 40), (17, 9), (32, 33)])
def test_network_widths(neurons, P, consistent):
    data, kw = _set("nn", [64] * 6 + [63, 64, 62, 64, 64, 64], 6, neurons=neurons)
    kw["nn2b_consistent"] = consistent
    _check(data, kw, P, synth.population(data, P, seed=neurons), 1e-7)


def test_forces_and_config_results():
    for data, kw in (_set("ri", [64, 62, 64, 30], 2), _set("nn", [64, 62, 64, 30], 2)):
        P = 3
        pop = synth.population(data, P, seed=2)
        with Fitness(arrays=data, **kw) as e:
            forces = e.batched_forces(pop)  # from the direct items
            e.compute(P, pop)
            E, W, F2 = e.config_results(P)
            N, Nf, starts = e.N, e.N_force, np.concatenate([[0], np.cumsum(data["Na"])])
            for p in range(P):
                F, w, pe = e.find_force64(e.decode(pop[p]).astype(np.float64))
                F = F.reshape(3, N)[:, :Nf]
                assert np.abs(forces[p] - F).max() <= 1e-6 * np.abs(F).max()
                d2 = ((F - data["force_ref"].reshape(3, N)[:, :Nf]) ** 2).sum(0)
                for c in range(len(data["Na"])):
                    a, b = starts[c], starts[c + 1]
                    if c < 2:
                        assert abs(F2[p, c] / d2[a:b].sum() - 1) <= 1e-7 and E[p, c] == 0 and not W[p, c].any()
                    else:
                        wc = w.reshape(6, N)[:, a:b].sum(1)
                        assert abs(E[p, c] - pe[a:b].sum()) <= 1e-7 * np.abs(pe[a:b]).sum()
                        assert np.abs(W[p, c] - wc).max() <= 1e-7 * np.abs(w.reshape(6, N)[:, a:b]).sum()


@pytest.mark.parametrize("kind", ["ri", "nn"])
def test_individuals_left_to_the_direct_items(kind):
    """Parameters far outside their bounds (an exponential of 0.01 A, weights of 30): evaluated pair by
    pair, with the FP32 error of that form on such steep functions; every other individual keeps its bits."""
    data, kw = _set(kind, [64] * 8, 4)
    P = 70
    pop = synth.population(data, P, seed=5)
    steep = pop.copy()
    for p in (0, 33, 69):
        if kind == "ri":
            steep[p, 8] = (0.01 - 0.12) / 0.08  # rho11
        else:
            steep[p] = 5.5 * np.sign(steep[p] - 0.5) + 0.5
    left = np.isin(np.arange(P), (0, 33, 69))
    with Fitness(arrays=data, **kw) as e:
        alone = e.compute(P, pop)
        fit = e.compute(P, steep)
        again = e.compute(P, pop)
        f64 = e.compute(P, steep, path=PATH_PLAIN64)
    assert np.array_equal(alone, again)
    assert np.array_equal(fit[~left], alone[~left])
    assert np.abs(fit / f64 - 1)[left].max() <= 1e-4
