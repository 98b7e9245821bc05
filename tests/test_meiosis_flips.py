"""The fast M-sampler's rule on which toggled likelihoods it evaluates
(sl_problem_meiosis_flips) against the founder-allele-graph likelihood of the
C restatement, and its clusters against one another."""
import ctypes

import numpy as np
import pytest

from oracle import port
from swiftlink_gb300 import api, pedigree, synth


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()
    port.build()


def family(members, loops, markers, untyped, missing, seed):
    """A looped pedigree with whole members and single genotypes untyped, and a legal graph."""
    gens = 3 + (members >= 25) + (members >= 90)
    spec = synth.WorkloadSpec(n_members=members, generations=gens, loops=loops, affected=3, markers=markers,
                              spacing_cm=0.5, maf=(0.05, 0.5), missing_all=missing, disease_cm=0.4)
    for k in range(20):   # the first seed whose topology has the shape
        try:
            w = synth.make_workload(1, seed=seed + 1000 * k, spec=spec)
            break
        except RuntimeError:
            continue
    g = pedigree.problem_from_workload(w)
    rng = np.random.default_rng(seed)
    out = rng.random(g["N"]) < untyped
    g["genotypes"][:, out] = 0
    g["typed"] = (g["genotypes"] != 0).any(axis=0).astype(np.uint8)
    return g


def flips(g, dg=None):
    prob = api.Problem.from_arrays(g, with_legal=False)
    desc = prob.desc()
    out = np.zeros((2 * (g["N"] - g["F"]), g["M"]), np.uint8)
    at = None if dg is None else dg.ctypes.data_as(ctypes.c_void_p)
    assert api.lib().sl_problem_meiosis_flips(ctypes.byref(desc), at, out.ctypes.data_as(ctypes.c_void_p)) == 0
    return out


# pedigree sizes, loops (inbred members and marriages between relatives), untyped members, missing genotypes,
# marker counts on both sides of a mask word
@pytest.mark.parametrize("members,loops,markers,untyped,missing,seed", [
    (12, 0, 33, 0.0, 0.0, 1), (25, 1, 64, 0.0, 0.3, 2), (40, 3, 31, 0.3, 0.1, 3), (60, 2, 32, 0.6, 0.05, 4),
    (110, 4, 40, 0.1, 0.5, 5), (110, 3, 65, 0.0, 0.05, 6)])
def test_flips_follow_from_the_genotypes(members, loops, markers, untyped, missing, seed):
    """Every (meiosis, locus) that the rule decides, on two legal graphs (the
    gene drop's, and one moved away from it by legal toggles): the toggled
    likelihood is the current one (the same factors; 1e-12 covers their order)
    or zero."""
    g = family(members, loops, markers, untyped, missing, seed)
    rule = flips(g)
    assert not np.any(rule == 3)
    P = port.Port(dict(g, legal=np.full((g["M"], g["N"]), 15, np.uint8), trait_prior=np.zeros((g["M"], g["N"], 4))))
    rng = np.random.default_rng(seed + 100)
    dg = np.ascontiguousarray(g["dg0"], np.int32)
    decided = 0
    for graph in range(2):
        for l in range(g["M"]):
            base = P.fag(dg, l)
            assert base > 0.0
            for m in rng.permutation(rule.shape[0]):
                person, par = g["F"] + m // 2, m % 2
                if graph == 1 and rule[m, l] == 0 and rng.random() < 0.7:
                    continue
                dg[l, person, par] ^= 1
                lk = P.fag(dg, l)
                if rule[m, l] == 1:
                    assert abs(lk - base) <= 1e-12 * base, (m, l)
                elif rule[m, l] == 2:
                    assert lk == 0.0, (m, l)
                decided += rule[m, l] != 0
                if lk > 0.0 and rng.random() < 0.5:
                    base = lk   # keep the toggle: another legal graph
                else:
                    dg[l, person, par] ^= 1
    assert decided > 0


@pytest.mark.parametrize("members,loops,markers,untyped,missing,seed", [
    (12, 0, 33, 0.0, 0.0, 1), (30, 1, 64, 0.0, 0.3, 2), (40, 3, 31, 0.3, 0.1, 3), (60, 2, 32, 0.6, 0.05, 4),
    (110, 4, 40, 0.1, 0.5, 5), (110, 3, 65, 0.0, 0.05, 6)])
def test_flips_that_follow_from_the_graph(members, loops, markers, untyped, missing, seed):
    """The same with the graph's own meioses (relatives' alleles), on the gene
    drop's graph and on three graphs moved away from it by legal toggles."""
    g = family(members, loops, markers, untyped, missing, seed)
    P = port.Port(dict(g, legal=np.full((g["M"], g["N"]), 15, np.uint8), trait_prior=np.zeros((g["M"], g["N"], 4))))
    rng = np.random.default_rng(seed + 200)
    dg = np.ascontiguousarray(g["dg0"], np.int32)
    alone = flips(g)
    for graph in range(4):
        rule = flips(g, dg)
        assert not np.any(rule == 3) and np.array_equal(rule[alone != 0], alone[alone != 0])
        assert members < 30 or ((rule != 0) & (alone == 0)).any()
        for m, l in zip(*np.nonzero((rule != 0) & (alone == 0))):
            person, par = g["F"] + m // 2, m % 2
            base = P.fag(dg, int(l))
            dg[l, person, par] ^= 1
            lk = P.fag(dg, int(l))
            dg[l, person, par] ^= 1
            assert base > 0.0
            if rule[m, l] == 1:
                assert abs(lk - base) <= 1e-12 * base, (m, l)
            else:
                assert lk == 0.0, (m, l)
        for l in range(g["M"]):   # another legal graph
            for m in rng.permutation(rule.shape[0]):
                person, par = g["F"] + m // 2, m % 2
                dg[l, person, par] ^= 1
                if rng.random() < 0.5 or P.fag(dg, l) == 0.0:
                    dg[l, person, par] ^= 1


@pytest.mark.gpu
@pytest.mark.parametrize("members,markers,untyped", [(25, 2, 0.0), (25, 63, 0.3), (25, 65, 0.0), (40, 129, 0.2),
                                                     (60, 1000, 0.0), (110, 2113, 0.1)])
def test_sweep_is_the_same_whatever_the_cluster(members, markers, untyped):
    """Contexts of 1, 5 and 7 chains shape their clusters differently from a
    context of 600 chains' worth of load (a batch), and all sweep chain 0
    alike, bit for bit; 8 and 40 chains likewise (two graphs per warp there)."""
    g = family(members, 1, markers, untyped, 0.05, members + markers)
    nm = min(len(g["meioses"]), 30)
    prob = api.Problem.from_arrays(g, with_legal=False)
    u = np.random.default_rng(3).random((nm, markers))
    got = {}
    for chains in (1, 5, 7, 8, 40):
        with api.Context(prob, n_chains=chains, sampler_precision=api.SL_SAMPLER_FAST) as ctx:
            dg = np.ascontiguousarray(g["dg0"], np.int32)
            ctx.set_graphs(np.broadcast_to(dg, (chains,) + dg.shape))
            ctx.msampler_sweep(g["meioses"][:nm], np.broadcast_to(u, (chains,) + u.shape), n_chains=chains)
            out = ctx.get_graphs()
        assert all(np.array_equal(out[0], x) for x in out), f"{chains} chains: a chain differs from the first"
        got[chains] = out[0]
    assert not np.array_equal(got[1], dg)
    assert np.array_equal(got[1], got[5]) and np.array_equal(got[1], got[7])
    assert np.array_equal(got[8], got[40])


# groups of steps whose likelihoods are evaluated together: whole, cut short, more of them than a block keeps (untyped
# members), columns that change within a group
@pytest.mark.gpu
@pytest.mark.parametrize("members,markers,untyped,missing,steps", [
    (25, 40, 0.0, 0.05, 1), (25, 40, 0.0, 0.05, 3), (25, 70, 0.3, 0.05, 4), (25, 70, 0.6, 0.4, 5),
    (40, 129, 0.0, 0.7, 22), (60, 1000, 0.4, 0.2, 31)])
@pytest.mark.parametrize("chains", [2, 8])
def test_sweep_is_its_steps_one_by_one(members, markers, untyped, missing, steps, chains):
    g = family(members, 1, markers, untyped, missing, members + markers)
    nm = min(len(g["meioses"]), steps)
    prob = api.Problem.from_arrays(g, with_legal=False)
    u = np.random.default_rng(steps).random((chains, nm, markers))
    dg = np.broadcast_to(np.ascontiguousarray(g["dg0"], np.int32), (chains,) + g["dg0"].shape)
    out = []
    for step in (nm, 1):
        with api.Context(prob, n_chains=chains, sampler_precision=api.SL_SAMPLER_FAST) as ctx:
            ctx.set_graphs(dg)
            for k in range(0, nm, step):
                ctx.msampler_sweep(g["meioses"][k:k + step], np.ascontiguousarray(u[:, k:k + step]), n_chains=chains)
            out.append(ctx.get_graphs())
    assert np.array_equal(out[0], out[1])


# clusters of every size between 16 and 1 blocks, as the number of chains shapes them, and scan warps that a size does not divide
@pytest.mark.gpu
@pytest.mark.parametrize("members,markers", [(30, 200), (60, 1000), (110, 2113)])
def test_sweep_is_the_same_in_clusters_of_any_size(members, markers):
    g = family(members, 1, markers, 0.1, 0.05, members)
    prob = api.Problem.from_arrays(g, with_legal=False)
    u = np.random.default_rng(4).random((6, markers))
    dg = np.ascontiguousarray(g["dg0"], np.int32)
    got = []
    for chains in (8, 9, 13, 16, 20, 28, 36, 48, 70, 160):
        with api.Context(prob, n_chains=chains, sampler_precision=api.SL_SAMPLER_FAST) as ctx:
            ctx.set_graphs(np.broadcast_to(dg, (chains,) + dg.shape))
            ctx.msampler_sweep(g["meioses"][:6], np.broadcast_to(u, (chains,) + u.shape), n_chains=chains)
            out = ctx.get_graphs()
        assert all(np.array_equal(out[0], x) for x in out), f"{chains} chains: a chain differs from the first"
        got.append(out[0])
    assert all(np.array_equal(got[0], x) for x in got)
