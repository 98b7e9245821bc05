"""Fast M-sweeps by a cluster against the launches per meiosis that a shape
outside a cluster's shared memory takes: the same graphs bit for bit."""
import numpy as np
import pytest

from swiftlink_gb300 import api, pedigree, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()


def family(members, markers, untyped, seed):
    gens = 3 + (members >= 25) + (members >= 90) + (members >= 200)
    spec = synth.WorkloadSpec(n_members=members, generations=gens, loops=int(members >= 25), affected=3, markers=markers,
                              spacing_cm=0.5, maf=(0.05, 0.5), missing_all=0.05, disease_cm=0.4)
    for k in range(20):
        try:
            g = pedigree.problem_from_workload(synth.make_workload(1, seed=seed + 1000 * k, spec=spec))
            break
        except RuntimeError:
            continue
    g["genotypes"][:, np.random.default_rng(seed).random(g["N"]) < untyped] = 0
    g["typed"] = (g["genotypes"] != 0).any(axis=0).astype(np.uint8)
    return g


def contexts(prob, chains):
    for form in (api.SL_MSAMPLER_AUTO, api.SL_MSAMPLER_LAUNCHES):
        with api.Context(prob, n_chains=chains, sampler_precision=api.SL_SAMPLER_FAST) as ctx:
            ctx.msampler_set_form(form)
            yield form, ctx


# a warp a locus and two loci a warp (8 chains and more, up to 16 words a column: under 257 children), one locus past a
# mask word and a scan warp, most members untyped, columns kept in shared memory and (100,003 loci) not
@pytest.mark.parametrize("members,markers,untyped,chains", [
    (12, 2, 0.0, 1), (25, 65, 0.0, 7), (25, 65, 0.0, 8), (60, 1001, 0.6, 2), (60, 1001, 0.0, 40), (110, 2113, 0.1, 1),
    (110, 2113, 0.1, 9), (300, 333, 0.0, 9), (12, 100003, 0.0, 1)])
def test_sweeps(members, markers, untyped, chains):
    g = family(members, markers, untyped, members + markers)
    prob = api.Problem.from_arrays(g, with_legal=False)
    rng = np.random.default_rng(chains)
    meioses = rng.permutation(g["meioses"])[:7]
    u = rng.random((chains, meioses.size, markers))
    dg = np.broadcast_to(np.ascontiguousarray(g["dg0"], np.int32), (chains,) + g["dg0"].shape)
    got, launches = [], []
    for form, ctx in contexts(prob, chains):
        ctx.set_graphs(dg)
        at = ctx.launches
        ctx.msampler_sweep(meioses, u, n_chains=chains)   # injected draws, then the device's own
        launches.append(ctx.launches - at)
        got.append(ctx.get_graphs())
        if markers < 10000:
            ctx.run(iterations=0, burnin=2, lprob=0.0, seed=7)
            got.append(ctx.get_graphs())
    assert launches == [1, 1 + 2 * meioses.size]
    half = len(got) // 2
    assert markers < 10 or not np.array_equal(got[0], dg)
    assert all(np.array_equal(a, b) for a, b in zip(got[:half], got[half:]))


def test_form_changes_between_runs():
    """One context from form to form: the graphs of runs in one form."""
    g = family(40, 129, 0.0, 3)
    prob = api.Problem.from_arrays(g, with_legal=False)
    dg = np.broadcast_to(np.ascontiguousarray(g["dg0"], np.int32), (3,) + g["dg0"].shape)
    want = []
    for form, ctx in contexts(prob, 3):
        ctx.set_graphs(dg)
        for k in range(3):
            ctx.run(iterations=0, burnin=2 * k + 2, first_iteration=2 * k, lprob=0.5, seed=7)
        want.append(ctx.get_graphs())
    with api.Context(prob, n_chains=3, sampler_precision=api.SL_SAMPLER_FAST) as ctx:
        ctx.set_graphs(dg)
        for k, form in enumerate((api.SL_MSAMPLER_AUTO, api.SL_MSAMPLER_LAUNCHES, api.SL_MSAMPLER_AUTO)):
            ctx.msampler_set_form(form)
            ctx.run(iterations=0, burnin=2 * k + 2, first_iteration=2 * k, lprob=0.5, seed=7)
        got = ctx.get_graphs()
        with pytest.raises(api.SwiftLinkError):
            ctx.msampler_set_form(2)
    assert np.array_equal(want[0], want[1]) and np.array_equal(want[0], got)


def test_batch_shapes_smaller_clusters():
    """Contexts in a batch, whose load shapes their clusters, draw what each draws alone in either form."""
    gs = [family(m, k, 0.1, m) for m, k in ((25, 200), (60, 301), (110, 450))]
    probs = [api.Problem.from_arrays(g, with_legal=False) for g in gs]
    chains = 60
    dgs = [np.broadcast_to(np.ascontiguousarray(g["dg0"], np.int32), (chains,) + g["dg0"].shape) for g in gs]
    alone = []
    for prob, dg in zip(probs, dgs):
        for form, ctx in contexts(prob, chains):
            ctx.set_graphs(dg)
            ctx.run(iterations=0, burnin=2, lprob=0.0, seed=9)
            alone.append(ctx.get_graphs())
    ctxs = [api.Context(p, n_chains=chains, sampler_precision=api.SL_SAMPLER_FAST) for p in probs]
    for ctx, dg in zip(ctxs, dgs):
        ctx.set_graphs(dg)
    batch = api.Batch(ctxs)
    batch.run(iterations=0, burnin=2, lprob=0.0, seed=9)
    for k, ctx in enumerate(ctxs):
        got = ctx.get_graphs()
        assert np.array_equal(got, alone[2 * k]) and np.array_equal(got, alone[2 * k + 1])
    batch.close()
    for ctx in ctxs:
        ctx.close()
