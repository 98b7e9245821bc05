"""The L-sampler's lanes where nothing is asked for: four by rule on narrow
rfunctions, by timing on wide ones; the graphs are those of 32 lanes."""
import numpy as np
import pytest

from swiftlink_gb300 import api, pedigree, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()


# cells an operation at the widest locus: 4; 19; 12 with fewer tasks than warps fit, and with more
@pytest.mark.parametrize("members,generations,loops,untyped,markers,chains,timed", [
    (30, 4, 1, 0.0, 21, 2, False), (45, 4, 6, 0.3, 7, 13, True), (45, 4, 6, 0.4, 21, 13, True),
    (45, 4, 6, 0.4, 21, 200, False)])
def test_choice(members, generations, loops, untyped, markers, chains, timed):
    spec = synth.WorkloadSpec(n_members=members, generations=generations, loops=loops, affected=members // 10,
                              markers=markers, spacing_cm=0.5, maf=(0.05, 0.5), missing_all=0.05, disease_cm=0.4)
    for k in range(30):
        try:
            g = pedigree.problem_from_workload(synth.make_workload(1, seed=299000 + k, spec=spec))
            break
        except RuntimeError:
            continue
    g["genotypes"][:, np.random.default_rng(299000).random(g["N"]) < untyped] = 0
    g["typed"] = (g["genotypes"] != 0).any(axis=0).astype(np.uint8)
    prob = api.Problem.from_arrays(g, with_legal=False)
    dg = np.ascontiguousarray(g["dg0"], np.int32)
    got = []
    for form in (api.SL_LS_KERNEL_GENERIC, api.SL_LS_KERNEL_GENERIC32):
        with api.Context(prob, n_chains=chains, sampler_precision=api.SL_SAMPLER_FAST, ls_kernel=form) as ctx:
            ctx.set_graphs(np.broadcast_to(dg, (chains,) + dg.shape))
            ctx.run(iterations=0, burnin=2, lprob=1.0, seed=5)
            got.append(ctx.get_graphs())
            lanes, times = ctx.ls_tuning()
            if form == api.SL_LS_KERNEL_GENERIC:
                assert (times[0] > 0) == timed and (timed or lanes == 4)
    assert np.array_equal(got[0], got[1])
