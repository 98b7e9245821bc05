"""The L-sampler with four lanes per task against the one with 32: the same
graphs bit for bit, in both arithmetics."""
import numpy as np
import pytest

from swiftlink_gb300 import api, pedigree, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()


def family(members, loops, markers, untyped, missing, seed):
    gens = 3 + (members >= 25) + (members >= 90) + (members >= 200)
    spec = synth.WorkloadSpec(n_members=members, generations=gens, loops=loops, affected=3, markers=markers,
                              spacing_cm=0.5, maf=(0.05, 0.5), missing_all=missing, disease_cm=0.4)
    for k in range(20):
        try:
            w = synth.make_workload(1, seed=seed + 1000 * k, spec=spec)
            break
        except RuntimeError:
            continue
    g = pedigree.problem_from_workload(w)
    out = np.random.default_rng(seed).random(g["N"]) < untyped
    g["genotypes"][:, out] = 0
    g["typed"] = (g["genotypes"] != 0).any(axis=0).astype(np.uint8)
    return g


# the last warp's idle lanes and a chain boundary inside a warp (markers x chains), wide cells (untyped members,
# rfunctions past the four cells kept in registers), the rfunctions in shared and in global memory
@pytest.mark.parametrize("members,loops,markers,untyped,missing,chains,seed", [
    (12, 0, 2, 0.0, 0.0, 1, 1), (25, 1, 17, 0.0, 0.3, 3, 2), (40, 2, 64, 0.25, 0.1, 2, 3),
    (60, 2, 101, 0.4, 0.3, 1, 4), (120, 3, 33, 0.1, 0.2, 5, 5), (250, 3, 40, 0.0, 0.05, 2, 6)])
@pytest.mark.parametrize("precision", [api.SL_SAMPLER_FAST, api.SL_SAMPLER_EXACT])
def test_four_lanes_draw_the_graphs_of_32(members, loops, markers, untyped, missing, chains, seed, precision):
    g = family(members, loops, markers, untyped, missing, seed)
    prob = api.Problem.from_arrays(g, with_legal=False)
    u = np.random.default_rng(seed).random((chains, markers, g["K"] + 2 * g["N"]))
    got = {}
    for form in (api.SL_LS_KERNEL_GENERIC32, api.SL_LS_KERNEL_GENERIC4):
        with api.Context(prob, n_chains=chains, sampler_precision=precision, ls_kernel=form) as ctx:
            dg = np.ascontiguousarray(g["dg0"], np.int32)
            ctx.set_graphs(np.broadcast_to(dg, (chains,) + dg.shape))
            out = []
            for sweep in range(2):   # injected draws, then the device's own
                if sweep == 0:
                    ctx.lsampler_sweep(u, n_chains=chains)
                else:
                    ctx.run(iterations=0, burnin=2, lprob=1.0, seed=9)
                out.append(ctx.get_graphs())
            loci = np.arange(0, markers, 3, dtype=np.int32)[::-1]   # a list of its own, out of order
            ctx.lsampler_loci(loci, u, n_chains=chains)
            out.append(ctx.get_graphs())
            got[form] = out
            assert ctx.ls_tuning()[0] == (32 if form == api.SL_LS_KERNEL_GENERIC32 else 4)
    a, b = got.values()
    assert markers < 10 or not np.array_equal(a[0][0], g["dg0"])
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
