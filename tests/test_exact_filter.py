"""The exact M-sampler's split filter against the C restatement's serial one:
the same graphs bit for bit, with and without loci that start the filter anew,
and where likelihoods are so small that it falls back to one run."""
import numpy as np
import pytest

from oracle import port
from swiftlink_gb300 import api, pedigree, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()
    port.build()


# marker counts around the runs' 32-locus warps, the block's threads and its longest strides; untyped members leave
# few loci that start anew; tiny: loci where everybody is homozygous for one rare allele
@pytest.mark.parametrize("members,markers,untyped,tiny,seed", [
    (12, 2, 0.0, False, 1), (12, 31, 0.9, False, 2), (25, 33, 0.0, False, 3), (25, 65, 0.5, False, 4),
    (40, 511, 0.8, False, 5), (40, 515, 0.0, False, 6), (25, 1100, 0.3, False, 7), (40, 130, 0.0, True, 8),
    (25, 64, 0.5, True, 9)])
def test_exact_sweeps_equal_the_restatement(members, markers, untyped, tiny, seed):
    spec = synth.WorkloadSpec(n_members=members, generations=3 + (members >= 40), loops=1 if members >= 40 else 0,
                              affected=2, markers=markers, spacing_cm=0.5, maf=(0.05, 0.5), missing_all=0.05,
                              disease_cm=0.4)
    for k in range(20):
        try:
            g = pedigree.problem_from_workload(synth.make_workload(1, seed=seed + 1000 * k, spec=spec))
            break
        except RuntimeError:
            continue
    rng = np.random.default_rng(seed)
    g["genotypes"][:, rng.random(g["N"]) < untyped] = 0
    at = rng.permutation(markers)[:max(1, markers // 20)] if tiny else []
    g["genotypes"][at] = 3
    g["typed"] = (g["genotypes"] != 0).any(axis=0).astype(np.uint8)
    dg = np.ascontiguousarray(g["dg0"], np.int32)
    blank = dict(legal=np.full((markers, g["N"]), 15, np.uint8), trait_prior=np.zeros((markers, g["N"], 4)))
    g["minor"][at] = 0.5
    P = port.Port(dict(g, **blank))
    for l in at:   # the alleles in use there share a likelihood of about 1e-290
        g["minor"][l] = 10.0 ** (290 / np.log2(P.fag(dg, int(l))))
    meioses = rng.permutation(g["meioses"])[:12]
    u = rng.random((2, meioses.size, markers))
    with api.Context(api.Problem.from_arrays(g, with_legal=False), n_chains=2) as ctx:
        P = port.Port(dict(g, legal=ctx.legal_masks(), trait_prior=ctx.trait_priors()))
        ctx.set_graphs(np.stack([dg, dg]))
        ctx.msampler_sweep(meioses, u, n_chains=2)
        got = ctx.get_graphs()
    for l in at:
        assert 0.0 < P.fag(dg, int(l)) < 1e-280
    for c in range(2):
        want, _ = P.msweep(dg, meioses, u[c])
        assert np.array_equal(got[c], want), f"chain {c}"
