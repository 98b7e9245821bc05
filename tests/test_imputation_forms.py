"""Sequential imputation by four lanes and by a warp a pass against the oracle's
pass: more passes than a half-sweep has loci, the rfunctions in shared and in
global memory, wide ones, chains from the middle of a context."""
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


# cells an operation at the widest locus: 2 (in shared memory), 4, 19 and 26 (in global memory), 89 (9 and 75 passes by a warp each)
@pytest.mark.parametrize("members,generations,loops,untyped,seed", [
    (30, 4, 1, 0.0, 1000), (120, 6, 3, 0.4, 2000), (45, 4, 6, 0.3, 299000), (45, 4, 9, 0.3, 2004000),
    (45, 4, 9, 0.6, 2004000)])
@pytest.mark.parametrize("passes", [1, 9, 75])
def test_passes_equal_the_oracle(members, generations, loops, untyped, seed, passes):
    spec = synth.WorkloadSpec(n_members=members, generations=generations, loops=loops, affected=members // 10, markers=7,
                              spacing_cm=0.5, maf=(0.05, 0.5), missing_all=0.05, disease_cm=0.4)
    for k in range(30):
        try:
            g = pedigree.problem_from_workload(synth.make_workload(1, seed=seed + k, spec=spec))
            break
        except RuntimeError:
            continue
    rng = np.random.default_rng(seed)
    g["genotypes"][:, rng.random(g["N"]) < untyped] = 0
    g["typed"] = (g["genotypes"] != 0).any(axis=0).astype(np.uint8)
    M, N = g["M"], g["N"]
    starts = rng.integers(0, M, passes).astype(np.int32)
    u = rng.random((passes, M * (g["K"] + 2 * N)))
    none = np.zeros((M, N, 2), np.int32)
    with api.Context(api.Problem.from_arrays(g, with_legal=False), n_chains=passes + 2) as ctx:
        P = port.Port(dict(g, legal=ctx.legal_masks(), trait_prior=ctx.trait_priors()))
        ctx.set_graphs(np.broadcast_to(none, (passes + 2,) + none.shape))
        w = ctx.sequential_imputation(starts, u, first=1)
        got = ctx.get_graphs()
    assert not got[0].any() and not got[-1].any()
    for c in range(passes):
        dg, _, weight = P.si(none, int(starts[c]), u[c])
        assert np.array_equal(got[1 + c], dg), c
        assert abs(w[c] - weight) <= 1e-12 * abs(weight)
