"""The exact M-sampler where recombination fractions are so small that their
product with a filtered value underflows: the C restatement's graphs, bit for bit."""
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


# Two loci without genotypes above one where a meiosis shows: the first of them is filtered to (1, first); times second,
# its smaller value is zero, and the choice there takes no draw.  1e-20: the smallest fraction that leaves the runs apart.
@pytest.mark.parametrize("first,second", [(1e-250, 1e-100), (1e-200, 1e-300), (1e-20, 1e-20), (0.005, 1e-300)])
def test_tiny_recombination_fractions(first, second):
    spec = synth.WorkloadSpec(n_members=25, generations=3, loops=0, affected=2, markers=65, spacing_cm=0.5,
                              maf=(0.05, 0.5), missing_all=0.05, disease_cm=0.4)
    g = pedigree.problem_from_workload(synth.make_workload(1, seed=11, spec=spec))
    g["theta"] = np.array(g["theta"], np.float64)
    for at in range(10, 60, 5):
        g["genotypes"][at:at + 2] = 0
        g["theta"][at - 1:at + 1] = first, second
    rng = np.random.default_rng(12)
    meioses = rng.permutation(g["meioses"])[:20]
    u = rng.random((2, meioses.size, g["M"]))
    dg = np.ascontiguousarray(g["dg0"], np.int32)
    with api.Context(api.Problem.from_arrays(g, with_legal=False), n_chains=2) as ctx:
        P = port.Port(dict(g, legal=ctx.legal_masks(), trait_prior=ctx.trait_priors()))
        ctx.set_graphs(np.stack([dg, dg]))
        ctx.msampler_sweep(meioses, u, n_chains=2)
        got = ctx.get_graphs()
    for c in range(2):
        want, _ = P.msweep(dg, meioses, u[c])
        assert np.array_equal(got[c], want), f"chain {c}"
