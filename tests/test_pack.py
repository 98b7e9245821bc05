"""The caller's graphs packed by the device from host memory: every shape of
column, alignments of the caller's array, both sides of the size from which
the device does it."""
import numpy as np
import pytest

from conftest import load_golden
from swiftlink_gb300 import api, pedigree, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()


# 2 (N - F) below, at and above whole words; under and over 256 KB
@pytest.mark.parametrize("members,markers,chains", [(12, 40, 1), (12, 3001, 1), (24, 2000, 3), (33, 1023, 2), (60, 700, 5)])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_graphs_come_back(members, markers, chains, shift):
    spec = synth.WorkloadSpec(n_members=members, generations=3, loops=0, affected=2, markers=markers, spacing_cm=0.5,
                              maf=(0.05, 0.5), disease_cm=0.4)
    g = pedigree.problem_from_workload(synth.make_workload(1, seed=members, spec=spec))
    rng = np.random.default_rng(markers)
    want = rng.integers(-2**31, 2**31, (chains, markers, g["N"], 2)).astype(np.int32)   # only the lowest bit counts
    raw = np.empty(want.size + 4, np.int32)
    dg = raw[shift:shift + want.size].reshape(want.shape)   # 4-byte aligned only
    dg[:] = want
    want &= 1
    want[:, :, :g["F"]] = 0
    with api.Context(api.Problem.from_arrays(g, with_legal=False), n_chains=chains + 1) as ctx:
        ctx._check(api.lib().sl_set_descent_graphs(ctx.h, 1, chains, api._p(dg)))
        got = ctx.get_graphs()
        assert not got[0].any() and np.array_equal(got[1:], want)


def test_scores_of_packed_graphs():
    """Scoring n graphs in one call (packed by the device) or one at a time
    (below the size) gives one table."""
    g = load_golden("cfg1")
    graphs = np.concatenate([g["lod_graphs"]] * 24)
    prob = api.Problem.from_arrays(g)
    out = []
    for step in (1, graphs.shape[0]):
        with api.Context(prob) as ctx:
            for k in range(0, graphs.shape[0], step):
                ctx.lod_score_graphs(graphs[k:k + step])
            out.append(ctx.lod_results()[0])
    assert graphs.nbytes > 256 << 10 and graphs[:1].nbytes < 256 << 10
    assert np.array_equal(out[0], out[1])
