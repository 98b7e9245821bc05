"""The FP64 trait peel on pedigrees with several loops, whose matrices leave
room for four, two or one position in a warp's shared memory."""
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


# cells of the peel's matrices: 156, 528, 672, 1,256, 4,336, 12,832 (four positions' past a block's shared memory),
# 15,672 and 17,088 (two positions' past it)
@pytest.mark.parametrize("members,generations,loops,seed", [
    (45, 4, 1, 3), (120, 6, 3, 2), (45, 4, 4, 27), (120, 6, 7, 0), (45, 4, 7, 33), (60, 5, 9, 2), (120, 6, 7, 16),
    (60, 5, 9, 11)])
def test_wide_cutsets(members, generations, loops, seed):
    """From one graph to 20,000 positions and more, in both forms; the table
    within the tolerance of the other FP64 tables."""
    spec = synth.WorkloadSpec(n_members=members, generations=generations, loops=loops, affected=members // 10, markers=81,
                              spacing_cm=0.5, maf=(0.05, 0.5), penetrance=(0.01, 0.8, 0.9), disease_freq=1e-3,
                              disease_cm=0.4)
    for k in range(30):
        try:
            g = pedigree.problem_from_workload(synth.make_workload(1, seed=seed + 1000 * k, spec=spec))
            break
        except RuntimeError:
            continue
    dg = np.ascontiguousarray(g["dg0"], np.int32)
    other = dg.copy()
    other[:, g["F"]:] ^= (np.random.default_rng(seed).random((g["M"], g["N"] - g["F"], 2)) < 0.02).astype(np.int32)
    pair = np.stack([dg, other])
    legal = dict(legal=np.full((g["M"], g["N"]), 15, np.uint8), trait_prior=np.zeros((g["M"], g["N"], 4)))
    want = {n: api.lod_table(*port.Port(dict(g, **legal)).lod(pair[:n])) for n in (1, 2)}
    for precision in (api.SL_LOD_FP64, api.SL_LOD_FP64_RESCALED):
        with api.Context(api.Problem.from_arrays(g, with_legal=False), n_chains=1, lod_precision=precision) as ctx:
            for graphs in (1, 2, 64):   # 400 positions a graph
                ctx.lod_reset()
                ctx.lod_score_graphs(pair[np.arange(graphs) % 2])
                got = api.lod_table(*ctx.lod_results())
                assert np.abs(got - want[min(graphs, 2)]).max() <= 1e-10, (precision, graphs)
