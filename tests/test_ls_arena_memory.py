"""The four-lane L-sampler's arena in global memory: its bound, and that a
context whose timing chose another kernel does not keep it."""
import numpy as np
import pytest

from swiftlink_gb300 import api, pedigree, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()


def wide(markers, untyped):
    """45 members and 9 loops, most untyped, every marker alike."""
    spec = synth.WorkloadSpec(n_members=45, generations=4, loops=9, affected=4, markers=markers, spacing_cm=0.5,
                              maf=(0.05, 0.5), disease_cm=0.4)
    for k in range(30):
        try:
            g = pedigree.problem_from_workload(synth.make_workload(1, seed=2004000 + k, spec=spec))
            break
        except RuntimeError:
            continue
    g["genotypes"][:, np.random.default_rng(2004000).random(g["N"]) < untyped] = 0
    g["genotypes"][:] = g["genotypes"][0]
    g["dg0"] = np.broadcast_to(g["dg0"][:1], g["dg0"].shape)
    g["typed"] = (g["genotypes"] != 0).any(axis=0).astype(np.uint8)
    return g


def used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_bound():
    """3,000 chains at eight warps and 7,458 cells each would take 5.3 GiB; every chain's sweep is 32 lanes' still."""
    g, chains = wide(4, 0.8), 3000
    prob = api.Problem.from_arrays(g, with_legal=False)
    got, grown = [], []
    for form in (api.SL_LS_KERNEL_GENERIC32, api.SL_LS_KERNEL_GENERIC4):
        before = used()
        with api.Context(prob, n_chains=chains, sampler_precision=api.SL_SAMPLER_FAST, ls_kernel=form) as ctx:
            grown.append(used() - before)
            ctx.set_graphs(np.broadcast_to(np.ascontiguousarray(g["dg0"], np.int32), (chains,) + g["dg0"].shape))
            u = np.random.default_rng(1).random((chains, g["M"], g["K"] + 2 * g["N"]))
            ctx.lsampler_sweep(u, n_chains=chains)
            got.append(ctx.get_graphs())
    assert 1 << 30 < grown[1] - grown[0] <= (4 << 30) + (64 << 20)
    assert np.array_equal(got[0], got[1])


def test_given_back():
    g, chains = wide(21, 0.6), 50
    prob = api.Problem.from_arrays(g, with_legal=False)
    grown = []
    for form in (api.SL_LS_KERNEL_GENERIC32, api.SL_LS_KERNEL_GENERIC32, api.SL_LS_KERNEL_GENERIC):
        with api.Context(prob, n_chains=chains, sampler_precision=api.SL_SAMPLER_EXACT, ls_kernel=form) as ctx:
            ctx.set_graphs(np.broadcast_to(np.ascontiguousarray(g["dg0"], np.int32), (chains,) + g["dg0"].shape))
            before = used()
            u = np.random.default_rng(1).random((chains, g["M"], g["K"] + 2 * g["N"]))
            ctx.lsampler_sweep(u, n_chains=chains)
            grown.append(used() - before)
            assert form == api.SL_LS_KERNEL_GENERIC32 or ctx.ls_tuning()[0] != 4
    assert grown[2] - grown[1] < 32 << 20   # the arena takes 83 MB
