"""A call that is refused, because a lane group's arenas do not fit a block's
shared memory, leaves the contexts made after it as they are."""
import numpy as np
import pytest

from conftest import load_golden
from swiftlink_gb300 import api, pedigree, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()


def wide():
    """45 members and 9 loops, most untyped: 10,000 cells a locus."""
    spec = synth.WorkloadSpec(n_members=45, generations=4, loops=9, affected=4, markers=21, spacing_cm=0.5,
                              maf=(0.05, 0.5), disease_cm=0.4)
    for k in range(30):
        try:
            g = pedigree.problem_from_workload(synth.make_workload(1, seed=2004000 + k, spec=spec))
            break
        except RuntimeError:
            continue
    g["genotypes"][:, np.random.default_rng(2004000).random(g["N"]) < 0.8] = 0
    g["genotypes"][:] = g["genotypes"][0]
    g["dg0"] = np.ascontiguousarray(np.broadcast_to(g["dg0"][:1], g["dg0"].shape), np.int32)
    g["typed"] = (g["genotypes"] != 0).any(axis=0).astype(np.uint8)
    return g


def test_the_next_context_works():
    g = wide()
    u = np.random.default_rng(1).random((1, g["M"], g["K"] + 2 * g["N"]))
    with api.Context(api.Problem.from_arrays(g, with_legal=False), ls_kernel=api.SL_LS_KERNEL_GENERIC8) as ctx:
        ctx.set_graphs(g["dg0"])
        with pytest.raises(api.SwiftLinkError):   # four tasks of 80 KB to a warp
            ctx.lsampler_sweep(u)
    small = load_golden("loop")
    with api.Context(api.Problem.from_arrays(small), n_chains=1) as ctx:
        ctx.set_graphs(small["dg0"])
        ctx.lsampler_sweep(small["lsweep_u"][None])
        assert np.array_equal(ctx.get_graphs()[0], small["lsweep_after"])
