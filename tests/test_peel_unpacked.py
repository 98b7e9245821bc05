"""A peel sequence that the four-lane L-sampler does not pack (more than 31
previous rfunctions at an operation): sweeps and imputation by the kernels of a
warp a task, against the oracle."""
import numpy as np
import pytest

from oracle import port
from swiftlink_gb300 import api, pedigree
from swiftlink_gb300.workloads import disease_probs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from swiftlink_gb300 import build
    build.build()
    port.build()


def half_sibs(wives, markers, seed):
    """A man, a child by each of his wives; his operation, the last, gathers every wife's rfunction."""
    rng = np.random.default_rng(seed)
    N, F, M = 1 + 2 * wives, 1 + wives, markers
    mother = np.array([-1] * F + list(range(1, F)), np.int32)
    father = np.array([-1] * F + [0] * wives, np.int32)
    child, partner, last = 1, 3, 4   # the peel operations' types
    ot = np.array([child] * wives + [partner] * wives + [last], np.int32)
    op = np.array(list(range(F, N)) + list(range(1, F)) + [0], np.int32)
    cut = [np.array([1 + i, 0], np.int32) for i in range(wives)] + [np.array([0], np.int32)] * wives + [np.zeros(0, np.int32)]
    none = np.zeros(0, np.int32)
    prev = [none] * wives + [np.array([i], np.int32) for i in range(wives)] + [np.arange(wives, 2 * wives, dtype=np.int32)]
    ch = [none] * N
    minor = rng.uniform(0.2, 0.5, M)
    theta, partial = pedigree.map_thetas(0.5 * np.arange(M), 5)
    dg = np.zeros((M, N, 2), np.int32)
    dg[:, F:] = np.cumsum(rng.random((M, wives, 2)) < 0.05, axis=0) & 1
    hap = np.zeros((N, 2, M), int)
    hap[:F] = rng.random((F, 2, M)) < minor
    for i in range(F, N):
        for side, parent in ((0, mother[i]), (1, father[i])):
            hap[i, side] = np.where(dg[:, i, side], hap[parent, 1], hap[parent, 0])
    a, b = hap[:, 0], hap[:, 1]
    geno = np.where(a != b, 1, np.where(a == 0, 2, 3)).astype(np.uint8)
    geno[rng.random((N, M)) < 0.3] = 0
    aff, pen = np.ones(N, np.int32), (0.01, 0.8, 0.9)
    return dict(N=N, F=F, M=M, K=N, n_lod=5, mother=mother, father=father, sex=np.array([1] + [2] * wives + [1] * wives, np.int32),
                typed=np.ones(N, np.uint8), genotypes=np.ascontiguousarray(geno.T), minor=minor, theta=theta,
                partial=partial, affection=aff, freq=1e-3, penetrance=pen,
                disease_prob=disease_probs(aff, mother < 0, 1e-3, pen), op_type=ot, op_peel=op, op_cutset=cut, op_prev=prev,
                op_children=ch, dg0=dg)


# 31 previous rfunctions are packed, 32 are not
@pytest.mark.parametrize("wives,packed", [(31, True), (32, False), (40, False)])
def test_equal_to_the_oracle(wives, packed):
    g = half_sibs(wives, 9, wives)
    M, dg = g["M"], g["dg0"]
    prob = api.Problem.from_arrays(g)
    rng = np.random.default_rng(wives)
    u = rng.random((3, M, g["K"] + 2 * g["N"]))
    w = rng.random((3, M * (g["K"] + 2 * g["N"])))
    starts = np.array([0, 4, M - 1], np.int32)
    if not packed:
        with pytest.raises(api.SwiftLinkError):
            api.Context(prob, ls_kernel=api.SL_LS_KERNEL_GENERIC4)
    with api.Context(prob, n_chains=3) as ctx:
        P = port.Port(dict(g, legal=ctx.legal_masks(), trait_prior=ctx.trait_priors()))
        ctx.set_graphs(np.stack([dg] * 3))
        ctx.lsampler_sweep(u, n_chains=3)
        swept = ctx.get_graphs()
        assert (ctx.ls_tuning()[0] == 4) == packed
        ctx.sequential_imputation(starts, w)
        imputed = ctx.get_graphs()
    for c in range(3):
        assert np.array_equal(swept[c], P.lsweep(dg.copy(), u[c]))
        assert np.array_equal(imputed[c], P.si(np.zeros_like(dg), int(starts[c]), w[c])[0])
