"""Measured cases: the work a linkage analysis has the library do, through
`swiftlink_gb300.api`, from one small family to a 400-member pedigree.

A case is a dict of plain values:

  kind      "run"     sl_run: MCMC of `chains` replicate chains, scored every
                      `period` iterations (0: burn-in, nothing scored); with
                      `batch` pedigrees of uneven sizes, one sl_batch_run with
                      MC3 exchanges
            "impute"  sl_sequential_imputation_run: legal starting graphs
            "score"   sl_lod_score_graphs: stored graphs scored
            "adjoint" sl_trait_backward: gradients of the trait peel
  members, generations, loops, affected, pedigree (the topology's seed)
  markers, untyped (share of the founders with no genotypes at all), model
  and the numbers of chains, graphs, iterations of the kind.

The pedigrees, maps and models are those of the synthetic configurations
(synth.CONFIGS, synth.uneven_batch) and of shapes between them.  The
pedigree's topology, disease statuses and peel sequence belong to the case;
the genotypes, graphs and draws follow from the seed.
"""
import math
from functools import lru_cache

import numpy as np
import torch

from swiftlink_gb300 import api, pedigree, synth
from swiftlink_gb300.workloads import disease_probs, position_bytes, step_bytes

# (penetrance of 0, 1, 2 disease alleles), disease-allele frequency
MODELS = {"recessive": ((0.0, 0.0, 1.0), 1e-4), "dominant": ((0.01, 0.8, 0.9), 1e-3)}
N_LOD = 5                     # LOD positions per interval, the program's default
MAF = (0.05, 0.5)
MISSING = 0.05                # share of single genotypes missing, as in the configurations
TEMPER = 0.3                  # MC3: chain j of C at temperature TEMPER^(j / (C - 1))


def listed():
    small = dict(members=30, generations=4, loops=1, affected=5, pedigree=1, markers=200, spacing=0.5, untyped=0.0,
                 model="recessive")
    mid = dict(members=120, generations=6, loops=3, affected=35, pedigree=2, markers=2000, spacing=0.2, untyped=0.0,
               model="recessive")
    large = dict(members=400, generations=8, loops=10, affected=60, pedigree=5, markers=10000, spacing=0.1,
                 untyped=0.0, model="recessive")
    fast = dict(kind="run", precision="fast", batch=1, lprob=0.5)
    return [
        # one small family, one chain: every launch counts
        dict(small, **fast, name="run 30x200 c1", chains=1, iterations=10, period=5),
        # the same family in the reference's FP64 arithmetic (the program's -E)
        dict(small, **dict(fast, precision="exact"), name="run exact 30x200 c2", chains=2, iterations=4, period=2),
        # the program's ordinary run: a large family, replicate chains, L- and M-sweeps mixed, graphs scored
        dict(mid, **fast, name="run 120x2000 c10", chains=10, iterations=10, period=5),
        # burn-in with its two sweeps apart: locus sampler only, meiosis sampler only
        dict(mid, **dict(fast, lprob=1.0), name="lsweep 120x2000 c10", chains=10, iterations=8, period=0),
        dict(mid, **dict(fast, lprob=0.0), name="msweep 120x2000 c10", chains=10, iterations=4, period=0),
        # the same on the largest pedigree that the configurations hold, dense map
        dict(large, **dict(fast, lprob=1.0), name="lsweep 400x10000 c8", chains=8, iterations=4, period=0),
        dict(large, **dict(fast, lprob=0.0), name="msweep 400x10000 c8", chains=8, iterations=2, period=0),
        # a batch of uneven pedigrees, some founders untyped, MC3 chains with exchanges, odd marker count
        dict(small, **fast, name="batch mc3 6x301 c8", members=100, generations=5, loops=2, affected=10, pedigree=11,
             markers=301, untyped=0.2) | dict(batch=6, chains=8, iterations=10, period=5),
        # starting graphs by sequential imputation (the program's -s passes)
        dict(mid, name="impute 120x301", kind="impute", precision="fast", markers=301, chains=4, passes=250),
        # stored graphs scored in the batched FP32 form, and in the plain FP64 form on a smaller family
        dict(mid, name="score fp32 120x2000 g32", kind="score", lod="fp32", graphs=32),
        dict(small, name="score fp64 45x401 g4", kind="score", lod="fp64", graphs=4, members=45, affected=6,
             pedigree=3, markers=401, model="dominant"),
        # gradients for fitting the disease model
        dict(mid, name="adjoint 120x2000 g16", kind="adjoint", graphs=16, model="dominant"),
    ]


def draw(rng):
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["run", "run", "run", "impute", "score", "adjoint"])
    n = log(24, 400 if kind == "run" else 130)
    big = n > 150
    gens = 3 + (n >= 40) + (n >= 90) + (n >= 200) + (n >= 300)
    c = dict(kind=kind, members=n, generations=gens, loops=rng.randint(0, 3 if gens > 3 else 1), affected=max(2, n // 10),
             pedigree=rng.randrange(1 << 20), markers=log(60, 1200 if big else 2200),
             spacing=rng.choice([0.1, 0.2, 0.5]), untyped=0.0 if n > 100 else rng.choice([0.0, 0.0, 0.2]),
             model=rng.choice(sorted(MODELS)))
    if kind == "run":
        exact = n <= 60 and rng.random() < 0.25
        c |= dict(precision="exact" if exact else "fast", batch=1, lprob=rng.choice([0.0, 0.5, 1.0]),
                  chains=log(1, 3 if exact else 12), iterations=2 if exact else 4)
        # pedigrees whose compiled scorer takes long to build: burn-in
        c["period"] = 0 if n > 130 else rng.choice([0, 2])
        if exact:
            c["markers"] = min(c["markers"], 300)
        elif n <= 100 and rng.random() < 0.3:
            c |= dict(batch=rng.randint(2, 5), markers=min(c["markers"], 500), lprob=0.5, chains=rng.randint(2, 8), period=2)
    elif kind == "impute":
        c |= dict(precision="fast", markers=log(60, 400), chains=rng.randint(1, 6), passes=log(8, 250))
    elif kind == "score":
        fp64 = n <= 60 and rng.random() < 0.4
        c |= dict(lod="fp64" if fp64 else "fp32", graphs=log(1, 4 if fp64 else 32), markers=min(c["markers"], 500 if fp64 else 2000))
        if fp64:
            c["model"] = "dominant"
    else:
        c |= dict(graphs=log(1, 12), model="dominant", markers=min(c["markers"], 2000))
    return c


# ---- pedigrees ---------------------------------------------------------------


@lru_cache(maxsize=64)
def _family(members, generations, loops, affected, seed, spacing, markers, model):
    """A pedigree's workload without its genotypes' seed: topology, statuses, map."""
    pen, q = MODELS[model]
    for k in range(40):
        # a shape that the topology builder cannot reach is tried again with one loop or one generation fewer
        spec = synth.WorkloadSpec(n_members=members, generations=max(3, generations - k // 12), loops=max(0, loops - k // 6),
                                  affected=affected, markers=2, spacing_cm=spacing, maf=MAF, penetrance=pen,
                                  disease_freq=q, disease_cm=0.9 * spacing)
        try:
            w = synth.make_workload(1, seed=1000 * seed + k, spec=spec)
            break
        except RuntimeError:
            continue
    else:
        raise RuntimeError("no pedigree of this shape")
    w.marker_cm = spacing * (np.arange(markers) + 0.5)
    order = [i for i, p in enumerate(w.persons) if p.founder] + [i for i, p in enumerate(w.persons) if not p.founder]
    at = {w.persons[k].pid: i for i, k in enumerate(order)}
    mother = np.array([at[w.persons[k].mother] if w.persons[k].mother else -1 for k in order], np.int32)
    father = np.array([at[w.persons[k].father] if w.persons[k].father else -1 for k in order], np.int32)
    sex = np.array([w.persons[k].sex for k in order], np.int32)
    affection = np.array([w.persons[k].affection for k in order], np.int32)
    theta, partial = pedigree.map_thetas(w.marker_cm, N_LOD)
    ot, op, cut, prev, ch = api.peel_sequence(mother, father)
    return dict(N=len(order), F=int((mother < 0).sum()), mother=mother, father=father, sex=sex, affection=affection,
                theta=theta, partial=partial, freq=q, penetrance=pen,
                disease_prob=disease_probs(affection, mother < 0, q, pen),
                op_type=ot, op_peel=op, op_cutset=cut, op_prev=prev, op_children=ch)


def _families(case):
    """The case's pedigrees: one, or a batch of uneven sizes."""
    n = case.get("batch", 1)
    out = []
    for k in range(n):
        m = case["members"] if n == 1 else max(24, case["members"] * (k + 1) // n)
        gens = case["generations"] if n == 1 else min(case["generations"], 3 + (m >= 40) + (m >= 90))
        out.append(_family(m, gens, case["loops"] if gens > 3 else min(1, case["loops"]), case["affected"] if n == 1 else max(2, m // 10),
                           case["pedigree"] + k, case["spacing"], case["markers"], case["model"]))
    return out


def _inheritance(rng, fam, markers, copies):
    """Meiosis indicators [copies][markers][N][2] of gene drops along the map (founders 0)."""
    N, F = fam["N"], fam["F"]
    bits = np.zeros((copies, markers, N, 2), np.int32)
    start = rng.random((copies, 1, N - F, 2)) < 0.5
    cross = rng.random((copies, markers - 1, N - F, 2), dtype=np.float32) < fam["theta"][None, :, None, None]
    steps = np.concatenate([start, cross], 1)
    bits[:, :, F:] = np.logical_xor.accumulate(steps, axis=1)
    return bits


def _problem(rng, fam, markers, untyped):
    """The pedigree's tables with genotypes dropped from the seed, and the drop's own legal graph [markers][N][2]."""
    N, F = fam["N"], fam["F"]
    minor = rng.uniform(MAF[0], MAF[1], size=markers)
    dg = _inheritance(rng, fam, markers, 1)[0]
    hap = np.zeros((N, 2, markers), np.int8)
    hap[:F] = rng.random((F, 2, markers), dtype=np.float32) < minor
    todo = list(range(F, N))
    done = set(range(F))
    while todo:
        left = []
        for i in todo:
            if fam["mother"][i] in done and fam["father"][i] in done:
                for side, parent in ((0, fam["mother"][i]), (1, fam["father"][i])):
                    hap[i, side] = np.where(dg[:, i, side], hap[parent, 1], hap[parent, 0])
                done.add(i)
            else:
                left.append(i)
        todo = left
    a, b = hap[:, 0], hap[:, 1]
    geno = np.where(a != b, 1, np.where(a == 0, 2, 3)).astype(np.uint8)
    geno[rng.random((N, markers), dtype=np.float32) < MISSING] = 0
    geno[rng.permutation(F)[:int(round(untyped * F))]] = 0
    p = dict(fam, M=markers, n_lod=N_LOD, genotypes=np.ascontiguousarray(geno.T), minor=minor,
             typed=(geno != 0).any(axis=1).astype(np.uint8))
    return api.Problem.from_arrays(p), dg


# ---- a pass ------------------------------------------------------------------


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    fams = _families(case)
    s = {"case": case, "seed": 1 + seed, "ctx": [], "dg": []}
    M = case["markers"]
    for fam in fams:
        prob, dg = _problem(rng, fam, M, case["untyped"])
        opt = dict(n_chains=case.get("chains", 1), lod_flags=api.SL_LOD_ZERO_OK)
        if case["kind"] == "run" and case["precision"] == "exact":
            # the plain FP64 peel may underflow to a zero term on larger families, as the reference's does
            opt |= dict(sampler_precision=api.SL_SAMPLER_EXACT, lod_precision=api.SL_LOD_FP64)
        elif case.get("lod") == "fp64" or case["kind"] == "adjoint":
            opt |= dict(sampler_precision=api.SL_SAMPLER_FAST, lod_precision=api.SL_LOD_FP64)
        else:
            # the program's choice of scorer: the form compiled for the pedigree; the batch's pedigrees are scored
            # by the interpreter, and nothing is compiled where nothing is scored
            jit = case["kind"] == "score" or (case["kind"] == "run" and case["period"] > 0 and len(fams) == 1)
            opt |= dict(sampler_precision=api.SL_SAMPLER_FAST, lod_precision=api.SL_LOD_FP32_RESCALED,
                        lod_kernel=api.SL_LOD_KERNEL_JIT_REG if jit else api.SL_LOD_KERNEL_INTERP)
        ctx = api.Context(prob, **opt)
        s["ctx"].append(ctx)
        if case["kind"] == "run":
            C = case["chains"]
            s["dg"].append(np.ascontiguousarray(np.broadcast_to(dg, (C,) + dg.shape)))
            if len(fams) > 1:
                ctx.set_temperatures(TEMPER ** (np.arange(C) / max(1, C - 1)))
        elif case["kind"] in ("score", "adjoint"):
            s["dg"].append(_inheritance(rng, fam, M, case["graphs"]))
            if case["kind"] == "adjoint":
                # a fixed form, so that results do not depend on a timing; the compiled one up to 4-member cutsets
                widest = max(len(c) for c in fam["op_cutset"])
                ctx.adjoint_set_form(api.SL_ADJOINT_SPECIALISED if widest <= 4 else api.SL_ADJOINT_THREAD)
    if len(fams) > 1:
        s["batch"] = api.Batch(s["ctx"])
    s["out"] = [np.empty_like(d) for d in s["dg"]] if case["kind"] == "run" else []
    return s


def run(s):
    case, out = s["case"], {}
    if case["kind"] == "run":
        for ctx, dg in zip(s["ctx"], s["dg"]):
            ctx.set_graphs(dg)
            ctx.lod_reset()
        o = dict(lprob=case["lprob"], seed=s["seed"])
        o |= (dict(iterations=case["iterations"], period=case["period"]) if case["period"]
              else dict(iterations=0, burnin=case["iterations"]))
        if "batch" in s:
            s["batch"].run(exchange_period=case["period"], **o)
        else:
            s["ctx"][0].run(**o)
        for k, (ctx, g) in enumerate(zip(s["ctx"], s["out"])):
            if case["period"]:
                raw, count, tp = ctx.lod_results()
                out["lod%d" % k], out["count%d" % k], out["trait%d" % k] = raw, int(count), tp
            out["graphs%d" % k] = ctx.get_graphs(out=g)
    elif case["kind"] == "impute":
        ctx = s["ctx"][0]
        out["weights"] = ctx.sequential_imputation_run(case["passes"], seed=s["seed"])
        out["graphs"] = ctx.get_graphs()
    elif case["kind"] == "score":
        ctx = s["ctx"][0]
        ctx.lod_reset()
        ctx.lod_score_graphs(s["dg"][0])
        raw, count, tp = ctx.lod_results()
        out = {"lod": raw, "count": int(count), "trait": tp}
    else:
        grad, ptrait = s["ctx"][0].trait_backward(s["dg"][0])
        out = {"grad": grad, "ptrait": ptrait}
    return out


def work(case):
    """What a pass cannot do without.  Bytes: the caller's graphs read and
    written as 32-bit indicators, the 2-bit genotypes, packed indicators and
    map of every sweep, the scored positions.  Operations: a few per member
    (or allowed rfunction cell) at each locus and sweep, or per scored position."""
    M, npos = case["markers"], (case["markers"] - 1) * N_LOD
    b = f = 0.0
    for fam in _families(case):
        N, F = fam["N"], fam["F"]
        K = len(fam["op_type"])
        graph = 8.0 * M * N
        cells = sum(4.0 ** (len(c) + 1) for c in fam["op_cutset"])   # a trait peel's terms over every state
        if case["kind"] == "run":
            C, it = case["chains"], case["iterations"]
            scored = C * (-(-it // case["period"])) if case["period"] else 0
            b += C * (2 * graph + it * step_bytes(N, F, M)) + scored * npos * position_bytes(N, F, N_LOD)
            # an L-sweep: two passes over the peel, about two allowed cells of two states each, four factors a term
            l_sweep = 2.0 * M * K * 2 * 2 * 4
            # an M-sweep: at every meiosis and locus a likelihood over the founder alleles, and a 2x2 filter step
            m_sweep = 2.0 * (N - F) * M * (2 * F + 20)
            f += C * it * (case["lprob"] * l_sweep + (1 - case["lprob"]) * m_sweep) + scored * npos * 3 * cells
        elif case["kind"] == "impute":
            n = case["chains"] * case["passes"]
            b += case["chains"] * graph + n * step_bytes(N, F, M)
            f += n * 2.0 * M * K * 2 * 2 * 4
        elif case["kind"] == "score":
            b += case["graphs"] * (graph + npos * position_bytes(N, F, N_LOD))
            f += case["graphs"] * npos * 3 * cells
        else:
            b += case["graphs"] * (graph + npos * 6 * 8)
            f += case["graphs"] * npos * 9 * cells
    return {"bytes": b, "flops": f}


# ---- the trait peel in 64 bits -----------------------------------------------


def _transmission(mat, pat):
    """[..., mother state, father state, child state]: a child's transmission term given its recombination
    factors mat, pat [..., 2] by grandparental origin; states UU, AA, AU, UA (maternal allele first)."""
    first, second = [0, 1, 1, 0], [0, 1, 0, 1]   # a state's maternal and paternal allele
    parts = []
    for m in range(4):
        for p in range(4):
            for kid in range(4):
                v = 0.0
                for i in range(2):
                    for j in range(2):
                        if (first[m], second[m])[i] == first[kid] and (first[p], second[p])[j] == second[kid]:
                            v = v + 0.25 * mat[..., i] * pat[..., j]
                parts.append(v if torch.is_tensor(v) else torch.zeros_like(mat[..., 0]))
    return torch.stack(parts, -1).reshape(mat.shape[:-1] + (4, 4, 4))


def _log_likelihood(fam, state, trans):
    """log of the sum over everybody's states of prod state[person] * trans[person], by variable elimination;
    state: [N] of [P, 4]; trans: {child: [P, 4, 4, 4]}."""
    factors = [((i,), t) for i, t in enumerate(state)]
    factors += [((int(fam["mother"][i]), int(fam["father"][i]), i), t) for i, t in trans.items()]
    left = set(range(fam["N"]))
    log = torch.zeros_like(state[0][:, 0])
    while left:
        def scope(v):
            return set().union(*(f[0] for f in factors if v in f[0])) - {v}
        v = min(left, key=lambda x: (len(scope(x)), x))
        use = [f for f in factors if v in f[0]]
        factors = [f for f in factors if v not in f[0]]
        dims = sorted(set().union(*(f[0] for f in use)), key=lambda x: (x == v, x))
        prod = None
        for names, t in use:
            order = [n for n in dims if n in names]
            t = t.permute([0] + [1 + names.index(n) for n in order])
            t = t.reshape([t.shape[0]] + [4 if n in names else 1 for n in dims])
            prod = t if prod is None else prod * t
        prod = prod.expand([-1] + [4] * len(dims)).sum(-1)
        top = prod.detach().reshape(len(log), -1).amax(1)
        top = torch.where(top > 0, top, torch.ones_like(top))
        log = log + top.log()
        factors.append((tuple(dims[:-1]), prod / top.reshape([-1] + [1] * (len(dims) - 1))))
        left.remove(v)
    for _, t in factors:
        log = log + t.reshape(log.shape[0]).log()
    return log


def exact(case, seed):
    if case["kind"] not in ("score", "adjoint"):
        return None        # samples: whole numbers, and tables of the graphs they led to
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.default_rng([seed, 77])
    fam = _families(case)[0]
    N, F, M = fam["N"], fam["F"], case["markers"]
    _problem(rng, fam, M, case["untyped"])
    dgs = _inheritance(rng, fam, M, case["graphs"])
    f8 = lambda x: torch.as_tensor(np.asarray(x, np.float64), device=dev)  # noqa: E731
    npos = (M - 1) * N_LOD
    interval = torch.arange(npos, device=dev) // N_LOD
    offset = torch.arange(npos, device=dev) % N_LOD + 1
    partial = f8(fam["partial"])
    with_grad = case["kind"] == "adjoint"

    def states(pen, q, n):
        """A person's state terms [n, 4] from the penetrances [n, 3] and the allele frequency [n]."""
        out = []
        dose = [0, 2, 1, 1]
        for i in range(N):
            cols = []
            for v in range(4):
                t, aff = dose[v], fam["affection"][i]
                prior = ((1 - q) ** 2, q * (1 - q), q * q)[t]
                p = pen[:, t]
                if i < F:
                    cols.append(prior * p if aff == 2 else prior * (1 - p) if aff == 1 else prior)
                else:
                    cols.append(p if aff == 2 else 1 - p if aff == 1 else torch.full_like(p, 0.25))
            out.append(torch.stack(cols, -1).expand(n, 4))
        return out

    def leaf(x):
        return x.clone().requires_grad_(with_grad)

    plain = torch.full((1, 2), 1.0, dtype=torch.float64, device=dev)
    pen0, q0 = leaf(f8(fam["penetrance"])[None]), leaf(f8([fam["freq"]]))
    t0 = _transmission(plain, plain)
    trait = _log_likelihood(fam, states(pen0, q0, 1), {i: t0 for i in range(F, N)})
    raw, grads = None, []
    for g in range(case["graphs"]):
        bits = torch.as_tensor(dgs[g], device=dev)
        th = leaf(partial[interval] * offset)
        th2 = leaf(partial[interval] * (N_LOD + 1 - offset))
        pen = leaf(f8(fam["penetrance"])[None].expand(npos, 3))
        q = leaf(f8([fam["freq"]]).expand(npos))
        trans = {}
        for i in range(F, N):
            rec = []
            for side in range(2):
                left, right = bits[:-1, i, side][interval], bits[1:, i, side][interval]
                rec.append(torch.stack([torch.where(left == o, 1 - th, th) * torch.where(right == o, 1 - th2, th2)
                                        for o in range(2)], -1))
            trans[i] = _transmission(rec[0], rec[1])
        logl = _log_likelihood(fam, states(pen, q, npos), trans)
        if with_grad:
            d = torch.autograd.grad(logl.sum(), [th, th2, pen, q])
            grads.append(torch.cat([d[0][:, None], d[1][:, None], d[2], d[3][:, None]], 1).reshape(M - 1, N_LOD, 6))
            continue
        cross = (bits[1:, F:] != bits[:-1, F:]).sum((1, 2)).double()
        th_m = f8(fam["theta"])
        marker = cross * th_m.log() + (2 * (N - F) - cross) * (1 - th_m).log()
        v = logl - marker[interval] - math.log(0.5) * 2 * (N - F)
        raw = v if raw is None else torch.logaddexp(raw, v)
    if with_grad:
        d = torch.autograd.grad(trait.sum(), [pen0, q0])
        return {"grad": torch.stack(grads).cpu().numpy(), "ptrait": torch.cat([d[0][0], d[1]]).cpu().numpy()}
    return {"lod": raw.cpu().numpy(), "count": None, "trait": float(trait[0])}
