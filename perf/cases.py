"""What the framework's speed is measured on: the screens a generation loop
runs, from a trial of 2e5 candidates to the full generation and the twenty
islands, and the surrogate's refit, scoring and gradient calls. Every case
goes through the public entry points (`screen.screen`, `islands.screen_batch`,
`surrogate.*`) as a caller's program uses them: host buffers in and survivors
out for a screen, device tensors for the surrogate.
"""
import math
import os

import numpy as np
import torch

from codec_arena_gb300 import _lib, genome, islands, screen, surrogate, workloads

POP_SEED = os.path.join(workloads.GOLDEN_DIR, "pop_seed_96.txt")
_TC = {"f32": 0, "bf16": _lib.FLAG_TC_BF16, "fp16": _lib.FLAG_TC_FP16}


def listed():
    return [
        # a trial run of the loop: the smallest screen the tests and the smoke run use
        {"name": "screen_trial_2e5", "kind": "screen", "lam": 200_000, "keep": 32, "threads": 4, "ne": 64,
         "elites": "uniform", "nf": 161, "sigma": 0.12, "form": "f32"},
        # the plain CPU-sized screen: 1e6 candidates, a 153-term surface, top 32
        {"name": "screen_1e6", "kind": "screen", "lam": 1_000_000, "keep": 32, "threads": 4, "ne": 64,
         "elites": "uniform", "nf": 153, "sigma": 0.12, "form": "f32"},
        # the reference's `make screen`: its seed population, its committed surrogate, top 192
        {"name": "screen_make_1e8", "kind": "screen", "lam": 100_000_000, "keep": 192, "threads": 4, "ne": 96,
         "elites": "pop", "nf": 161, "sigma": 0.12, "form": "f32"},
        # a later generation of a run after a refit: every linear weight nonzero, sigma decayed, pop / 8
        # elites, an odd budget over an odd number of streams
        {"name": "screen_refit_gen5", "kind": "screen", "lam": 333_333_337, "keep": 192, "threads": 7, "ne": 32,
         "elites": "pop", "nf": 166, "sigma": 0.0835, "form": "f32"},
        # the full generation of one CI shard
        {"name": "screen_generation", "kind": "screen", "lam": 2_650_000_000, "keep": 256, "threads": 4, "ne": 64,
         "elites": "uniform", "nf": 161, "sigma": 0.12, "form": "f32"},
        # the precision form (survivors ranked in FP64), an odd budget
        {"name": "screen_bf16", "kind": "screen", "lam": 1_000_000_007, "keep": 256, "threads": 4, "ne": 64,
         "elites": "uniform", "nf": 161, "sigma": 0.12, "form": "bf16"},
        # a screen on the full 29-gene quadratic surface
        {"name": "screen_full_surface", "kind": "screen", "lam": 265_000_000, "keep": 256, "threads": 4, "ne": 64,
         "elites": "uniform", "nf": 465, "sigma": 0.12, "form": "f32"},
        # twenty islands in one call: budgets log-uniform over 1e8..2.65e9, 16..256 elites each
        {"name": "islands_20", "kind": "islands", "n": 20, "lam_lo": 1e8, "lam_hi": 2.65e9, "plan": 4},
        # the refit after each generation: some thousands of evaluated genomes, the 166 layout, alpha 50
        {"name": "refit_generation", "kind": "refit", "n": 4_999, "ng": 29, "rows": "pop", "alpha": 50.0},
        # the refit over a run's whole table: 400k rows of 16 genes
        {"name": "refit_400k", "kind": "refit", "n": 400_000, "ng": 16, "rows": "uniform", "alpha": 1e-2},
        # a training step on the surrogate: scores, then the gradients of genes and coefficients
        {"name": "score_backward", "kind": "train", "n": 100_003, "ng": 29, "precision": "f32"},
        # gradient-guided mutation of a generation's survivors
        {"name": "mutate_survivors", "kind": "ascend", "n": 5_120, "ng": 29, "eta": 0.01, "steps": 10},
    ]


def _log_int(rng, lo, hi):
    return min(int(hi), max(int(lo), int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["screen", "screen", "screen", "screen", "islands", "refit", "train", "ascend"])
    if kind == "screen":
        elites = rng.choice(["uniform", "pop"])
        nf = rng.choice([153, 159, 161, 164, 165, 166, 166, 465])
        form = "f32" if nf == 465 else rng.choice(["f32", "f32", "f32", "bf16", "fp16"])
        lam = _log_int(rng, 2e5, 6e8 if nf == 465 else 2.65e9)
        return {"kind": kind, "lam": lam, "keep": rng.choice([32, 128, 192, 256, 1000]),
                "threads": rng.choice([1, 2, 4, 4, 7, 16, 64]),
                "ne": rng.randint(16, 96) if elites == "pop" else rng.randint(16, 256), "elites": elites, "nf": nf,
                "sigma": round(0.12 * 0.93 ** rng.randint(0, 20), 4), "form": form}
    if kind == "islands":
        hi = 10 ** rng.uniform(7.5, 8.8)
        return {"kind": kind, "n": rng.randint(2, 20), "lam_lo": hi / 26.5, "lam_hi": hi,
                "plan": rng.randint(0, 99)}
    if kind == "refit":
        return {"kind": kind, "n": _log_int(rng, 300, 400_000), "ng": rng.choice([16, 18, 24, 28, 29, 29]),
                "rows": rng.choice(["pop", "uniform"]), "alpha": rng.choice([1e-2, 1.0, 50.0])}
    if kind == "train":
        return {"kind": kind, "n": _log_int(rng, 256, 400_000), "ng": rng.choice([16, 24, 29]),
                "precision": rng.choice(["f32", "f32", "bf16"])}
    return {"kind": kind, "n": _log_int(rng, 256, 200_000), "ng": rng.choice([16, 29]), "eta": 0.01,
            "steps": rng.randint(1, 20)}


def _elites(kind, ne, seed):
    if kind == "pop":  # a population as a run holds it: the reference's seed genomes, a seeded choice of ne
        pop = genome.load_elites(POP_SEED, v6_fix=True)
        return pop[np.sort(np.random.default_rng(seed).permutation(len(pop))[:ne])]
    return workloads.seeded_elites(ne, seed=seed + 1)


def _weights(nf, seed):
    """A surrogate of the layout: the committed one for 161 (and, with small refitted tail weights, for the
    layouts that extend it), else a seeded N(0, 0.1) one."""
    if nf == 161:
        return workloads.surrogate_161()
    if nf in (164, 165, 166):
        w = workloads.surrogate_161()
        tail = np.random.default_rng(seed).normal(0.0, 0.5, nf - 161).astype(np.float32)
        w = np.concatenate([w[:19], tail, w[19:]])
        w[17:19] += np.float32(0.25)
        return w
    return workloads.seeded_normal_model(seed=seed + 2, n=nf)


def _islands(case):
    """Budgets, keeps and elite counts of a batch."""
    return workloads.seeded_islands(case["n"], seed=case["plan"], lam_lo=case["lam_lo"], lam_hi=case["lam_hi"])


def _rows(kind, n, ng, seed):
    """Evaluated genomes: uniform, or a population's (a seed genome moved a little, 4 decimals, some immigrants)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "uniform":
        return torch.rand((n, ng), generator=gen, device="cuda")
    pop = torch.from_numpy(np.ascontiguousarray(genome.load_elites(POP_SEED, v6_fix=True)["g"])).cuda()
    g = pop[torch.randint(0, pop.shape[0], (n,), generator=gen, device="cuda"), :ng]
    g = g + 0.24 * (torch.rand((n, ng), generator=gen, device="cuda") - 0.5)
    imm = torch.rand((n, 1), generator=gen, device="cuda") < 0.05
    g = torch.where(imm, torch.rand((n, ng), generator=gen, device="cuda"), g)
    return (torch.round(g.clamp(0.0, 1.0) * 10000.0) / 10000.0).contiguous()


def _features(g):
    """[1 | genes | g_i g_j, j <= i < 16] of rows, in the rows' type."""
    ii, jj = torch.tril_indices(16, 16, device=g.device)
    return torch.cat([torch.ones_like(g[:, :1]), g, g[:, ii] * g[:, jj]], dim=1)


def _refit_inputs(case, seed):
    n, ng = case["n"], case["ng"]
    genes = _rows(case["rows"], n, ng, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    nf = 1 + ng + 136
    truth = torch.randn(nf, generator=gen, device="cuda", dtype=torch.float64)
    noise = torch.randn(4, n, generator=gen, device="cuda", dtype=torch.float64)
    t3 = noise[0] / torch.sqrt((noise[1:] ** 2).mean(0))  # Student-t, 3 degrees of freedom
    fit = 0.5 * t3
    for a in range(0, n, 65536):
        fit[a:a + 65536] += _features(genes[a:a + 65536].double()) @ truth
    prior = truth + 0.1 * torch.randn(nf, generator=gen, device="cuda", dtype=torch.float64)
    return genes, fit, prior


def _train_inputs(case, seed):
    n, ng = case["n"], case["ng"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    genes = torch.rand((n, ng), generator=gen, device="cuda")
    coef = torch.randn(1 + ng + 136, generator=gen, device="cuda")
    gout = torch.randn(n, generator=gen, device="cuda")
    return genes, coef, gout


def prepare(case, seed):
    kind = case["kind"]
    if kind == "screen":
        w = _weights(case["nf"], seed)
        model = screen.ModelFull.from_compact(w) if case["nf"] == 465 else screen.Model.from_compact(w)
        cfg = screen.Cfg(case["lam"], case["keep"], 7 + 1_000_003 * seed, threads=case["threads"],
                         sigma=case["sigma"], jump_p=0.02, imm_p=0.01, flags=_TC[case["form"]])
        return {"kind": kind, "cfg": cfg, "model": model, "elites": _elites(case["elites"], case["ne"], seed)}
    if kind == "islands":
        isl = _islands(case)
        return {"kind": kind,
                "cfgs": [screen.Cfg(d["lambda"], d["keep"], d["seed"] + 1000 * seed, threads=d["threads"])
                         for d in isl],
                "models": [screen.Model.from_compact(_weights(153, 100 * seed + i)) for i in range(len(isl))],
                "elites": [_elites("uniform", len(d["elites"]), 100 * seed + i) for i, d in enumerate(isl)]}
    if kind == "refit":
        genes, fit, prior = _refit_inputs(case, seed)
        return {"kind": kind, "genes": genes, "fit": fit, "prior": prior, "alpha": case["alpha"]}
    if kind == "train":
        genes, coef, gout = _train_inputs(case, seed)
        prec = _lib.SG_BF16 if case["precision"] == "bf16" else _lib.SG_FP32
        return {"kind": kind, "genes": genes.requires_grad_(True), "coef": coef.requires_grad_(True), "gout": gout,
                "precision": prec}
    genes, coef, _ = _train_inputs(case, seed)
    return {"kind": kind, "genes": genes, "coef": 0.2 * coef, "eta": case["eta"], "steps": case["steps"]}


def _survivors(surv, screened):
    out = {f: np.ascontiguousarray(surv[f]) for f in ("score", "g", "tribe", "pa", "pb", "stream", "index", "draw")}
    out["screened"] = int(screened)
    return out


def run(state):
    kind = state["kind"]
    if kind == "screen":
        return _survivors(*screen.screen(state["cfg"], state["model"], state["elites"]))
    if kind == "islands":
        res = islands.screen_batch(state["cfgs"], state["models"], state["elites"])
        out = _survivors(np.concatenate([s for s, _ in res]), 0)
        out["screened"] = np.array([n for _, n in res])
        out["kept"] = np.array([len(s) for s, _ in res])
        return out
    if kind == "refit":
        return surrogate.refit(state["genes"], state["fit"], state["prior"], alpha=state["alpha"])
    if kind == "train":
        s = surrogate.score(state["genes"], state["coef"], state["precision"])
        dg, dc = torch.autograd.grad(s, (state["genes"], state["coef"]), state["gout"])
        return {"score": s.detach(), "dgenes": dg, "dcoef": dc}
    new, sc = surrogate.ascend(state["genes"], state["coef"], state["eta"], state["steps"])
    return {"genes": new, "score": sc}


def work(case):
    kind = case["kind"]
    if kind == "screen":  # every candidate judged once by its score's terms; elites in, survivors out
        terms = 465 if case["nf"] == 465 else 153
        return {"bytes": 152 * case["ne"] + 168 * case["keep"] + 4 * case["nf"], "flops": 2 * terms * case["lam"]}
    if kind == "islands":
        lam = sum(d["lambda"] for d in _islands(case))
        return {"bytes": case["n"] * (152 * 128 + 168 * 128 + 612), "flops": 2 * 153 * lam}
    n, ng = case["n"], case["ng"]
    nf = 1 + ng + 136
    if kind == "refit":  # the distinct products of two features and the right side, then the solve
        x = ng - 16
        moments = math.comb(20, 4) + 153 * x + x * (x + 1) // 2
        return {"bytes": n * (4 * ng + 8) + 16 * nf, "flops": 2 * n * (moments + nf) + nf ** 3 // 3}
    if kind == "train":  # score, gene gradient, coefficient gradient
        return {"bytes": n * (8 * ng + 8) + 8 * nf, "flops": 3 * 2 * n * (136 + ng)}
    return {"bytes": n * (8 * ng + 4) + 4 * nf, "flops": case["steps"] * 2 * n * (272 + ng) + 2 * n * (136 + ng)}


_G, _M1, _M2 = np.uint64(0x9E3779B97F4A7C15), np.uint64(0xBF58476D1CE4E5B9), np.uint64(0x94D049BB133111EB)


def _mix(z):
    z = (z ^ (z >> np.uint64(30))) * _M1
    z = (z ^ (z >> np.uint64(27))) * _M2
    return z ^ (z >> np.uint64(31))


def _screen_exact(case, seed):
    """The screen of src/screen.zig:225-343 restated with numpy: the survivors by their f32 scores, and of
    those the genes and scores in 64 bits."""
    w = _weights(case["nf"], seed).astype(np.float32)
    el = _elites(case["elites"], case["ne"], seed)
    E, ne, sig, T = el["g"], len(el), np.float32(case["sigma"]), case["threads"]
    lin = np.zeros(29, np.float32)
    nlin = case["nf"] - 137
    lin[:nlin] = w[1:1 + nlin]
    Q = np.zeros((16, 16), np.float32)
    Q[np.tril_indices(16)] = w[1 + nlin:]
    found = []
    with np.errstate(over="ignore"):
        for t in range(T):
            my = case["lam"] // T if t < T - 1 else case["lam"] - (T - 1) * (case["lam"] // T)
            st = np.uint64(7 + 1_000_003 * seed) ^ (_G * np.uint64(t + 1))
            z = _mix(st + _G * np.arange(1, 64 * my + 65, dtype=np.uint64))
            u24 = (z >> np.uint64(40)).astype(np.uint32)
            imm_thr, jump_thr = (math.ceil(float(np.float32(p)) * 2.0 ** 24) for p in (0.01, 0.02))
            imm_at, jump_at = (u24 < imm_thr), (u24 < jump_thr)
            pos, p = np.empty(my, np.int64), 0
            imm_b, jump_b = imm_at.tobytes(), jump_at.tobytes()
            for i in range(my):
                pos[i] = p
                n = 32 if imm_b[p + 2] else 61
                p += n + (3 if jump_b[p + n] else 1)
            imm = imm_at[pos + 2]
            pa, pb = ((z[pos + q] >> np.uint64(32)) % np.uint64(ne) for q in (0, 1))
            at = pos + np.where(imm, 32, 61)
            jump = jump_at[at]
            jg, jv = (z[at + jump] >> np.uint64(32)) % np.uint64(29), u24[at + 2 * jump]
            best = np.empty(my, np.float32)
            for a in range(0, my, 100_000):
                s = slice(a, min(my, a + 100_000))
                g = _genes(z, u24, pos[s], imm[s], pa[s], pb[s], jump[s], jg[s], jv[s], E, sig, np.float32)
                best[s] = _score_f32(g, w[0], lin, Q)
            for i in np.lexsort((np.arange(my), -best))[:case["keep"]]:
                one = [x[i:i + 1] for x in (pos, imm, pa, pb, jump, jg, jv)]
                g64 = _genes(z, u24, *one, E, sig, np.float64)[0]
                f = 16.0 * float(w[0]) + g64 @ lin.astype(float) + g64[:16] @ Q.astype(float) @ g64[:16]
                found.append((-float(best[i]), t, i, f, g64))
    found.sort(key=lambda r: r[:3])
    found = found[:case["keep"]]
    return {"score": np.array([r[3] for r in found]), "g": np.array([r[4] for r in found]), "tribe": None, "pa": None,
            "pb": None, "stream": None, "index": None, "draw": None, "screened": None}


def _genes(z, u24, pos, imm, pa, pb, jump, jg, jv, E, sig, dt):
    k = np.arange(29)
    bit = (z[pos[:, None] + 3 + 2 * k] & np.uint64(1)).astype(bool)
    u = u24[pos[:, None] + np.where(imm[:, None], 3 + k, 4 + 2 * k)].astype(dt) * dt(2.0 ** -24)
    par = np.where(bit, E[pb.astype(np.int64)], E[pa.astype(np.int64)]).astype(dt)
    g = np.where(imm[:, None], u, np.clip(par + (u - dt(0.5)) * dt(2) * dt(sig), dt(0), dt(1)))
    r = np.nonzero(jump)[0]
    g[r, jg[r].astype(np.int64)] = jv[r].astype(dt) * dt(2.0 ** -24)
    return g


def _score_f32(g, w0, lin, Q):
    lanes = []
    for j in range(16):
        acc = np.zeros(len(g), np.float32)
        for i in range(j, 16):
            acc = acc + Q[i, j] * (g[:, j] * g[:, i])
        lanes.append((w0 + lin[j] * g[:, j]) + acc)
    r = lanes[0]
    for j in range(1, 16):
        r = r + lanes[j]
    tail = np.zeros(len(g), np.float32)
    for j in range(16, 29):
        tail = tail + lin[j] * g[:, j]
    return r + tail


def exact(case, seed):
    kind = case["kind"]
    if kind == "screen":  # larger ones would take minutes on the host
        return _screen_exact(case, seed) if case["lam"] <= 1_000_000 and case["nf"] != 465 and \
            case["form"] == "f32" else None
    if kind == "islands":
        return None
    if kind == "refit":
        genes, fit, prior = _refit_inputs(case, seed)
        n, nf, alpha = case["n"], prior.numel(), case["alpha"]
        gram = alpha * torch.eye(nf, dtype=torch.float64, device="cuda")
        for a in range(0, n, 32768):
            phi = _features(genes[a:a + 32768].double())
            gram += phi.T @ phi
        chol = torch.linalg.cholesky(gram)
        w = prior.clone()
        for _ in range(4):  # Newton steps on the residual: the error of the normal equations drops out
            r = alpha * (prior - w)
            for a in range(0, n, 32768):
                phi = _features(genes[a:a + 32768].double())
                r += phi.T @ (fit[a:a + 32768] - phi @ w)
            w = w + torch.cholesky_solve(r[:, None], chol)[:, 0]
        return w
    if kind == "train":
        genes, coef, gout = _train_inputs(case, seed)
        go, dc = gout.double(), _features(genes.double()).T @ gout.double()  # the features unrounded in both
        if case["precision"] == "bf16":
            genes, coef = genes.bfloat16(), coef.bfloat16()
        g, c = genes.double().requires_grad_(True), coef.double()
        s = _features(g) @ c
        (dg,) = torch.autograd.grad(s, g, go)
        return {"score": s.detach(), "dgenes": dg, "dcoef": dc}
    genes, coef, _ = _train_inputs(case, seed)
    g, c = genes.double(), (0.2 * coef).double()
    for _ in range(case["steps"]):
        x = g.detach().requires_grad_(True)
        (d,) = torch.autograd.grad((_features(x) @ c).sum(), x)
        g = (g + case["eta"] * d).clamp(0.0, 1.0)
    return {"genes": g, "score": _features(g) @ c}
