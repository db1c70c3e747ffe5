"""Timed cases of the framework's main paths, through its public entry points.

Each case is a dict of plain values with a ``kind``:

  gw_call    gwldcore.gw_ldscore: a whole genome-wide estimate in one call from host BED rows
  gw_plan    GwSession.plan: a genome-wide (partitioned) estimate on a resident image
  win_plan   WinPlan: a windowed + partitioned estimate on a resident image
  win_call   session.windowed_ldscore: the windowed estimate in one call from pinned host BED rows
  blocks     the per-block drop-in calls (phase 1 over all SNP blocks, then phase 2) on a BED fileset
  window_ld  GwSession.window_ld: exact windowed LD scores on a resident image
  gxe        GxeReference.run: a multi-environment GxE reference on a resident image
  two_pass   generalized_gxe.two_pass: the generalized per-variant GxE estimator
  surrogate  Surrogate.forward over all rows and Surrogate.loss_grad over one mini-batch

Genotypes are hard calls with p ~ U[0.05, 0.5], autocorrelation 0.9 between
neighbours inside blocks of 32 SNPs, and 1 % missing calls; annotations are
Bernoulli(0.1) (one all-ones column when K = 1).  ``exact`` restates every
estimate densely in FP64 torch.
"""
import math
import tempfile

import numpy as np
import torch

M64 = (1 << 64) - 1


def listed():
    return [
        # the smallest whole call: a pilot of a few hundred probes' work, latency and launches
        {"name": "gw_call small", "kind": "gw_call", "n": 1003, "m": 2001, "k": 2, "b": 24,
         "step": 200, "impute": "mean"},
        # the plain genome-wide configuration (N = 5,000, M = 20,000, B = 20)
        {"name": "gw_plan 5k x 20k", "kind": "gw_plan", "n": 5000, "m": 20000, "k": 1, "b": 20,
         "step": 1000, "impute": "mean"},
        # annotation-partitioned genome-wide scores at the windowed configuration's N, K and B
        {"name": "gw_plan 50k x 40k K24", "kind": "gw_plan", "n": 50000, "m": 40000, "k": 24,
         "b": 50, "step": 2000, "impute": "mean"},
        # a biobank's sample count (ragged), few SNPs: long sample reductions, one bin
        {"name": "gw_plan 200k x 16k", "kind": "gw_plan", "n": 200003, "m": 16001, "k": 1, "b": 50,
         "step": 1000, "impute": "mean"},
        # the windowed + partitioned headline configuration, a chromosome's worth of SNPs
        {"name": "win_plan 50k x 60k K24", "kind": "win_plan", "n": 50000, "m": 60000, "k": 24,
         "b": 50, "step": 1000, "impute": "mean"},
        # ragged sizes, HWE-completed genotypes, the few probes of a control-variate run
        {"name": "win_plan 10k x 20k hwe", "kind": "win_plan", "n": 10007, "m": 20011, "k": 6,
         "b": 10, "step": 500, "impute": "hwe"},
        # the one-call windowed estimate from host rows, upload included
        {"name": "win_call 20k x 40k", "kind": "win_call", "n": 20000, "m": 40000, "k": 10, "b": 20,
         "step": 1000, "impute": "mean"},
        # what the reference's driver calls block by block (its default imputation)
        {"name": "blocks 5k x 4k", "kind": "blocks", "n": 5000, "m": 4000, "k": 2, "b": 20,
         "step": 1000, "impute": "hwe", "dtype": "float64"},
        # exact windowed scores, 1 Mb windows at 1 SNP per 500 bp
        {"name": "window_ld 50k x 12k", "kind": "window_ld", "n": 50000, "m": 12000, "k": 3,
         "reach": 2000, "impute": "mean"},
        # a GxE reference over 4 exposures
        {"name": "gxe 20k x 20k E4", "kind": "gxe", "n": 20000, "m": 20000, "e": 4, "b": 32,
         "impute": "mean"},
        # the two-pass estimator with an intercept and a covariate projected out
        {"name": "two_pass 4k x 6k", "kind": "two_pass", "n": 4000, "m": 6000, "q": 2, "r": 2,
         "k": 2, "b": 16, "impute": "mean"},
        # the control variate's network: inference on every SNP, one training mini-batch
        {"name": "surrogate 100k", "kind": "surrogate", "rows": 100003, "batch": 4096, "k": 24},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["gw_call", "gw_plan", "gw_plan", "win_plan", "win_plan", "win_call",
                       "blocks", "window_ld", "gxe", "two_pass", "surrogate"])
    impute = rng.choice(["mean", "mean", "hwe"])
    if kind == "gw_call":
        return {"kind": kind, "n": size(500, 3000), "m": size(1000, 5000), "k": rng.randint(1, 4),
                "b": rng.randint(8, 50), "step": size(100, 1000), "impute": impute}
    if kind in ("gw_plan", "win_plan"):
        n, k, b = size(5000, 200000), rng.choice([1, 2, 5, 10, 24]), rng.randint(8, 50)
        cap = 2.2e12 / (n * (k if kind == "gw_plan" else max(k, 4)) * b)
        lo = 2000 if kind == "gw_plan" else 4000
        return {"kind": kind, "n": n, "m": size(lo, max(lo + 1, min(60000, cap, 3.3e9 / n))),
                "k": k, "b": b, "step": size(200, 2000), "impute": impute}
    if kind == "win_call":
        return {"kind": kind, "n": size(5000, 30000), "m": size(5000, 40000),
                "k": rng.randint(1, 10), "b": rng.randint(8, 30), "step": size(200, 2000),
                "impute": impute}
    if kind == "blocks":
        return {"kind": kind, "n": size(1000, 8000), "m": size(1000, 5000), "k": rng.randint(1, 4),
                "b": rng.randint(8, 30), "step": size(300, 2000), "impute": impute,
                "dtype": rng.choice(["float64", "float32"])}
    if kind == "window_ld":
        return {"kind": kind, "n": size(5000, 60000), "m": size(2000, 12000),
                "k": rng.randint(1, 24), "reach": size(100, 2000), "impute": impute}
    if kind == "gxe":
        return {"kind": kind, "n": size(5000, 30000), "m": size(2000, 20000), "e": rng.randint(1, 4),
                "b": rng.randint(8, 40), "impute": "mean"}
    if kind == "two_pass":
        return {"kind": kind, "n": size(1000, 5000), "m": size(1000, 7000), "q": rng.randint(1, 3),
                "r": rng.randint(0, 3), "k": rng.randint(1, 3), "b": rng.randint(4, 16),
                "impute": "mean"}
    return {"kind": kind, "rows": size(1000, 200000), "batch": size(512, 8192),
            "k": rng.randint(1, 24)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def bed_rows(case, seed):
    """Packed SNP-major rows (M x ceil(N/4) uint8, on the device)."""
    n, m = case["n"], case["m"]
    p = 0.05 + 0.45 * np.random.default_rng([seed, 1]).random(m)
    q0 = torch.special.ndtri(torch.from_numpy((1 - p) ** 2)).float().cuda()
    q1 = torch.special.ndtri(torch.from_numpy(1 - p * p)).float().cuda()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    blocks, nb = -(-m // 32), -(-n // 4)
    out = torch.zeros((blocks * 32, nb), dtype=torch.uint8, device="cuda")
    z = None
    for t in range(32):
        e = torch.randn((blocks, n), generator=gen, device="cuda")
        z = e if z is None else z.mul_(0.9).add_(e, alpha=math.sqrt(1 - 0.81))
        have = -(-(m - t) // 32)   # blocks whose SNP t exists
        g = (z[:have] > q0[t::32, None]).to(torch.uint8)
        g += g & (z[:have] > q1[t::32, None]).to(torch.uint8)
        code = torch.where(g > 0, g + 1, g)          # 0, 2, 3 for 0, 1, 2 copies
        miss = torch.rand((have, n), generator=gen, device="cuda") < 0.01
        code[miss] = 1
        quad = torch.zeros((have, nb * 4), dtype=torch.uint8, device="cuda")
        quad[:, :n] = code
        quad = quad.view(have, nb, 4)
        out[t::32][:have] = quad[:, :, 0] | quad[:, :, 1] << 2 | quad[:, :, 2] << 4 | quad[:, :, 3] << 6
    return out[:m].contiguous()


def annotations(case, seed):
    m, k = case["m"], case["k"]
    if k == 1:
        return np.ones((m, 1))
    a = (np.random.default_rng([seed, 2]).random((m, k)) < 0.1).astype(np.float64)
    a[0] = 1.0
    return a


def windows(case, seed):
    """Window starts: sizes log-uniform in 200..5000 SNPs."""
    rng, ws = np.random.default_rng([seed, 3]), [0]
    while ws[-1] < case["m"]:
        ws.append(ws[-1] + int(round(math.exp(rng.uniform(math.log(200), math.log(5000))))))
    ws[-1] = case["m"]
    if len(ws) > 2 and ws[-1] - ws[-2] < 50:
        del ws[-2]
    return np.array(ws, dtype=np.int64)


def partners(case):
    j = np.arange(case["m"])
    return (np.maximum(0, j - case["reach"]), np.minimum(case["m"], j + case["reach"] + 1))


def gxe_inputs(case, seed):
    """Environments (pairwise correlation 0.2), the intercept-and-covariate basis, the
    environments' unit directions off it, probes and positive scales."""
    n, m, e = case["n"], case["m"], case["e"]
    rng = np.random.default_rng([seed, 4])
    env = rng.multivariate_normal(np.zeros(e), 0.2 + 0.8 * np.eye(e), size=n)
    u = np.linalg.qr(np.column_stack([np.ones(n), rng.normal(size=n)]))[0]
    d = env - u @ (u.T @ env)
    d /= np.linalg.norm(d, axis=0)
    z = rng.normal(size=(case["b"], m))
    sx, sw = 0.8 + 0.4 * rng.random((2, e, m))
    return np.asfortranarray(env), np.asfortranarray(u), np.asfortranarray(d), z, sx, sw


def two_pass_inputs(case, seed):
    n, q, r = case["n"], case["q"], case["r"]
    rng = np.random.default_rng([seed, 5])
    basis = np.column_stack([np.ones(n)] + [rng.normal(size=n) for _ in range(q - 1)])
    fixed = np.column_stack([np.ones(n)] + [rng.normal(size=n) for _ in range(r)])[:, :r]
    return basis, np.linalg.qr(fixed)[0] if r else np.zeros((n, 0))


def network_inputs(case, seed):
    """Standardized features, targets, and He-normal parameters of the 3 x 128 network."""
    n_out, n_in = case["k"], 20 + 2 * case["k"]
    rng = np.random.default_rng([seed, 6])
    parts = []
    for rows, cols in ((128, n_in), (128, 128), (128, 128), (n_out, 128)):
        parts += [rng.normal(0.0, math.sqrt(2.0 / cols), rows * cols), 0.01 * rng.normal(size=rows)]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    x = torch.randn((case["rows"], n_in), generator=gen, device="cuda")
    t = torch.randn((case["rows"], n_out), generator=gen, device="cuda")
    return np.concatenate(parts).astype(np.float32), x, t, n_in, n_out


# ---------------------------------------------------------------------------
# The public calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    from summit_b200 import bedfile, gxe, surrogate
    from summit_b200.generalized_gxe import GlobalVariantProbeSpec
    from summit_b200.session import GwSession, WinPlan

    kind, s = case["kind"], {"case": case, "seed": seed % 100003}
    if kind == "surrogate":
        params, s["x"], s["t"], n_in, n_out = network_inputs(case, seed)
        s["net"] = surrogate.Surrogate(n_in, n_out, params=params)
        s["xb"], s["tb"] = (v[:case["batch"]].contiguous() for v in (s["x"], s["t"]))
        return s
    rows = bed_rows(case, seed)
    if kind == "win_call":
        s["rows"] = torch.empty(rows.shape, dtype=torch.uint8, pin_memory=True).copy_(rows).numpy()
    else:
        s["rows"] = rows.cpu().numpy()
    del rows
    if kind in ("gw_plan", "win_plan", "window_ld", "gxe", "two_pass"):
        s["session"] = GwSession(s.pop("rows"), case["n"], impute_mode=case["impute"], impute_seed=7)
    if kind in ("gw_call", "gw_plan", "win_plan", "win_call", "blocks", "window_ld", "two_pass"):
        s["annot"] = annotations(case, seed)
    if kind == "gw_plan":
        s["plan"] = s["session"].plan(s["annot"], case["b"], case["step"], s["seed"])
    elif kind == "win_plan":
        s["plan"] = WinPlan(s["session"], s["annot"], windows(case, seed), case["b"], case["step"],
                            s["seed"])
    elif kind == "win_call":
        s["windows"] = windows(case, seed)
    elif kind == "blocks":
        s["dir"] = tempfile.TemporaryDirectory()
        s["prefix"] = bedfile.write_plink(s["dir"].name + "/geno", packed=s.pop("rows"), n=case["n"])
        s["annot"] = s["annot"].astype(case["dtype"])
    elif kind == "window_ld":
        s["lo"], s["hi"] = partners(case)
    elif kind == "gxe":
        env, u, d, z, sx, sw = gxe_inputs(case, seed)
        e, r = case["e"], u.shape[1]
        idx = np.array([list(range(r)) + [r + c] for c in range(e) for _ in range(4)], dtype=np.int64)
        eye = np.tile(np.eye(r + 1).ravel(), e)
        s["ref"] = gxe.GxeReference(
            s["session"], env, np.asfortranarray(np.hstack([u, d])), idx.ravel(),
            np.arange(4 * e + 1, dtype=np.int64) * (r + 1), np.full(e, r + 1, np.int32), eye,
            np.arange(e + 1, dtype=np.int64) * (r + 1) ** 2, eye.copy(), u, d)
        s["z"], s["sx"], s["sw"] = (torch.from_numpy(v).cuda().t() for v in (z, sx, sw))
        s["ones"] = torch.ones((1, case["m"]), dtype=torch.float64, device="cuda").t()
    elif kind == "two_pass":
        s["basis"], s["fixed"] = two_pass_inputs(case, seed)
        s["annot"] += 0.1
        s["probes"] = GlobalVariantProbeSpec(s["seed"], 0, case["b"])
    return s


def run_blocks(s):
    """The reference driver's call sequence of one estimate, block by block."""
    from summit_b200 import gwldcore

    case, annot, prefix = s["case"], s["annot"], s["prefix"]
    n, m, step, v, k = case["n"], case["m"], case["step"], case["b"], case["k"]
    bed = {"bed_prefix": prefix, "fam_path": prefix + ".fam", "ddof": 1,
           "impute_mode": case["impute"], "impute_seed": 7}
    spans = [(a, min(m, a + step)) for a in range(0, m, step)]
    inv = np.empty(m, dtype=annot.dtype)
    xz = np.zeros((n, k * v), dtype=annot.dtype, order="F")
    init = np.zeros(k, dtype=np.uint8)
    meansq = np.zeros((m, k), dtype=annot.dtype)
    for a, e in spans:
        gwldcore.phase1_compute_Xz_bed_chunk(
            blk_start=a, blk_end=e, annot_blk=annot[a:e], inv_right=inv[a:e], v_start=0, v_count=v,
            kmax_hint=e - a, seed=s["seed"], Xz2d_chunk=xz, bin_init_mask=init, inv_out=inv[a:e],
            **bed)
    for a, e in spans:
        gwldcore.phase2_accum_XtXz_bed(blk_start=a, blk_end=e, inv_left=inv[a:e], tile_nvecs=v,
                                       Xz2d=xz, meansq_accum=meansq, N_denom=n, **bed)
    return {"inv": inv, "xz": xz, "meansq": meansq}


def run(s):
    from summit_b200 import generalized_gxe, gwldcore
    from summit_b200.session import windowed_ldscore

    case, kind = s["case"], s["case"]["kind"]
    if kind == "gw_call":
        r = gwldcore.gw_ldscore(s["rows"], case["n"], s["annot"], case["b"], case["step"], s["seed"],
                                impute_mode=case["impute"], impute_seed=7)
        return {"ldscore": r["ldscore"], "inv": r["inv"]}
    if kind in ("gw_plan", "win_plan"):
        s["plan"].execute()
        r = s["plan"].results()
        return {"ldscore": r["ldscore"], "meansq": r["meansq_accum"], "inv": r["inv"]}
    if kind == "win_call":
        r = windowed_ldscore(s["rows"], case["n"], s["annot"], s["windows"], case["b"], case["step"],
                             s["seed"], impute_mode=case["impute"], impute_seed=7)
        return {"ldscore": r["ldscore"]}
    if kind == "blocks":
        return run_blocks(s)
    if kind == "window_ld":
        return {"ld": s["session"].window_ld(s["lo"], s["hi"], s["annot"], corr_dim=case["n"] - 1)}
    if kind == "gxe":
        r = s["ref"].run(s["z"], s["ones"], s["sx"], s["sw"])
        return {w: r["accum_" + w] for w in ("xx", "xw", "wx", "ww")}
    if kind == "two_pass":
        p1, p2 = generalized_gxe.two_pass(s["session"], s["basis"], s["fixed"], s["annot"], s["probes"])
        return {"sources": p1.contextual_sources, "scores": p2.directional_ldscores,
                "gram": p2.genetic_gram, "diagonal": p2.component_kernel_diagonal,
                "same_person": p2.same_person}
    out = s["net"].forward(s["x"])
    loss, grad = s["net"].loss_grad(s["xb"], s["tb"])
    return {"out": out, "loss": loss, "grad": grad}


def work(case):
    """Genotype codes, annotations and outputs once each; 2 operations per multiply-add of
    the products over annotated SNPs (density 0.1 for K > 1)."""
    if case["kind"] == "surrogate":
        k, n_in = case["k"], 20 + 2 * case["k"]
        per_row = 2.0 * (128 * n_in + 2 * 128 * 128 + 128 * k)
        return {"bytes": 4.0 * (case["rows"] + case["batch"]) * (n_in + k),
                "flops": per_row * (case["rows"] + 3 * min(case["batch"], case["rows"]))}
    n, m, codes = case["n"], case["m"], case["n"] * case["m"] / 4.0
    if case["kind"] == "window_ld":
        pairs = m * min(m, 2 * case["reach"] + 1.0)
        return {"bytes": codes + 16.0 * m * case["k"], "flops": pairs * (n + 2.0 * case["k"])}
    b = case["b"]
    if case["kind"] == "gxe":
        c = 2 * case["e"] * b
        return {"bytes": codes + 8.0 * m * (b + 6 * case["e"]), "flops": 2.0 * n * m * (c + 2 * c)}
    k = case["k"]
    if case["kind"] == "two_pass":
        q = case["q"]
        pairs = q * (q + 1) // 2
        families = q * q if case["r"] else pairs
        return {"bytes": codes + 8.0 * (n * k * (q * b + pairs) + m * k * pairs * pairs),
                "flops": 2.0 * n * m * k * (b + b * families + pairs)}
    density = 1.0 if k == 1 else 0.1
    sketch = 16.0 * n * k * b if case["kind"] == "blocks" else 0.0
    return {"bytes": codes + 24.0 * m * k + sketch,
            "flops": 2.0 * n * m * k * b * (density + 1.0)}


# ---------------------------------------------------------------------------
# FP64 restatements
# ---------------------------------------------------------------------------
def mix64(x):
    with np.errstate(over="ignore"):
        x = np.asarray(x, dtype=np.uint64) + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))


def mt19937_64_bits(seeds, count):
    """The low bit of the first `count` draws of one generator per seed."""
    u = np.uint64
    mt = np.empty((len(seeds), 312), dtype=np.uint64)
    mt[:, 0] = seeds
    out = np.empty((len(seeds), count), dtype=np.int8)
    with np.errstate(over="ignore"):
        for i in range(1, 312):
            mt[:, i] = u(6364136223846793005) * (mt[:, i - 1] ^ (mt[:, i - 1] >> u(62))) + u(i)

        def step(a, b, nxt, far):
            x = (mt[:, a:b] & u(0xFFFFFFFF80000000)) | (nxt & u(0x7FFFFFFF))
            mt[:, a:b] = far ^ (x >> u(1)) ^ ((x & u(1)) * u(0xB5026F5AA96619E9))

        for at in range(0, count, 312):
            step(0, 156, mt[:, 1:157], mt[:, 156:312])
            step(156, 311, mt[:, 157:312], mt[:, 0:155])
            step(311, 312, mt[:, 0:1], mt[:, 155:156])
            x = mt ^ ((mt >> u(29)) & u(0x5555555555555555))
            x ^= (x << u(17)) & u(0x71D67FFFEDA60000)
            x ^= (x << u(37)) & u(0xFFF7EEE000000000)
            x ^= x >> u(43)
            w = min(312, count - at)
            out[:, at:at + w] = (x[:, :w] & u(1)).astype(np.int8)
    return out


def rademacher(m, b, spans):
    """M x B probes; a span (first SNP, SNPs, root seed, block start) has its own stream
    per tile of probes."""
    width = b if b < 64 else b // 64 * 64
    z = np.empty((m, b))
    size = max(c for _, c, _, _ in spans)
    for v0 in range(0, b, width):
        v = min(width, b - v0)
        seeds = [0x1234ABCD ^ int(mix64(root)) ^ int(mix64(blk + 0x9E37)) ^ int(mix64(v0 + 0x85EB))
                 for _, _, root, blk in spans]
        bits = mt19937_64_bits(np.array(seeds, dtype=np.uint64), size * v)
        for (a, c, _, _), row in zip(spans, bits):
            z[a:a + c, v0:v0 + v] = 2.0 * row[:c * v].reshape(v, c).T - 1.0
    return torch.from_numpy(z).cuda()


def genotypes(case, seed, ddof=1):
    """Standardized genotypes (M x N FP64): mean imputation leaves zeros, HWE completion
    draws each missing call from its SNP's Hardy-Weinberg cells."""
    n, m = case["n"], case["m"]
    rows = bed_rows(case, seed)
    x = torch.empty((m, n), dtype=torch.float64, device="cuda")
    value = torch.tensor([0.0, -9.0, 1.0, 2.0], dtype=torch.float64, device="cuda")
    for a in range(0, m, 1024):
        r = rows[a:a + 1024]
        codes = torch.stack([r >> 2 * t & 3 for t in range(4)], -1).reshape(r.shape[0], -1)[:, :n]
        g = value[codes.long()]
        seen = g >= 0
        count, total = seen.sum(1).double(), torch.where(seen, g, 0.0).sum(1)
        if case["impute"] == "hwe":
            p = (total / (2 * count)).cpu().numpy()
            j, i = (v.cpu().numpy() for v in torch.nonzero(~seen, as_tuple=True))
            base = int(mix64(7)) ^ mix64(np.arange(a, a + len(p), dtype=np.uint64)
                                         + np.uint64(0x243F6A8885A308D3))
            h = mix64(base[j] ^ mix64(i.astype(np.uint64) + np.uint64(0x9E3779B97F4A7C15)))
            u = (h >> np.uint64(11)).astype(np.float64) / 9007199254740992.0
            q0 = (1 - p) * (1 - p)
            q01 = q0 + 2 * p * (1 - p)
            g[~seen] = torch.from_numpy((u >= q0[j]).astype(np.float64) + (u >= q01[j])).cuda()
            seen = torch.ones_like(seen)
            count, total = torch.full_like(count, n), g.sum(1)
        mu = (total / count)[:, None]
        d = torch.where(seen, g - mu, 0.0)
        x[a:a + 1024] = d / (d.square().sum(1) / (count - ddof)).sqrt()[:, None]
    return x


def ld_scores(x, annot, z, spans, b):
    """Raw sums, scores, inverse residual sds, and the last span's sketch (N x K*B)."""
    m, n = x.shape
    k = annot.shape[1]
    annot = torch.from_numpy(annot).cuda()
    inv = 1.0 / (x.square().sum(1) / (n - 1)).clamp_min(1e-10).sqrt()
    raw = torch.empty((m, k), dtype=torch.float64, device="cuda")
    null = torch.empty_like(raw)
    for a, e in spans:
        y = torch.empty((n, k * b), dtype=torch.float64, device="cuda")
        for c in range(k):
            at = a + torch.nonzero(annot[a:e, c] > 0)[:, 0]
            y[:, c * b:(c + 1) * b] = x[at].t() @ ((inv[at] * annot[at, c].sqrt())[:, None] * z[at])
        w = (x[a:e] @ y).view(e - a, k, b)
        raw[a:e] = w.square().sum(2) * (inv[a:e] / (n - 1)).square()[:, None]
        null[a:e] = annot[a:e].sum(0) / (n - 1)
    return raw, raw / b - null, inv, y


def exact_gxe(case, seed):
    env, u, d, z, sx, sw = (torch.from_numpy(np.ascontiguousarray(v)).cuda()
                            for v in gxe_inputs(case, seed))
    x = genotypes(case, seed)
    (m, n), e, b = x.shape, case["e"], case["b"]
    out = {w: torch.zeros((e * m, 1), dtype=torch.float64, device="cuda")
           for w in ("xx", "xw", "wx", "ww")}
    for c in range(e):
        for h, s in (("x", sx[c]), ("w", sw[c])):
            y = x.t() @ (z * s).t()
            if h == "w":
                y *= env[:, c:c + 1]
            y -= u @ (u.t() @ y)
            y -= d[:, c:c + 1] * (d[:, c] @ y) + y.mean(0)
            for p, t, v in (("x", sx[c], y), ("w", sw[c], env[:, c:c + 1] * y)):
                score = (x @ v).square().sum(1) * t * t / (n - u.shape[1] - 1) ** 2 / b
                out[p + h][c * m:(c + 1) * m, 0] = score
    return out


def exact_two_pass(case, seed):
    basis, fixed = (torch.from_numpy(v).cuda() for v in two_pass_inputs(case, seed))
    annot = torch.from_numpy(annotations(case, seed) + 0.1).cuda()
    x = genotypes(case, seed)
    (m, n), k, q, b = x.shape, case["k"], case["q"], case["b"]
    key = 0xCBF29CE484222325
    for byte in b"summit.generalized_gxe.variant_ldscore.reference":
        key = ((key ^ byte) * 0x100000001B3) & M64
    sign = mix64((mix64(seed % 100003 ^ key ^ 0x9E3779B97F4A7C15)
                  ^ mix64(np.arange(m, dtype=np.uint64) + np.uint64(0xD2B74407B1CE6E93)))[:, None]
                 ^ mix64(np.arange(b, dtype=np.uint64) + np.uint64(0xCA5A826395121157)))
    z = torch.from_numpy(np.where(sign >> np.uint64(63), 1.0, -1.0)).cuda()
    off = lambda v: v - fixed @ (fixed.t() @ v)  # noqa: E731
    sources = torch.stack([torch.stack([off(basis[:, t:t + 1] * (x.t() @ (annot[:, c:c + 1].sqrt() * z)))
                                        for t in range(q)]) for c in range(k)])
    cross = {(t, s, c): x @ (basis[:, t:t + 1] * sources[c, s]) / (n - fixed.shape[1])
             for t in range(q) for s in range(q) for c in range(k)}
    pairs = [(t, t) for t in range(q)] + [(t, s) for t in range(q - 1) for s in range(t + 1, q)]
    both = lambda p: [p] if p[0] == p[1] else [p, p[::-1]]  # noqa: E731
    scores = torch.zeros((m, len(pairs), k * len(pairs)), dtype=torch.float64, device="cuda")
    for i, target in enumerate(pairs):
        for j, source in enumerate(pairs):
            for c in range(k):
                for tl, tr in both(target):
                    for sl, sr in both(source):
                        scores[:, i, c * len(pairs) + j] += (
                            cross[tr, sl, c] * cross[tl, sr, c]).sum(1) / b
    directed = torch.einsum("vk,vpc->kpc", annot, scores).reshape(k * len(pairs), -1)
    mass = annot.sum(0).repeat_interleave(len(pairs))
    gram = (n - fixed.shape[1]) ** 2 * 0.5 * (directed + directed.t()) / torch.outer(mass, mass)
    features = [off(basis[:, t:t + 1] * x.t()) for t in range(q)]
    diag = torch.stack([((1.0 if t == s else 2.0) * features[t] * features[s]) @ annot[:, c]
                        for c in range(k) for t, s in pairs]) / mass[:, None]
    return {"sources": sources, "scores": scores, "gram": gram, "diagonal": diag,
            "same_person": diag @ diag.t()}


def exact_surrogate(case, seed):
    params, x, t, n_in, n_out = network_inputs(case, seed)
    p = torch.from_numpy(params).cuda().double().requires_grad_()

    def forward(h):
        at = 0
        for rows, cols in ((128, n_in), (128, 128), (128, 128), (n_out, 128)):
            w = p[at:at + rows * cols].view(rows, cols)
            h = h @ w.t() + p[at + rows * cols:at + rows * cols + rows]
            at += rows * cols + rows
            h = torch.nn.functional.gelu(h) if at < p.numel() else h
        return h

    with torch.no_grad():
        out = forward(x.double())
    loss = (forward(x[:case["batch"]].double()) - t[:case["batch"]]).square().mean()
    return {"out": out, "loss": loss.item(), "grad": torch.autograd.grad(loss, p)[0]}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("gxe", "two_pass", "surrogate"):
        return {"gxe": exact_gxe, "two_pass": exact_two_pass, "surrogate": exact_surrogate}[kind](
            case, seed)
    x, annot, m = genotypes(case, seed), annotations(case, seed), case["m"]
    if kind == "window_ld":
        x /= x.square().sum(1).sqrt()[:, None]
        lo, hi = (torch.from_numpy(v).cuda() for v in partners(case))
        i, ld = torch.arange(m, device="cuda"), []
        for a in range(0, m, 2048):
            f = (x[a:a + 2048] @ x.t()).square()
            f -= (1 - f) / (case["n"] - 2)
            f *= (i >= lo[a:a + 2048, None]) & (i < hi[a:a + 2048, None])
            ld.append(f @ torch.from_numpy(annot).cuda())
        return {"ld": torch.cat(ld)}
    step, root = case["step"], seed % 100003
    spans = [(0, m)]
    if kind in ("win_plan", "win_call"):
        ws = windows(case, seed)
        spans = list(zip(ws[:-1].tolist(), ws[1:].tolist()))
    streams = []
    for w, (a, e) in enumerate(spans):
        r = root if len(spans) == 1 and kind[:3] != "win" else int(
            mix64(root ^ int(mix64(0x77696E646F77 + w))))
        streams += [(a + s, min(step, e - a - s), r, s) for s in range(0, e - a, step)]
    raw, ld, inv, y = ld_scores(x, annot, rademacher(m, case["b"], streams), spans, case["b"])
    if kind == "blocks":
        return {"inv": inv, "xz": y, "meansq": raw}
    if kind == "win_call":
        return {"ldscore": ld}
    return {"ldscore": ld, "inv": inv} if kind == "gw_call" else {
        "ldscore": ld, "meansq": raw, "inv": inv}
