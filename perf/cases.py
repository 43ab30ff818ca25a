"""Performance cases of the f2 block-tensor extraction: what a program has this package do.

Each case goes through a public entry point of ``steppecu_b200`` over inputs drawn on the
GPU from a Balding-Nichols-like model: SNP-major PACKEDANCESTRYMAP records, populations
interleaved in file order, half of the samples pseudo-haploid, a per-sample missing rate of
Beta(2, 3), F in U(0.01, 0.15), 5 cM jackknife blocks on human-like chromosomes (or lognormal
block sizes). Kinds of a case:

- ``pass``: ``Plan.run`` (or ``run_graph``), records and outputs resident on the device;
- ``host``: ``Context.extract_blocks`` with pinned host records and outputs, plan included;
- ``batch``: ``Context.extract_batch``, many requests over one panel, each its own block map;
- ``keep``: ``Context.snp_keep_mask``, the SNP filters that run before the block walk;
- ``counts``: ``Context.decode_counts_noalloc``, exact allele counts on the device;
- ``qvn``: ``Context.f2_from_qvn`` on device frequencies (compute_f2_blocks_device);
- ``fstats``: ``Context.fstats`` (f4 quartets with their jackknife) on a device f2 tensor.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import steppecu_b200 as st
from steppecu_b200 import _lib
from steppecu_b200.synth import HUMAN_CM

# Limits of a drawn case, those of the largest listed one.
_MAX_PAIRS = 1.15e12     # P^2 M
_MAX_GENO = 1.15e10      # N M
_MAX_SLAB = 7.2e8        # P^2 n_block


def _case(name, kind, P, size, M, chroms=22, **kw):
    c = {"name": name, "kind": kind, "P": P, "size": size, "M": M, "chroms": chroms, "precision": "fixed_i8",
         "lognormal_pops": False, "lognormal_blocks": False, "graph": False, "n_req": 1, "n_stat": 0}
    c.update(kw)
    return c


def listed() -> list[dict]:
    return [
        # A small study: 20 populations of 20 samples on two chromosomes, the pass replayed
        # as one CUDA graph: launches and latency.
        _case("pass_20x20_50k", "pass", 20, 20, 50_000, 2, graph=True),
        # A curated reference set over a full 1.15M-SNP array: decode-heavy.
        _case("pass_100x20_1150k", "pass", 100, 20, 1_150_000),
        # A whole-database extraction, every population: the contraction at its largest.
        _case("pass_1000x10_1150k", "pass", 1000, 10, 1_150_000),
        # As databases are: population sizes from 1 to 60, blocks from 50 to 6,000 SNPs,
        # nothing a multiple of a tile.
        _case("pass_ragged_603_401k", "pass", 603, 12, 401_113, lognormal_pops=True, lognormal_blocks=True),
        # The 16-bit split arithmetic.
        _case("pass_f16_300x10_400k", "pass", 300, 10, 400_000, precision="split_f16"),
        # The plain FP32 arithmetic (what a caller asking for Tf32 gets).
        _case("pass_fp32_100x20_200k", "pass", 100, 20, 200_000, precision="fp32"),
        # Many users' requests over one panel in one call.
        _case("batch_24_of_300x20_400k", "batch", 300, 20, 400_000, n_req=24),
        # One extraction out of host memory into host memory, as extract_f2 makes it.
        _case("host_150x10_300k", "host", 150, 10, 300_000),
        # The filters of one extract_f2 call: maf and missingness over every SNP.
        _case("keep_200x10_600k", "keep", 200, 10, 600_000),
        # Exact counts of a small window for a caller that cannot allocate.
        _case("counts_50x8_30k", "counts", 50, 8, 30_000, 2),
        # Frequencies that another program decoded, f2 left on the device.
        _case("qvn_300_200k", "qvn", 300, 10, 200_000),
        # A screen of f4 quartets over an extracted tensor.
        _case("f4_300x700_5000", "fstats", 300, 0, 1_150_000, n_stat=5000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["pass"] * 6 + ["batch", "host", "keep", "counts", "qvn", "fstats"])
    chroms = rng.randint(1, 22)
    if kind == "pass":
        precision = rng.choice(["fixed_i8"] * 4 + ["split_f16", "split_bf16", "fp32"])
        P, M = _log(rng, 3, 1000), _log(rng, 5_000, 1_150_000)
        size = _log(rng, 1, 40)
        M = int(min(M, _MAX_PAIRS / P ** 2, _MAX_GENO / (1.3 * P * size)))
        if precision == "fp32":
            M = int(min(M, 2e10 / P ** 2))
        return _case("", kind, P, size, max(M, 1000), chroms, precision=precision, graph=rng.random() < 0.3,
                     lognormal_pops=rng.random() < 0.4, lognormal_blocks=rng.random() < 0.4)
    if kind == "batch":
        return _case("", kind, _log(rng, 40, 300), rng.randint(4, 20), _log(rng, 50_000, 400_000), chroms,
                     n_req=rng.randint(2, 24))
    if kind == "host":
        return _case("", kind, _log(rng, 5, 180), rng.randint(2, 20), _log(rng, 20_000, 300_000), chroms,
                     lognormal_pops=rng.random() < 0.5)
    if kind == "keep":
        return _case("", kind, _log(rng, 5, 300), rng.randint(1, 20), _log(rng, 20_000, 600_000), chroms,
                     lognormal_pops=rng.random() < 0.5)
    if kind == "counts":  # the scratch of the allocation-free form is 32 MiB
        P, size = _log(rng, 2, 100), rng.randint(1, 12)
        return _case("", kind, P, size, int(min(_log(rng, 1_000, 60_000), 4e7 / (P * size))), min(chroms, 2))
    if kind == "qvn":
        return _case("", kind, _log(rng, 5, 400), rng.randint(2, 20), _log(rng, 10_000, 200_000), chroms,
                     lognormal_blocks=rng.random() < 0.5)
    return _case("", kind, _log(rng, 5, 400), 0, 1_150_000, chroms, n_stat=_log(rng, 50, 20_000))


# ---- inputs ------------------------------------------------------------------------------

def _shape_rng(case, stream):
    """What gives the outputs their shapes (population sizes, positions, blocks, which
    populations a request takes) is the case's; samples and genotypes are the seed's."""
    return np.random.default_rng([case["P"], case["size"], case["M"], case["chroms"], stream])


def _positions(case):
    rng, M, chroms = _shape_rng(case, 0), case["M"], case["chroms"]
    lens = np.asarray(HUMAN_CM[:chroms], np.float64)
    per = np.floor(M * lens / lens.sum()).astype(np.int64)
    per[: M - per.sum()] += 1
    chrom = np.repeat(np.arange(1, chroms + 1, dtype=np.int32), per)
    phys = np.concatenate([np.sort(rng.integers(1, int(L * 1e6), size=k)) for L, k in zip(lens, per)]).astype(np.float64)
    return chrom, phys


def _blocks(case, chrom, phys, scale=1.0):
    rng, M = _shape_rng(case, 1), case["M"]
    if case["lognormal_blocks"]:
        sizes, total = [], 0
        while total < M:
            k = min(int(np.clip(round(1500 * math.exp(rng.normal(0.0, 0.8))), 50, 6000)), M - total)
            sizes.append(k)
            total += k
        return np.repeat(np.arange(len(sizes), dtype=np.int32), sizes), len(sizes)
    return st.assign_blocks(chrom, phys * 1e-8 * scale, 0.05, phys)


def _sizes(case):
    rng = _shape_rng(case, 2)
    if case["lognormal_pops"]:
        return np.clip(np.round(case["size"] * np.exp(rng.normal(0.0, 0.7, size=case["P"]))), 1, 60).astype(np.int64)
    return np.full(case["P"], case["size"], np.int64)


def _panel(case, seed):
    """Records on the device and what selects from them."""
    rng = np.random.default_rng([seed, 7])
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    P, M = case["P"], case["M"]
    ind_pop = np.repeat(np.arange(P, dtype=np.int64), _sizes(case))
    rng.shuffle(ind_pop)
    N = ind_pop.size
    dip = rng.random(N) < 0.5
    miss = torch.as_tensor(rng.beta(2.0, 3.0, size=N), dtype=torch.float32, device="cuda")[None]
    F = torch.as_tensor(rng.uniform(0.01, 0.15, size=P), dtype=torch.float32, device="cuda")[None]
    chrom, phys = _positions(case)
    pop = torch.as_tensor(ind_pop, device="cuda")
    dipt = torch.as_tensor(dip, device="cuda")[None]
    bpr = max(48, (N + 3) // 4)
    rec = torch.zeros((M, bpr), dtype=torch.uint8, device="cuda")
    n4 = (N + 3) // 4 * 4
    step = max(1, min(M, (1 << 28) // n4))
    for s0 in range(0, M, step):
        m = min(step, M - s0)
        anc = 0.05 + 0.9 * torch.rand(m, 1, generator=g, device="cuda")
        p = (anc + (F * anc * (1 - anc)).sqrt() * torch.randn(m, P, generator=g, device="cuda")).clamp_(0, 1)
        p = p.index_select(1, pop)
        u = torch.rand(m, N, generator=g, device="cuda")
        code = torch.where(dipt, (u < p * p).to(torch.uint8) + (u < p * (2 - p)), (u < p).to(torch.uint8) * 2)
        u.uniform_(generator=g)
        code.masked_fill_(u < miss, 3)
        c = torch.nn.functional.pad(code, (0, n4 - N)).view(m, -1, 4)
        rec[s0:s0 + m, :n4 // 4] = (c[:, :, 0] << 6) | (c[:, :, 1] << 4) | (c[:, :, 2] << 2) | c[:, :, 3]
        del p, u, code, c
    return {"rec": rec, "N": N, "chrom": chrom, "phys": phys, "ind_pop": ind_pop, "rng": rng}


def _selection(ind_pop, P, pops=None):
    order = np.argsort(ind_pop, kind="stable")
    start = np.concatenate([[0], np.cumsum(np.bincount(ind_pop, minlength=P))])
    pops = range(P) if pops is None else pops
    rows = [order[start[i]:start[i + 1]] for i in pops]
    return np.concatenate(rows).astype(np.int64), np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int64)


def _alleles(rng, M):
    ref = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, M)]
    alt = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, M)]
    return ref, alt


_FILTER = {"maf_min": 0.05, "maxmiss": 0.05, "autosomes_only": True}


def _requests(p, case):
    rng, out = _shape_rng(case, 3), []
    for _ in range(case["n_req"]):
        k = max(2, min(case["P"], int(round(math.exp(rng.uniform(math.log(4), math.log(case["P"])))))))
        sel, po = _selection(p["ind_pop"], case["P"], np.sort(rng.choice(case["P"], k, replace=False)))
        bid, nb = _blocks(case, p["chrom"], p["phys"], rng.uniform(0.9, 1.1))
        out.append({"sel_rows": sel, "pop_offsets": po, "block_id": bid, "n_block": nb})
    return out


def _qvn(case, seed):
    """Frequencies, validity and called alleles [M, P] of a decoded panel."""
    rng = np.random.default_rng([seed, 7])
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    P, M = case["P"], case["M"]
    chrom, phys = _positions(case)
    bid, nb = _blocks(case, chrom, phys)
    anc = 0.05 + 0.9 * torch.rand(M, 1, generator=g, device="cuda", dtype=torch.float64)
    p = (anc + 0.28 * (anc * (1 - anc)).sqrt() * torch.randn(M, P, generator=g, device="cuda")).clamp_(0, 1)
    N = torch.randint(0, 2 * case["size"] + 1, (M, P), generator=g, device="cuda").double()
    Q = (torch.round(p * N) / N).nan_to_num_(0.0)
    return Q, (N > 0).double(), N, bid, nb


def _tensor(case, seed):
    """An f2 tensor of realistic values, its counts and block sizes."""
    rng = np.random.default_rng([seed, 7])
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    P = case["P"]
    chrom, phys = _positions(case)
    bid, nb = st.assign_blocks(chrom, phys * 1e-8, 0.05, phys)
    bs = np.bincount(bid, minlength=nb).astype(np.int32)
    d = 0.02 + 0.13 * torch.rand(P, generator=g, device="cuda", dtype=torch.float64)
    f2 = (d[None, :, None] + d[None, None, :]) * (1 + 0.1 * torch.randn(nb, P, P, generator=g, device="cuda"))
    f2 = 0.5 * (f2 + f2.transpose(1, 2))
    vp = torch.as_tensor(bs, device="cuda").double()[:, None, None].expand(nb, P, P).contiguous()
    quart = np.stack([rng.permutation(P)[:4] for _ in range(case["n_stat"])]).astype(np.int32)
    return f2.contiguous(), vp, bs, nb, quart


def _dev(n):
    return torch.empty(n, dtype=torch.float64, device="cuda")


def prepare(case, seed) -> dict:
    ctx, kind, P = st.context(0), case["kind"], case["P"]
    s = {"kind": kind, "ctx": ctx, "P": P, "graph": case["graph"], "precision": case["precision"]}
    if kind == "qvn":
        Q, V, N, bid, nb = _qvn(case, seed)
        s.update(q=Q.view(-1), v=V.view(-1), n=N.view(-1), bid=bid, nb=nb, out=(_dev(P * P * nb), _dev(P * P * nb)))
    elif kind == "fstats":
        f2, vp, bs, nb, quart = _tensor(case, seed)
        s.update(f2=f2.view(-1), vp=vp.view(-1), bs=bs, nb=nb, quart=quart.reshape(-1), n_stat=case["n_stat"])
    else:
        p = _panel(case, seed)
        s.update(rec=p["rec"], N=p["N"])
        if kind == "batch":
            s["reqs"] = _requests(p, case)
            s["out"] = [tuple(_dev((q["pop_offsets"].size - 1) ** 2 * q["n_block"]) for _ in range(2)) for q in s["reqs"]]
        elif kind == "counts":
            s["sel"], s["po"] = _selection(p["ind_pop"], P)
            pitch = (p["rec"].shape[1] + 15) // 16 * 16
            s["rec"] = torch.nn.functional.pad(p["rec"], (0, pitch - p["rec"].shape[1]))
            s["out"] = tuple(torch.empty(P * case["M"], dtype=torch.int32, device="cuda") for _ in range(2))
        elif kind == "keep":
            s["sel"], s["po"] = _selection(p["ind_pop"], P)
            s["ref"], s["alt"] = _alleles(p["rng"], case["M"])
            s["chrom"] = p["chrom"]
        else:
            s["sel"], s["po"] = _selection(p["ind_pop"], P)
            s["bid"], s["nb"] = _blocks(case, p["chrom"], p["phys"])
            n = P * P * s["nb"]
            if kind == "host":
                s["rec"] = torch.empty(p["rec"].shape, dtype=torch.uint8, pin_memory=True).copy_(p["rec"]).numpy()
                s["out"] = tuple(torch.empty(n, dtype=torch.float64, pin_memory=True).numpy() for _ in range(2))
            else:
                s["out"] = (_dev(n), _dev(n))
                s["plan"] = ctx.plan(s["rec"], s["N"], s["sel"], s["po"], s["bid"], s["nb"], case["precision"])
    torch.cuda.synchronize()  # the library works on its own stream
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "pass":
        (s["plan"].run_graph if s["graph"] else s["plan"].run)(s["rec"], *s["out"])
        return s["out"]
    if kind == "host":
        t = ctx.extract_blocks(s["rec"], s["N"], s["sel"], s["po"], s["bid"], s["nb"], s["precision"], out=s["out"])
        return t.f2, t.vpair, t.block_sizes
    if kind == "batch":
        return [r[:2] for r in ctx.extract_batch(s["rec"], s["N"], s["reqs"], s["precision"], out=s["out"])]
    if kind == "keep":
        return ctx.snp_keep_mask(s["rec"], s["N"], s["sel"], s["po"], s["ref"], s["alt"], s["chrom"], **_FILTER)
    if kind == "counts":
        ctx.decode_counts_noalloc(s["rec"], s["N"], s["sel"], s["po"], *s["out"])
        return s["out"]
    if kind == "qvn":
        return ctx.f2_from_qvn(s["q"], s["v"], s["n"], s["P"], s["bid"], s["nb"], s["precision"], out=s["out"])
    est, var, n = ctx.fstats(s["f2"], s["vp"], s["bs"], s["P"], s["nb"], _lib.FSTAT_F4, s["quart"], s["n_stat"])
    return est, var, n


# ---- work, tolerance, 64-bit results -------------------------------------------------------

def _n_block(case):
    if case["lognormal_blocks"]:
        return max(1, case["M"] / 2000)
    return sum(max(1, c / 5) for c in HUMAN_CM[:case["chroms"]])


def work(case) -> dict:
    kind, P, M = case["kind"], case["P"], case["M"]
    N = P * case["size"] * (1.26 if case["lognormal_pops"] else 1.0)
    rec = N * M / 4
    if kind == "fstats":
        return {"bytes": 8 * P * P * _n_block(case) + 32 * case["n_stat"] * _n_block(case),
                "flops": 40 * case["n_stat"] * _n_block(case)}
    if kind == "keep":
        return {"bytes": rec + 7 * M, "flops": 2 * N * M}
    if kind == "counts":
        return {"bytes": rec + 8 * P * M, "flops": 2 * N * M}
    if kind == "qvn":
        return {"bytes": 24 * P * M + 16 * P * P * _n_block(case), "flops": 3 * P * (P + 1) * M}
    if kind == "batch":  # P_r is log-uniform on [4, P]
        span = max(math.log(P / 4), 1e-9)
        p2 = case["n_req"] * max(P * P - 16, 1) / (2 * span)
        return {"bytes": rec + 16 * p2 * _n_block(case), "flops": 3 * p2 * M}
    return {"bytes": rec + 16 * P * P * _n_block(case), "flops": 3 * P * (P + 1) * M}


def tolerance(case):
    if case["kind"] in ("keep", "counts"):
        return "exact"
    if case["kind"] == "fstats":
        return {"rel": 1e-12, "max": 1e-11}
    # f2 of the fixed point, the FP32 form, and the split 16-bit forms; whole counts agree.
    # About four times the error seen against exact() over listed and drawn cases.
    return {"fixed_i8": {"rel": 5e-9, "max": 5e-8}, "fp32": {"rel": 4e-7, "max": 4e-6},
            "split_f16": {"rel": 2e-6, "max": 1e-5}, "split_bf16": {"rel": 4e-5, "max": 4e-4}}[case["precision"]]


def _counts(rec, N, sel, po, s0, m):
    """Exact (ac2, n) [m, P] FP64 of SNPs s0 .. s0+m for the selected samples."""
    b = rec[s0:s0 + m, :(N + 3) // 4]
    code = torch.stack([(b >> k) & 3 for k in (6, 4, 2, 0)], 2).reshape(m, -1).index_select(1, sel["rows"])
    called = code != 3
    w = sel["ploidy"][None]
    a = torch.where(called, code.float() * w, 0.0) @ sel["member"]
    return a.double(), (called.float() * w) @ sel["member"]


def _select(rec, N, sel_rows, po):
    rows = torch.as_tensor(sel_rows, device="cuda")
    b = rec[:1000, :(N + 3) // 4]
    code = torch.stack([(b >> k) & 3 for k in (6, 4, 2, 0)], 2).reshape(b.shape[0], -1).index_select(1, rows)
    ploidy = 1.0 + (code == 1).any(0).float()
    member = torch.zeros(rows.numel(), po.size - 1, device="cuda")
    owner = torch.repeat_interleave(torch.arange(po.size - 1, device="cuda"), torch.as_tensor(np.diff(po), device="cuda"))
    member[torch.arange(rows.numel(), device="cuda"), owner] = 1.0
    return {"rows": rows, "ploidy": ploidy, "member": member}


def _block_f2(q, n):
    """f2 and both-present counts [P, P] of one block from q, n [k, P] FP64 (q = 0 at n = 0)."""
    m = (n > 0).double()
    x = (q - 0.5) * m
    a = (x * x - q * (1 - q) / (n - 1).clamp_min(1.0)) * m
    am = a.t() @ m
    v = m.t() @ m
    return torch.where(v > 0, (am + am.t() - 2 * (x.t() @ x)) / v.clamp_min(1.0), 0.0), v


def _f2_exact(counts, bid, nb, P):
    """f2, vpair [nb, P, P] flat, with counts(s0, m) -> (ac2, n) of a run of SNPs, as this
    tensor's layout i + P j + P^2 b (symmetric slabs)."""
    f2, vp = _dev(nb * P * P).view(nb, P, P), _dev(nb * P * P).view(nb, P, P)
    edge = np.searchsorted(bid, np.arange(nb + 1))
    for b in range(nb):
        q, n = counts(int(edge[b]), int(edge[b + 1] - edge[b]))
        f2[b], vp[b] = _block_f2(q, n)
    return f2.view(-1), vp.view(-1)


def _panel_f2(rec, N, sel_rows, po, bid, nb):
    sel = _select(rec, N, sel_rows, po)

    def counts(s0, m):
        a, n = _counts(rec, N, sel, po, s0, m)
        n = n.double()
        return (0.5 * a / n).nan_to_num_(0.0), n

    return _f2_exact(counts, bid, nb, po.size - 1)


def exact(case, seed):
    kind, P, M = case["kind"], case["P"], case["M"]
    torch.backends.cuda.matmul.allow_tf32 = False
    if kind == "qvn":
        Q, V, N, bid, nb = _qvn(case, seed)
        f2, vp = _f2_exact(lambda s0, m: (Q[s0:s0 + m], N[s0:s0 + m]), bid, nb, P)
        return f2, vp, np.bincount(bid, minlength=nb).astype(np.int32)
    if kind == "fstats":
        f2, _, bs, nb, quart = _tensor(case, seed)
        q = torch.as_tensor(quart, device="cuda").long()
        f = lambda i, j: f2[:, q[:, i], q[:, j]]  # noqa: E731
        x = 0.5 * (f(1, 2) + f(0, 3) - f(0, 2) - f(1, 3))
        n = float(bs.sum())
        w = torch.as_tensor(bs, device="cuda").double()[:, None]
        tot = (x * w).sum(0) / n
        rel = w / n
        loo = (tot - x * rel) / (1 - rel)
        line = (loo * (1 - rel)).sum(0) / (1 - rel).sum()
        est = (line - loo).sum(0) + (loo * w).sum(0) / n
        h = n / w
        var = (((est * h - loo * (h - 1) - line) ** 2) / (h - 1)).mean(0)
        return est, var, nb
    p = _panel(case, seed)
    rec, N = p["rec"], p["N"]
    if kind == "batch":
        return [_panel_f2(rec, N, q["sel_rows"], q["pop_offsets"], q["block_id"], q["n_block"]) for q in _requests(p, case)]
    sel_rows, po = _selection(p["ind_pop"], P)
    if kind in ("counts", "keep"):
        sel = _select(rec, N, sel_rows, po)
        step = max(1, min(M, (1 << 28) // max(N, 1)))
        parts = [_counts(rec, N, sel, po, s0, min(step, M - s0)) for s0 in range(0, M, step)]
        ac2, n = torch.cat([a for a, _ in parts]), torch.cat([n for _, n in parts]).double()
        if kind == "counts":
            return ac2.reshape(-1).int(), n.reshape(-1).int()
        ref, alt = _alleles(p["rng"], M)
        tot = n.sum(1)
        af = torch.where(tot > 0, 0.5 * ac2.sum(1) / tot.clamp_min(1.0), 0.0)
        keep = torch.minimum(af, 1 - af) >= _FILTER["maf_min"]
        keep &= (n == 0).double().mean(1) <= _FILTER["maxmiss"]
        pair = np.array([chr(r) + chr(a) in ("AC", "CA", "AG", "GA", "TC", "CT", "TG", "GT") for r, a in zip(ref, alt)])
        return keep & torch.as_tensor(pair, device="cuda")
    bid, nb = _blocks(case, p["chrom"], p["phys"])
    f2, vp = _panel_f2(rec, N, sel_rows, po, bid, nb)
    if kind == "host":
        return f2, vp, np.bincount(bid, minlength=nb).astype(np.int32)
    return f2, vp
