"""The work this library is measured on: its public entry points over the sizes
its users bring, from one gene family of some dozen sequences to the largest
matrix of the benchmark configurations.

Kinds of case
-------------
resident   an alignment already on the device: ``Context.alignment`` (packing) and
           ``Context.distance_into`` (counts, transform, post-process).  What a
           program does that parsed the file on the device or keeps its matrix there.
host       ``Context.distance_matrix_host``: host bytes in, host matrix out, the
           call that stands for rapidNJ's own ``computeDistances``.  ``pinned``:
           page-locked buffers, as a program that calls it often keeps.
batch      ``Batch``: many alignments (gene families) packed, counted and
           transformed together.
bootstrap  ``Context.bootstrap``: rapidNJ's ``-b`` replicates.
nj         ``Context.nj_init``: rapidNJ's set-up over the finished matrix.
f64        ``Context.distance_f64``: the matrix in double precision.

Inputs are seeded alignments evolved down a random binary tree (Kimura-2P or
equal-rate amino-acid substitution, then gaps), or independent random sites
(``tree`` false), which give the saturated pairs whose distances the
post-process replaces.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from rapidnj_b200 import api

DEVICE = "cuda:0"
DNA = np.frombuffer(b"AGTC", dtype=np.uint8).copy()  # code 0..3; code ^ 1 is the transition
AMINO = np.frombuffer(b"ARNDCQEGHILKMFPSTWYV", dtype=np.uint8).copy()
GAP = ord("-")


def listed():
    return [
        # the repository's DNA fixture (68 x 1,302): one gene family through the
        # host call, where launches, copies and synchronisations count
        dict(name="host_dna_k2p_68x1302", kind="host", type="dna", model="kim", n=68, L=1302,
             tree=True, pinned=False),
        # a small protein family, odd sizes, Jukes-Cantor
        dict(name="resident_protein_jc_301x421", kind="resident", type="protein", model="jc",
             n=301, L=421, tree=True, fastdist=True),
        # the benchmark's small configuration: independent sites, half the pairs saturated
        dict(name="resident_dna_jc_512x2000", kind="resident", type="dna", model="jc", n=512,
             L=2000, tree=False, fastdist=True),
        # the benchmark's headline configuration
        dict(name="resident_dna_k2p_10000x10000", kind="resident", type="dna", model="kim",
             n=10000, L=10000, tree=True, fastdist=True),
        # the benchmark's many-sequences configuration (an amplicon survey)
        dict(name="resident_dna_k2p_50000x1000", kind="resident", type="dna", model="kim",
             n=50000, L=1000, tree=True, fastdist=True),
        # the benchmark's protein configuration
        dict(name="resident_protein_kim_5000x1500", kind="resident", type="protein", model="kim",
             n=5000, L=1500, tree=True, fastdist=True),
        # rapidNJ's -f: the naive counting rules, ragged sizes
        dict(name="resident_dna_naive_3001x4003", kind="resident", type="dna", model="kim",
             n=3001, L=4003, tree=True, fastdist=False),
        # one matrix from host bytes to host rows, ragged sizes, page-locked buffers
        dict(name="host_dna_k2p_6001x4003", kind="host", type="dna", model="kim", n=6001, L=4003,
             tree=True, pinned=True),
        # the benchmark's batch: 256 gene families, 70 % DNA Kimura-2P, 30 % protein Kimura
        dict(name="batch_256", kind="batch", count=256, n_low=32, n_high=2048, l_low=300,
             l_high=5000, dna_share=0.7),
        # the benchmark's bootstrap configuration
        dict(name="bootstrap_100x2000x2000", kind="bootstrap", type="dna", model="kim", n=2000,
             L=2000, replicates=100),
        # the set-up of the join loops over a 10,000-sequence matrix
        dict(name="nj_10000", kind="nj", n=10000, L=1000),
        # the matrix in double precision
        dict(name="f64_dna_k2p_4000x3001", kind="f64", type="dna", model="kim", n=4000, L=3001,
             tree=True),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["resident", "resident", "resident", "naive", "host", "batch", "bootstrap",
                       "nj", "f64"])
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(16, 256), n_low=32, n_high=_log_int(rng, 256, 2048),
                    l_low=200, l_high=_log_int(rng, 1000, 5000),
                    dna_share=round(rng.uniform(0.3, 1.0), 2))
    if kind == "nj":
        return dict(kind=kind, n=_log_int(rng, 64, 12000), L=_log_int(rng, 200, 1000))
    if kind == "bootstrap":
        return dict(kind=kind, type=rng.choice(["dna", "dna", "protein"]), model="kim",
                    n=_log_int(rng, 32, 1500), L=_log_int(rng, 200, 2500),
                    replicates=rng.randint(10, 100))
    type_ = "dna" if kind == "naive" else rng.choice(["dna", "dna", "protein"])
    model = rng.choice(["kim", "kim", "jc"])
    n_high = {"resident": 40000, "naive": 4000, "host": 8000, "f64": 5000}[kind]
    if type_ == "protein":
        n_high = min(n_high, 8000)
    work = 4e10 if type_ == "protein" or kind in ("naive", "f64") else 8e11  # n * n * L at most
    n = _log_int(rng, 16, n_high)
    L = min(_log_int(rng, 64, 16000), max(64, int(work / n / n)))
    case = dict(kind="resident" if kind == "naive" else kind, type=type_, model=model, n=n, L=L,
                tree=rng.random() < 0.8)
    if kind == "host":
        case["pinned"] = rng.random() < 0.5
    elif kind != "f64":
        case["fastdist"] = kind != "naive"
    return case


# ------------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=1)
def _context():
    return api.Context(0)


def _substituted(codes, gen, mean, protein):
    """One branch of length ~ Exp(mean) under every row of ``codes``."""
    rows = codes.shape[0]
    t = torch.empty((rows, 1), device=DEVICE).exponential_(1.0 / mean, generator=gen)
    u = torch.rand(codes.shape, device=DEVICE, generator=gen)
    if protein:
        p = 0.95 * (1.0 - torch.exp(-t / 0.95))
        shift = 1 + (u / p * 19.0).clamp_(max=18.999).to(torch.uint8)
        return torch.where(u < p, (codes + shift) % 20, codes)
    # Kimura-2P with kappa = 4 (beta = 1/6, alpha = 2/3)
    e1, e2 = torch.exp(-4.0 / 6.0 * t), torch.exp(-2.0 * (5.0 / 6.0) * t)
    ts, tv = 0.25 + 0.25 * e1 - 0.5 * e2, 0.5 - 0.5 * e1
    flip = (u < ts + tv).to(torch.uint8) * 3
    flip -= (u < ts + 0.5 * tv).to(torch.uint8)
    flip -= (u < ts).to(torch.uint8)
    return codes ^ flip


def _alignment(n, L, protein, tree, gen):
    """n x L bytes on the device."""
    if tree:
        codes = torch.randint(0, 20 if protein else 4, (1, L), device=DEVICE, generator=gen,
                              dtype=torch.uint8)
        while codes.shape[0] < n:
            codes = codes.repeat(2, 1)[:n]
            codes = _substituted(codes, gen, 0.05 if protein else 0.02, protein)
        codes = codes[torch.randperm(n, device=DEVICE, generator=gen)]
    else:
        codes = torch.randint(0, 20 if protein else 4, (n, L), device=DEVICE, generator=gen,
                              dtype=torch.uint8)
    gaps = torch.rand((n, L), device=DEVICE, generator=gen) < (0.08 if protein else 0.03)
    letters = torch.from_numpy(AMINO if protein else DNA).to(DEVICE)
    out = torch.empty((n, L), dtype=torch.uint8, device=DEVICE)
    step = max(1, (1 << 28) // max(L, 1))
    for i in range(0, n, step):
        out[i:i + step] = letters[codes[i:i + step].int()]
    return out.masked_fill_(gaps, GAP)


def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _family(case, seed):
    return _alignment(case["n"], case["L"], case["type"] == "protein", case.get("tree", True),
                      _gen(seed))


def _batch_members(case, seed):
    """[(type, n, L)] of a batch; the sizes are the case's, the residues the seed's."""
    rng = np.random.default_rng(case["count"] * 7919 + case["n_high"])
    out = []
    for _ in range(case["count"]):
        n = int(rng.integers(case["n_low"], case["n_high"] + 1))
        L = int(rng.integers(case["l_low"], case["l_high"] + 1))
        out.append(("dna" if rng.random() < case["dna_share"] else "protein", n, L))
    return out


def _batch_alignments(case, seed):
    gen = _gen(seed)
    return [(t, _alignment(n, L, t == "protein", True, gen))
            for t, n, L in _batch_members(case, seed)]


def _nj_matrix(case, seed):
    """A Jukes-Cantor distance matrix as the distance step leaves it: symmetric,
    zero diagonal, with the ties that equal counts give."""
    n, L = case["n"], case["L"]
    chars = _alignment(n, L, False, True, _gen(seed))
    hot = torch.cat([chars == int(c) for c in DNA], 1).float()
    same = hot @ hot.T
    p = (1.0 - same / L).clamp_(0.0, 0.74)
    d = -0.75 * torch.log1p(-p / 0.75)
    d = torch.triu(d, 1)
    return d + d.T


def _replicate_columns(case, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(0, case["L"], size=(case["replicates"], case["L"]), dtype=np.int32)


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    state = dict(case=case, ctx=ctx)
    if kind == "nj":
        n = case["n"]
        state["matrix"] = _nj_matrix(case, seed)
        state["sorted"] = torch.zeros((n, max(1, n - 1), 2), dtype=torch.int32, device=DEVICE)
        return state
    if kind == "batch":
        members = _batch_alignments(case, seed)
        sizes = [s.shape[0] for _, s in members]
        flat = torch.zeros(sum(n * n for n in sizes), dtype=torch.float32, device=DEVICE)
        outs, at = [], 0
        for n in sizes:
            outs.append(flat[at:at + n * n].view(n, n))
            at += n * n
        tiles = sum((-(-n // 128)) * (-(-n // 128) + 1) // 2 for n in sizes)
        state.update(types=[t for t, _ in members], seqs=[s for _, s in members], flat=flat,
                     outs=outs, batch=api.Batch(ctx, max_alignments=len(members),
                                                max_tiles=tiles))
        return state
    chars = _family(case, seed)
    n = case["n"]
    if kind == "host":
        host = chars.cpu()
        out = torch.zeros((n, n), dtype=torch.float32)
        if case["pinned"]:
            host, out = host.pin_memory(), out.pin_memory()
        state.update(keep=(host, out), seqs=host.numpy(), out=out.numpy())
    elif kind == "bootstrap":
        outs = torch.zeros((case["replicates"], n, n), dtype=torch.float32, device=DEVICE)
        state.update(chars=chars, columns=_replicate_columns(case, seed), stack=outs,
                     outs=list(outs.unbind(0)))
    else:
        dtype = torch.float64 if kind == "f64" else torch.float32
        state.update(chars=chars, out=torch.zeros((n, n), dtype=dtype, device=DEVICE))
    return state


# ------------------------------------------------------------------ the call

def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "resident":
        aln = ctx.alignment(state["chars"], case["type"], fastdist=case["fastdist"])
        ctx.distance_into(aln, case["model"], state["out"])
        return state["out"]
    if kind == "host":
        out, largest = ctx.distance_matrix_host(state["seqs"], case["model"], case["type"],
                                                out=state["out"])
        return {"matrix": out, "max": largest}
    if kind == "batch":
        batch = state["batch"]
        batch.clear()
        batch.add_many(state["seqs"], state["types"], ["kim"] * len(state["seqs"]), state["outs"])
        batch.run()
        return state["flat"]
    if kind == "bootstrap":
        _, largest = ctx.bootstrap(state["chars"], state["columns"], case["type"], case["model"],
                                   outs=state["outs"])
        return {"matrices": state["stack"], "max": largest}
    if kind == "nj":
        return ctx.nj_init(state["matrix"], sorted_out=state["sorted"])
    aln = ctx.alignment(state["chars"], case["type"])
    out, largest = ctx.distance_f64(aln, case["model"], state["out"])
    return {"matrix": out, "max": largest}


# ------------------------------------------------------------------ its work

def _pair_work(n, L, type_, out_bytes=4):
    """Bytes in and out, and the multiply-adds of the pair counts: a Gram matrix of
    4 features a site for DNA (valid, ring class, two of the identity), of 21 for
    protein (valid, one for each of 20 residues)."""
    pairs = n * (n - 1) / 2
    return (n * L + n * n * out_bytes, 2.0 * (4 if type_ == "dna" else 21) * pairs * L)


def work(case):
    kind = case["kind"]
    if kind == "nj":
        n = case["n"]
        return {"bytes": n * n * 4 + n * (n - 1) / 2 * 8, "flops": float(n) * n}
    if kind == "batch":
        parts = [_pair_work(n, L, t) for t, n, L in _batch_members(case, 0)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    b, f = _pair_work(case["n"], case["L"], case["type"], 8 if kind == "f64" else 4)
    if kind == "bootstrap":
        n, L, r = case["n"], case["L"], case["replicates"]
        return {"bytes": n * L + 4 * r * L + 4.0 * r * n * n, "flops": f * r}
    return {"bytes": b, "flops": f}


# -------------------------------------------------- the same in plain torch

PAM = (  # Dayhoff distances x 100 of p = 0.750 .. 0.930 (rapidNJ KimuraDistance.cpp:30-49)
    195, 196, 197, 198, 199, 200, 200, 201, 202, 203, 204, 205, 206, 207, 208, 209, 209, 210, 211,
    212, 213, 214, 215, 216, 217, 218, 219, 220, 221, 222, 223, 224, 226, 227, 228, 229, 230, 231,
    232, 233, 234, 236, 237, 238, 239, 240, 241, 243, 244, 245, 246, 248, 249, 250, 252, 253, 254,
    255, 257, 258, 260, 261, 262, 264, 265, 267, 268, 270, 271, 273, 274, 276, 277, 279, 281, 282,
    284, 285, 287, 289, 291, 292, 294, 296, 298, 299, 301, 303, 305, 307, 309, 311, 313, 315, 317,
    319, 321, 323, 325, 328, 330, 332, 335, 337, 339, 342, 344, 347, 349, 352, 354, 357, 360, 362,
    365, 368, 371, 374, 377, 380, 383, 386, 389, 393, 396, 399, 403, 407, 410, 414, 418, 422, 426,
    430, 434, 438, 442, 447, 451, 456, 461, 466, 471, 476, 482, 487, 493, 498, 504, 511, 517, 524,
    531, 538, 545, 553, 560, 569, 577, 586, 595, 605, 615, 626, 637, 649, 661, 675, 688, 703, 719,
    736, 754, 775, 796, 819, 845, 874, 907, 945, 988)


def _exact_rows(hot, classes, valid, i0, i1, type_, model):
    """Distances of rows i0 .. i1 - 1 in 64 bits, -1 for saturated pairs.  Quotients
    are the floats that rapidNJ's distances are defined on."""
    V = (valid[i0:i1] @ valid.T).double()
    same = (hot[i0:i1] @ hot.T).double()
    if model == "jc":
        b = 0.95 if type_ == "protein" else 0.75
        p = torch.where(V > 0, (V - same).float() / V.float(), 0.0).double() / b
        return torch.where(p >= 1.0, -1.0, -b * torch.log(1.0 - p.clamp(max=1.0 - 1e-12)))
    if type_ == "protein":
        p32 = torch.where(V > 0, (V - same).float() / V.float(), -1.0)
        p = p32.double()
        d = -torch.log((1.0 - p - 0.2 * (p32 * p32).double()).clamp(min=1e-12))
        table = torch.tensor(PAM, dtype=torch.float64, device=p.device) / 100.0
        at = (p * 1000.0 - 750.0).clamp(0.0, 180.0).long()
        d = torch.where(p >= 0.75, table[at], d)
        d = torch.where(p > 0.930, 10.0, d)
        return torch.where(p > 0.0, d, p)
    ring = (classes[i0:i1] @ classes.T).double()
    ts = ((ring - same) / V).float().double()
    tv = ((V - ring) / V).float().double()
    a, b = 1.0 - 2.0 * ts - tv, 1.0 - 2.0 * tv
    ok = (V > 0) & (a > 0) & (b > 0)
    d = -0.5 * torch.log(torch.where(ok, a, 1.0)) - 0.25 * torch.log(torch.where(ok, b, 1.0))
    return torch.where(ok, d, -1.0)


def _exact_matrix(chars, type_, model):
    """(matrix in 64 bits, its maximum before saturated pairs are replaced).  The
    alignments hold upper-case letters and '-', for which the fast and the naive
    counting rules agree."""
    n = chars.shape[0]
    letters = AMINO if type_ == "protein" else DNA
    one = [(chars == int(c)) for c in letters]
    valid = torch.stack(one).any(0).float()
    hot = torch.cat(one, 1).float()
    classes = None
    if type_ == "dna":
        classes = torch.cat([one[0] | one[1], one[2] | one[3]], 1).float()
    del one
    out = torch.empty((n, n), dtype=torch.float64, device=chars.device)
    step = max(1, min(n, (1 << 26) // n))
    for i in range(0, n, step):
        out[i:i + step] = _exact_rows(hot, classes, valid, i, min(n, i + step), type_, model)
    out.fill_diagonal_(0.0)
    largest = max(0.0, max(float(out[i:i + step].max()) for i in range(0, n, step)))
    for i in range(0, n, step):
        rows = out[i:i + step]
        rows[rows == -1.0] = 2.0 * largest
    return out, largest


def exact(case, seed):
    kind = case["kind"]
    if kind == "nj":
        n = case["n"]
        sums = _nj_matrix(case, seed).double().sum(1).cpu().numpy()
        sep = sums / (n - 2)
        running = np.maximum.accumulate(np.concatenate([[np.finfo(np.float32).tiny], sep]))
        return {"separation_sums": sums, "separations": sep, "max_row_separations": running[:-1],
                "max_separation": float(running[-1]), "possible_redundant": None,
                "index_to_id": None, "redundant_to_master": None, "redundant_count": None,
                "row_lengths": None, "sorted": None, "sorted_distances": None}
    if kind == "batch":
        return torch.cat([_exact_matrix(s, t, "kim")[0].reshape(-1)
                          for t, s in _batch_alignments(case, seed)])
    chars = _family(case, seed)
    if kind == "bootstrap":
        cols = torch.from_numpy(_replicate_columns(case, seed)).to(DEVICE).long()
        got = [_exact_matrix(chars[:, c], case["type"], case["model"]) for c in cols]
        return {"matrices": torch.stack([m for m, _ in got]), "max": np.array([x for _, x in got])}
    out, largest = _exact_matrix(chars, case["type"], case["model"])
    return out if kind == "resident" else {"matrix": out, "max": largest}
