"""The work a user of sseqs_b200 has it do, as cases that can be timed.

Each case goes through the package's public entry points.  Databases are the
synthetic ones of the benchmark (log-normal lengths, median 250, clipped to
30..1000, a few planted homologs per query); query lengths follow the
benchmark's 50..1000 and, beyond, the package's limit of 2048.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

from sseqs_b200 import batched, conv, dbtools, learned, to_a3m
from sseqs_b200.database import Database

msa = importlib.import_module("sseqs_b200.msa")
sw = importlib.import_module("sseqs_b200.sw")

MEAN_LEN = 296            # mean of the clipped log-normal lengths
GELU_C = 0.7978845608


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest call: a short list of sequences scored against a query
        {"name": "score_list", "kind": "score_list", "qlen": 150, "n": 64},
        # one query searched exactly in a small database (the benchmark's
        # small configuration: 100k sequences, 200 residues, top 100)
        {"name": "exact_small", "kind": "exact", "qlen": 200, "seqs": 100_000, "top": 100},
        # one long query searched exactly in one large resident batch, its
        # best 4096 segments kept (the benchmark's headline step)
        {"name": "exact_large", "kind": "exact_batch", "qlen": 858, "seqs": 500_000, "top": 4096},
        # one query at msa()'s default settings: prefilter, linear and affine
        # scoring, over four batches of the default size
        {"name": "defaults", "kind": "defaults", "qlen": 301, "batches": 4, "bs": 50_000_000},
        # the prefilter alone on one resident batch, at the benchmark's
        # longest listed query
        {"name": "prefilter", "kind": "prefilter", "qlen": 858, "seqs": 300_000, "rank": 4},
        # and for a query beyond 1024 residues (transform length 2048), an
        # odd length and rank
        {"name": "prefilter_long", "kind": "prefilter", "qlen": 1501, "seqs": 100_000, "rank": 3},
        # a set of queries of uneven lengths against one resident database
        {"name": "batched", "kind": "batched", "queries": 12, "seqs": 60_000, "top": 4096},
        # the second half of msa(): hits aligned and written as a3m rows
        {"name": "a3m", "kind": "a3m", "qlen": 413, "n": 2048},
        # a packed chunk decoded into a resident batch with its tables
        {"name": "load", "kind": "load", "bs": 50_000_000},
        # sequences embedded for the learned index
        {"name": "embed", "kind": "embed", "n": 20_000},
        # one training step of the embedder: forward and backward
        {"name": "train_step", "kind": "train", "queries": 32, "targets": 32},
        # queries through the learned index: candidates, then exact scores
        {"name": "learned_search", "kind": "learned", "queries": 8, "seqs": 400_000,
         "cand": 32768, "dim": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["score_list", "exact", "exact_batch", "defaults", "prefilter", "prefilter",
                       "batched", "a3m", "load", "embed", "train", "learned"])
    if kind == "score_list":
        return {"kind": kind, "qlen": _log(rng, 40, 1000), "n": _log(rng, 1, 2000)}
    if kind == "exact":
        return {"kind": kind, "qlen": rng.randint(50, 1000), "seqs": _log(rng, 3000, 150_000),
                "top": _log(rng, 50, 4096)}
    if kind == "exact_batch":
        return {"kind": kind, "qlen": rng.randint(50, 850), "seqs": _log(rng, 30_000, 500_000),
                "top": rng.choice([100, 1000, 4096])}
    if kind == "defaults":
        return {"kind": kind, "qlen": rng.randint(50, 1000), "batches": rng.randint(1, 4),
                "bs": 5_000_000 * rng.randint(1, 10)}
    if kind == "prefilter":
        return {"kind": kind, "qlen": rng.choice([rng.randint(50, 1000), rng.randint(50, 1000),
                                                  rng.randint(1025, 2000)]),
                "seqs": _log(rng, 2000, 300_000), "rank": rng.choice([1, 2, 3, 4, 4, 4])}
    if kind == "batched":
        return {"kind": kind, "queries": rng.randint(2, 12), "seqs": _log(rng, 5000, 60_000),
                "top": _log(rng, 100, 4096)}
    if kind == "a3m":
        return {"kind": kind, "qlen": rng.randint(50, 1000), "n": _log(rng, 16, 2048)}
    if kind == "load":
        return {"kind": kind, "bs": 5 * _log(rng, 100_000, 20_000_000)}
    if kind == "embed":
        return {"kind": kind, "n": _log(rng, 200, 60_000)}
    if kind == "train":
        return {"kind": kind, "queries": rng.randint(4, 32), "targets": rng.randint(8, 32)}
    return {"kind": kind, "queries": rng.randint(1, 8), "seqs": _log(rng, 50_000, 400_000),
            "cand": rng.choice([4096, 16384, 32768]), "dim": rng.choice([256, 256, 128])}


# ----------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _chunks(queries, seqs, seed, chunk_bytes):
    frac = max(1, seqs // 2000) / seqs
    frac = min(frac, 0.5 / max(1, len(queries)))
    return dbtools.synthetic_db(queries, seqs, frac, (0.2, 0.95), seed=seed, device="cuda",
                                chunk_bytes=chunk_bytes).chunks


def _database(queries, seqs, seed):
    """One batch holding all ``seqs`` sequences."""
    size = (int(seqs * (MEAN_LEN + 20) * 5 / 8) // 8000 + 60) * 8000
    return Database(_chunks(queries, seqs, seed, size)[:1], bs=size)


def _packed(size, seed):
    """One packed chunk of ``size`` bytes, nearly full: sequences whose
    lengths are the same for every seed, in an order of its own."""
    lens = dbtools.lognormal_lengths(max(1, int(size * 8 / 5 / (MEAN_LEN + 1) * 0.95)),
                                     _gen(7), "cuda")
    gen = _gen(seed)
    lens = lens[torch.randperm(lens.numel(), generator=gen, device="cuda")]
    ends = torch.cumsum(lens + 1, 0)
    buf = dbtools.random_residues(int(ends[-1]), gen, "cuda")
    buf[ends - 1] = 64
    return dbtools.assemble_stream(buf, lens, size)[0][0]


def _query(qlen, seed):
    return dbtools.random_query(qlen, seed)


def _strings(buf, lengths):
    raw = buf.cpu().numpy().tobytes().decode()
    ends = np.cumsum(lengths.cpu().numpy())
    return [raw[e - n:e] for e, n in zip(ends.tolist(), lengths.cpu().tolist())]


def _targets(query, n, seed, width=500):
    """Half mutated copies of the query, half unrelated sequences, each cut
    to the ``width`` residues that msa() keeps of a hit, in mixed order."""
    gen = _gen(seed)
    h = (n + 1) // 2
    out = _strings(*dbtools.plant_homologs(query, h, 0.2, 0.95, gen, "cuda"))
    lens = dbtools.lognormal_lengths(n - h, gen, "cuda")
    if n > h:
        out += _strings(dbtools.random_residues(int(lens.sum()), gen, "cuda"), lens)
    order = np.random.default_rng(seed).permutation(n)
    return [out[i][:width] or "A" for i in order]


def _sequences(n, seed):
    """``n`` sequences in one '@'-separated buffer: bytes, offsets, lengths."""
    gen = _gen(seed)
    lens = dbtools.lognormal_lengths(n, gen, "cuda")
    ends = torch.cumsum(lens + 1, 0)
    buf = dbtools.random_residues(int(ends[-1]), gen, "cuda")
    buf[ends - 1] = 64
    return buf, ends - lens - 1, lens.to(torch.int32)


def _query_lengths(n, seed):
    rng = np.random.default_rng(seed)
    return np.clip(np.round(np.exp(rng.normal(math.log(300), 0.6, n))), 16, 2048).astype(int)


def _train_sequences(case, seed):
    """Queries (50..1000 residues) and their targets, half of them homologs."""
    rng = np.random.default_rng(seed)
    gen = _gen(seed)
    parts, lens = [], []
    t = case["targets"]
    for i in range(case["queries"]):
        q = _query(int(rng.integers(50, 1001)), seed * 1000 + i)
        parts.append(torch.tensor(list(q.encode()), dtype=torch.uint8, device="cuda"))
        lens.append(torch.tensor([len(q)], device="cuda"))
        res, ln = dbtools.plant_homologs(q, t // 2, 0.15, 1.0, gen, "cuda")
        bl = dbtools.lognormal_lengths(t - t // 2, gen, "cuda")
        parts += [res, dbtools.random_residues(int(bl.sum()), gen, "cuda")]
        lens += [ln, bl]
    lengths = torch.cat(lens)
    return torch.cat(parts), torch.cumsum(lengths, 0) - lengths, lengths.to(torch.int32)


def _codes(n, dim, gen):
    """FP8 codes of unit vectors with the spread of trained embeddings
    (unrelated pairs have a cosine of about 0.5)."""
    x = torch.randn(n, dim, generator=gen, device="cuda")
    x[:, 0] += math.sqrt(dim)
    x /= x.norm(dim=1, keepdim=True)
    return (learned.CODE_SCALE * x).to(torch.float8_e4m3fn).view(torch.uint8)


def prepare(case, seed):
    k = case["kind"]
    if k == "score_list":
        q = _query(case["qlen"], seed)
        return {"case": case, "query": q, "targets": _targets(q, case["n"], seed, 1000)}
    if k in ("exact", "exact_batch", "prefilter"):
        q = _query(case["qlen"], seed)
        st = {"case": case, "query": q, "db": _database([q], case["seqs"], seed)}
        if k == "exact_batch":
            st["enc"] = sw.encode_query(q)
        if k == "prefilter":
            st["luts"] = conv.prefilter_luts(q, case["rank"])
        return st
    if k == "defaults":
        q = _query(case["qlen"], seed)
        bs, nb = case["bs"], case["batches"]
        seqs = int(bs * nb * 8 / 5 / (MEAN_LEN + 1) * 0.97)
        chunks = _chunks([q], seqs, seed, bs * nb)
        return {"case": case, "query": q, "db": Database(chunks[:1], bs=bs)}
    if k == "batched":
        qs = [_query(int(n), seed * 100 + i)
              for i, n in enumerate(_query_lengths(case["queries"], 11))]
        db = _database(qs, case["seqs"], seed)
        return {"case": case, "queries": qs,
                "searcher": batched.BatchedSearcher(db, top_k=case["top"])}
    if k == "a3m":
        q = _query(case["qlen"], seed)
        return {"case": case, "query": q, "targets": _targets(q, case["n"], seed)}
    if k == "load":
        return {"case": case, "chunk": _packed(case["bs"], seed)}
    if k == "embed":
        buf, off, lens = _sequences(case["n"], seed)
        return {"case": case, "model": learned.Embedder(seed=seed), "buf": buf, "off": off,
                "lens": lens}
    if k == "train":
        buf, off, lens = _train_sequences(case, seed)
        grad = torch.randn(lens.numel(), learned.D, generator=_gen(seed + 1), device="cuda")
        return {"case": case, "model": learned.Embedder(seed=seed), "buf": buf, "off": off,
                "lens": lens, "grad": grad / lens.numel()}
    rng = np.random.default_rng(seed)
    qs = [_query(int(n), seed * 100 + i)
          for i, n in enumerate(rng.integers(50, 1001, case["queries"]))]
    db = _database(qs[:1], case["seqs"], seed)
    index = learned.LearnedIndex(learned.Embedder(seed=seed), db, dim=case["dim"])
    gen = _gen(seed + 2)
    index.codes[:index.n] = _codes(index.n, case["dim"], gen)
    return {"case": case, "queries": qs, "index": index,
            "codes": _codes(len(qs), case["dim"], gen)}


# -------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "score_list":
        return sw.sw(state["query"], state["targets"])
    if k == "exact":
        rows = msa.search(state["query"], state["db"], num_msas=case["top"], top_fft=1, top_sw=1,
                          top_sw_affine=case["top"])[0]
        return _rows(rows)
    if k == "exact_batch":
        b = msa.search_batch(state["enc"], state["query"], state["db"].batches[0], 0, top_fft=1,
                             top_sw=1, top_sw_affine=case["top"])
        return [b.g, b.affine, b.linear, b.hits, b.hit_len]
    if k == "defaults":
        return _rows(msa.search(state["query"], state["db"])[0])
    if k == "prefilter":
        return conv.prefilter_batch(state["query"], state["db"].batches[0], state["luts"],
                                    case["rank"])
    if k == "batched":
        hits = state["searcher"].search(state["queries"])
        return [np.concatenate([getattr(h, f) for h in hits])
                for f in ("scores", "batch", "segment")]
    if k == "a3m":
        text = to_a3m.a3m_text_raw(state["query"],
                                   to_a3m.traceback_all(state["query"], state["targets"]))
        # zero bytes up to the longest text that n rows can make
        size = 2 * case["qlen"] + case["n"] * (case["qlen"] + 540)
        return np.frombuffer(text.encode().ljust(size, b"\0"), np.uint8)
    if k == "load":
        b = Database([state["chunk"]], bs=case["bs"]).batches[0]
        return [b.ascii, b.delim, b.seg_index, b.lengths, b.offsets, b.maxlen, b.n_segments,
                b.n_residues]
    if k == "embed":
        return state["model"].embed(state["buf"], state["off"], state["lens"])
    if k == "train":
        lay = learned.make_layout(state["buf"], state["off"], state["lens"])
        emb = state["model"].forward(lay, train=True)
        g = state["model"].backward(state["grad"])
        return {"emb": emb, "W": g["W"], "b": g["b"], "demb": g["emb"]}
    index = state["index"]
    kq, kr, counts = index.candidates_flat(state["codes"], case["cand"])
    hits = index.rescore_flat(state["queries"], kq, kr)
    return [kq, kr, counts] + [np.concatenate([h[j] for h in hits]) for j in range(4)]


def _rows(rows):
    """The numbers of ranked hits: normalised score, and batch, segment,
    affine and linear score; and the hit strings, padded to their width."""
    return [np.array([r[0] for r in rows], np.float32),
            np.array([r[1:5] for r in rows], np.int64),
            np.frombuffer("".join(r[5].ljust(msa.HIT_WIDTH) for r in rows).encode("latin-1"),
                          np.uint8)]


# ------------------------------------------------------------ work and truth
def work(case):
    """Bytes and operations of one pass: residues, queries and results once;
    2 (linear) and 3.5 (affine) operations per cell, 2 per multiply-add."""
    k = case["kind"]
    L = MEAN_LEN
    if k == "score_list":
        return {"bytes": case["n"] * (L + 4), "flops": 3.5 * case["qlen"] * case["n"] * L}
    if k in ("exact", "exact_batch"):
        n = case["seqs"]
        return {"bytes": n * (L + 4) + case["top"] * 520, "flops": 5.5 * case["qlen"] * n * L}
    if k in ("defaults", "prefilter"):
        n = case["seqs"] if k == "prefilter" else case["bs"] * case["batches"] * 8 / 5 / (L + 1)
        rank = case.get("rank", 4)
        # every even lag's products, summed over the ranks
        return {"bytes": n * (L + 14), "flops": n * case["qlen"] * L * rank}
    if k == "batched":
        cells = int(_query_lengths(case["queries"], 11).sum()) * case["seqs"] * L
        return {"bytes": case["seqs"] * (L + 4) + case["queries"] * case["top"] * 12,
                "flops": 3.5 * cells}
    if k == "a3m":
        t = min(500, (case["qlen"] + L) // 2)
        return {"bytes": case["n"] * (t + case["qlen"] + 32),
                "flops": 5.0 * case["qlen"] * case["n"] * t}
    if k == "load":
        sym = case["bs"] * 8 / 5
        return {"bytes": case["bs"] + sym * (1 + 20 / (L + 1)), "flops": 3 * sym}
    if k in ("embed", "train"):
        n = case["n"] if k == "embed" else case["queries"] * (1 + case["targets"])
        rows = n * (L if k == "embed" else 410)
        mac = 5 * (32 + 3 * 256) * 256
        return {"bytes": rows + 1024 * n + (4 * 1_000_000 if k == "embed" else 12_000_000),
                "flops": 2 * mac * rows * (1 if k == "embed" else 3)}
    nq = case["queries"]
    return {"bytes": case["seqs"] * case["dim"] + nq * case["cand"] * (L / 2 + 16),
            "flops": 2 * nq * case["seqs"] * case["dim"] + 3.5 * 525 * nq * case["cand"] * L}


def _exact_prefilter(case, seed):
    st = prepare(case, seed)
    b, luts = st["db"].batches[0], st["luts"]
    n = 64
    while n < max(len(st["query"]), b.maxlen):
        n *= 2
    pos = torch.full((256,), 21, dtype=torch.int64)
    for i, c in enumerate("ARNDCQEGHILKMFPSTWYV"):
        pos[ord(c)] = i
    for c in "X-*":
        pos[ord(c)] = 20
    pos = pos.cuda()
    k = case["rank"]
    A, B = luts.A[:k].double().cuda(), luts.B[:k].double().cuda()
    # class 21 reads the next rank's first entry (0 for the last rank)
    B = torch.cat([B, torch.cat([B[1:, :1], torch.zeros(1, 1, device="cuda",
                                                        dtype=torch.float64)])], 1)
    fa = torch.fft.rfft(A[:, luts.qrev.long()], n)
    out = torch.empty(b.n_segments, dtype=torch.float64, device="cuda")
    col = torch.arange(n, device="cuda")
    for s in range(0, b.n_segments, 8192):
        off, ln = b.offsets[s:s + 8192], b.lengths[s:s + 8192].long()
        live = col[None, :] < ln[:, None]
        at = (off[:, None] + col[None, :]).clamp(max=b.ascii.numel() - 1)
        cls = pos[b.ascii[at].long()]
        f = 0
        for r in range(k):
            f = f + fa[r][None, :] * torch.fft.rfft(torch.where(live, B[r][cls], 0.0))
        out[s:s + 8192] = 0.5 * torch.fft.irfft(f, n)[:, ::2].amax(1)
    return out


def _net(st, chunk, grad):
    """Embeddings (and with ``grad`` the gradients) in 64 bits."""
    m = st["model"]
    W = [w.double().clone().requires_grad_(grad) for w in m.W]
    bias = [b.double().clone().requires_grad_(grad) for b in m.b]
    table = m.emb.double().clone().requires_grad_(grad)
    pos = torch.full((256,), 20, dtype=torch.int64)
    for i, c in enumerate("ARNDCQEGHILKMFPSTWYV"):
        pos[ord(c)] = i
    cls = pos.cuda()[st["buf"].long()]
    out = []
    for s in range(0, st["lens"].numel(), chunk):
        off, ln = st["off"][s:s + chunk].long(), st["lens"][s:s + chunk].long()
        sizes = ln + 2
        row0 = torch.cumsum(sizes, 0) - sizes + 2
        rows = int(2 + sizes.sum())
        seq = torch.repeat_interleave(torch.arange(ln.numel(), device="cuda"), ln)
        i = torch.arange(seq.numel(), device="cuda") - (torch.cumsum(ln, 0) - ln)[seq]
        at = row0[seq] + i
        x = torch.zeros(rows, learned.E, dtype=torch.float64, device="cuda").index_copy(
            0, at, table[cls[off[seq] + i]])
        keep = torch.zeros(rows, 1, dtype=torch.float64, device="cuda")
        keep[at] = 1
        for l in range(4):
            xp = torch.nn.functional.pad(x, (0, 0, 2, 2))
            z = bias[l] + sum(xp[t:t + rows] @ W[l][:, t].T for t in range(5))
            y = 0.5 * z * (1 + torch.tanh(GELU_C * (z + 0.044715 * z ** 3)))
            x = (y + x if l else y) * keep
        p = torch.zeros(ln.numel(), learned.D, dtype=torch.float64, device="cuda").index_add(
            0, seq, x[at]) / ln[:, None]
        out.append(p / p.norm(dim=1, keepdim=True))
    emb = torch.cat(out)
    if not grad:
        return emb
    (emb * st["grad"].double()).sum().backward()
    return {"emb": emb.detach(),
            "W": [w.grad.permute(1, 2, 0).reshape(-1, learned.D) for w in W],
            "b": [b.grad for b in bias], "demb": table.grad}


def exact(case, seed):
    k = case["kind"]
    if k == "prefilter":
        return _exact_prefilter(case, seed)
    if k == "embed":
        with torch.no_grad():
            return _net(prepare(case, seed), 2000, False)
    if k == "train":
        return _net(prepare(case, seed), 1 << 30, True)
    return None
