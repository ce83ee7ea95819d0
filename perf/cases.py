"""The work that users of this package have it do, as cases that can be timed.

Every case goes through the package's public entry points.  The inputs are
synthetic proteomes made on the GPU from the seed: protein lengths lognormal
(median 300, sigma 0.5), residues from the 20-letter background frequencies,
proteomes related by a binary tree whose branches substitute residues at rates
of U(0.01, 0.2) per site, each protein preceded by one newline (as the FASTA
reader leaves them).  Protein counts and lengths go with the case, residues with
the seed.  Sizes of uneven sets are the quantiles of the lognormal
protein counts (median 1,900, sigma 0.9, clipped to [300, 12,000]) that the
package's benchmark workloads use.

Kinds of case:

* ``build``    one proteome through the drop-in plug-in call
               (CompositionVectorKernels.build_vector_gpu): what the host runtime
               does once per input file;
* ``compare``  one pair of vectors through the drop-in plug-in call
               (CompositionVectorKernels.compare_vectors_gpu): what the host
               runtime does once per pair;
* ``batch``    many proteomes through BatchBuilder into a kept arena;
* ``pairs``    every pair of an indexed arena (PairEngine.run on a kept plan);
* ``query``    a batch of new proteomes built, indexed and compared with every
               vector of a resident database (a serving slot's work);
* ``set``      a whole run: build, key ranks and window index, all pairs.
"""
import math

import numpy as np
import torch

from rocket_gb300.engine import BatchBuilder, EngineConfig, PairEngine, auto_tile_cols
from rocket_gb300.kernels import CompositionVectorKernels

_LETTERS = "ARNDCQEGHILKMFPSTWYV"
_PERMILLE = (83, 55, 41, 55, 14, 39, 67, 71, 23, 59, 99, 58, 24, 39, 47, 65, 53, 11, 29, 68)
_ALPHABET = {"protein": "ACDEFGHIKLMNPQRSTVWYX", "DNA": "ACGT"}
_MEAN_PROTEIN = 300.0 * math.exp(0.125) + 1.0  # bytes per protein, with its newline


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def listed():
    return [
        # a very small input file (a phage, a plasmid): launches and waits are all of it
        dict(name="build_30", kind="build", alphabet="protein", k=6, proteins=30),
        # an ordinary bacterial proteome through the same call
        dict(name="build_1500", kind="build", alphabet="protein", k=6, proteins=1500),
        # two short vectors: the latency of the per-pair call
        dict(name="compare_30", kind="compare", alphabet="protein", k=6, left=30, right=41),
        # two vectors of ordinary size, millions of entries each
        dict(name="compare_2000", kind="compare", alphabet="protein", k=6, left=1900, right=2130),
        # batched construction of proteomes of very uneven sizes, the usual K
        dict(name="batch_uneven_k6", kind="batch", alphabet="protein", k=6, n=64, proteins=0),
        # the same at the largest protein K
        dict(name="batch_uneven_k7", kind="batch", alphabet="protein", k=7, n=29, proteins=0),
        # genomes over the DNA alphabet at its largest K, a million bases each
        dict(name="batch_dna_k10", kind="batch", alphabet="DNA", k=10, n=16, proteins=3300),
        # all pairs of a uniform set, K = 6
        dict(name="pairs_uniform_k6", kind="pairs", alphabet="protein", k=6, n=128, proteins=1500),
        # all pairs of an uneven set at K = 7, where vectors share few keys
        dict(name="pairs_uneven_k7", kind="pairs", alphabet="protein", k=7, n=93, proteins=0),
        # a query batch against a resident database
        dict(name="query_24_of_160", kind="query", alphabet="protein", k=6, n=24, db=160,
             proteins=0),
        # a small whole run: 16 proteomes of 1,500 proteins
        dict(name="set_16", kind="set", alphabet="protein", k=6, n=16, proteins=1500),
        # a large whole run: 512 proteomes of uneven sizes
        dict(name="set_uneven_512", kind="set", alphabet="protein", k=6, n=512, proteins=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _alphabet_k(rng):
    alphabet = rng.choice(["protein", "protein", "protein", "DNA"])
    return alphabet, (rng.choice([5, 6, 6, 7]) if alphabet == "protein" else rng.randint(6, 10))


def draw(rng):
    kind = rng.choice(["build", "compare", "batch", "pairs", "query", "set"])
    alphabet, k = _alphabet_k(rng)
    c = dict(kind=kind, alphabet=alphabet, k=k)
    if kind == "build":
        c["proteins"] = _log_int(rng, 10, 9000)
    elif kind == "compare":
        c["left"], c["right"] = _log_int(rng, 10, 9000), _log_int(rng, 10, 9000)
    elif kind == "batch":
        c["n"] = _log_int(rng, 2, 70)
        c["proteins"] = 0 if rng.random() < 0.5 else _log_int(rng, 30, 2500)
    elif kind == "pairs":
        c["n"] = _log_int(rng, 5, 130)
        c["proteins"] = 0 if rng.random() < 0.5 else _log_int(rng, 100, 1600)
    elif kind == "query":
        c["n"], c["db"] = _log_int(rng, 1, 40), _log_int(rng, 20, 170)
        c["proteins"] = 0 if rng.random() < 0.5 else _log_int(rng, 100, 1600)
    else:
        c["n"] = _log_int(rng, 4, 200)
        c["proteins"] = 0 if rng.random() < 0.5 else _log_int(rng, 100, 2000)
    return c


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _quantile(p):
    """Standard normal quantile by bisection of erf (a few hundred values at most)."""
    lo, hi = -8.0, 8.0
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        if 0.5 * (1.0 + math.erf(mid / math.sqrt(2.0))) < p:
            lo = mid
        else:
            hi = mid
    return 0.5 * (lo + hi)


def _counts(n, proteins):
    """Protein counts of n proteomes: all ``proteins``, or (0) the shuffled quantiles of
    the uneven sets' lognormal."""
    if proteins:
        return [proteins] * n
    q = [min(12000, max(300, round(1900.0 * math.exp(0.9 * _quantile((i + 0.5) / n)))))
         for i in range(n)]
    order = np.random.RandomState(n).permutation(n)
    return [int(q[i]) for i in order]


def _case_counts(c):
    if c["kind"] == "build":
        return [c["proteins"]]
    if c["kind"] == "compare":
        return [c["left"], c["right"]]
    n = c["n"] + (c["db"] if c["kind"] == "query" else 0)
    return _counts(n, c["proteins"])


def _generate(counts, seed, alphabet):
    """(residues uint8 on the GPU, offsets int64 on the host) of related proteomes; leaf i
    is leaf (i - 1) // 2 with substitutions, cut to its first counts[i] proteins."""
    rs = np.random.RandomState(seed % (1 << 31))
    most = max(counts)
    z = np.random.RandomState(most).standard_normal(most)  # lengths go with the sizes, not the seed
    lens = np.maximum(np.round(300.0 * np.exp(0.5 * z)), 1).astype(np.int64)
    ends = np.concatenate([[0], np.cumsum(lens + 1)])
    total = int(ends[-1])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if alphabet == "protein":
        letters = "".join(a * m for a, m in zip(_LETTERS, _PERMILLE))
    else:
        letters = "A" * 250 + "C" * 250 + "G" * 250 + "T" * 250
    table = torch.tensor(list(letters.encode()), dtype=torch.uint8, device="cuda")

    def residues():
        return table[torch.randint(0, len(letters), (total,), generator=gen, device="cuda")]

    newline = torch.zeros(total, dtype=torch.bool, device="cuda")
    newline[torch.from_numpy(ends[:-1]).cuda()] = True
    root = residues()
    root[newline] = 10
    sizes = [int(ends[m]) for m in counts]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    out = torch.empty(int(off[-1]), dtype=torch.uint8, device="cuda")
    parents = []
    for i in range(len(counts)):
        if i == 0:
            leaf = root
        else:
            rate = rs.uniform(0.01, 0.2)
            hit = torch.rand(total, generator=gen, device="cuda") < rate
            hit &= ~newline
            leaf = torch.where(hit, residues(), parents[(i - 1) // 2])
        parents.append(leaf if 2 * i + 1 < len(counts) else None)
        if i > 0 and i % 2 == 0:
            parents[(i - 1) // 2] = None  # both children made
        out[int(off[i]):int(off[i + 1])] = leaf[:sizes[i]]
    return out, off


def _max_entries(residues, alphabet, k):
    """The vector size a user of the plug-in sets aside for a proteome."""
    return min(len(_ALPHABET[alphabet]) ** k, 8 * residues + 1024)


def _arena(builder, off):
    lens = np.diff(off)
    arena = builder.new_arena(int(np.sum(8 * lens + 64)) + 1024, len(lens))
    arena.keys.zero_()
    arena.values.zero_()
    return arena


def prepare(case, seed):
    c = dict(case)
    alphabet, k = c["alphabet"], c["k"]
    counts = _case_counts(c)
    seq, off = _generate(counts, seed, alphabet)
    st = dict(case=c, seq=seq, off=off)
    if c["kind"] == "build":
        n = int(off[-1])
        size = _max_entries(n, alphabet, k)
        st["kernels"] = CompositionVectorKernels(alphabet, k, size, n)
        st["keys"] = torch.empty(size, dtype=torch.int32, device="cuda")
        st["values"] = torch.empty(size, dtype=torch.float32, device="cuda")
    elif c["kind"] == "compare":
        size = _max_entries(int(np.max(np.diff(off))), alphabet, k)
        ker = CompositionVectorKernels(alphabet, k, size, int(np.max(np.diff(off))))
        keys = torch.empty((2, size), dtype=torch.int32, device="cuda")
        vals = torch.empty((2, size), dtype=torch.float32, device="cuda")
        n = [ker.build_vector_gpu(seq[int(off[i]):int(off[i + 1])], keys[i], vals[i])
             for i in range(2)]
        st["kernels"] = ker
        st["vectors"] = [(keys[i, :n[i]], vals[i, :n[i]], n[i]) for i in range(2)]
        st["out"] = torch.zeros(1, dtype=torch.float64, device="cuda")
    elif c["kind"] == "query":
        db_n = c["db"]
        cut = int(off[db_n])
        cfg = EngineConfig(segments=16, compress=False)
        db = BatchBuilder(alphabet, k).build(seq[:cut], off[:db_n + 1])
        PairEngine(db, cfg).ensure_index()
        st["db"] = db
        st["seq"] = seq[cut:].clone()
        st["off"] = off[db_n:] - cut
        st["builder"] = BatchBuilder(alphabet, k, max_batch=64)
        st["arena"] = _arena(st["builder"], st["off"])
        st["engine"] = PairEngine(st["arena"], cfg)
        st["out"] = torch.zeros((c["n"], db_n), dtype=torch.float64, device="cuda")
    else:
        n = c["n"]
        st["builder"] = BatchBuilder(alphabet, k)
        st["arena"] = _arena(st["builder"], off)
        if c["kind"] != "batch":
            st["out"] = torch.zeros((n, n), dtype=torch.float64, device="cuda")
            st["engine"] = PairEngine(st["arena"], EngineConfig(tile_cols=auto_tile_cols(n)))
        if c["kind"] == "pairs":
            st["builder"].build(seq, off, arena=st["arena"])
            st["engine"].ensure_index()
            st["plan"] = st["engine"].plan_triangle()
    return st


def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "build":
        n = st["kernels"].build_vector_gpu(st["seq"], st["keys"], st["values"])
        return {"size": n, "keys": st["keys"], "values": st["values"]}
    if kind == "compare":
        (ka, va, na), (kb, vb, nb) = st["vectors"]
        st["kernels"].compare_vectors_gpu(ka, va, na, kb, vb, nb, st["out"])
        return {"c": st["out"]}
    if kind == "pairs":
        st["engine"].run(st["plan"], st["out"])
        return {"c": st["out"]}
    arena = st["builder"].build(st["seq"], st["off"], arena=st["arena"].reset())
    if kind == "batch":
        return {"keys": arena.keys, "values": arena.values, "offsets": arena.vec_off,
                "nnz": arena.nnz}
    eng = st["engine"]
    eng.arena = arena
    eng.ensure_index()
    if kind == "query":
        plan = eng.plan_rect(np.arange(c["n"]), np.arange(c["db"]), ldc=c["db"],
                             col_arena=st["db"])
        eng.run(plan, st["out"], diagonal=False, col_arena=st["db"])
    else:
        eng.run(eng.plan_triangle(), st["out"])
    return {"c": st["out"]}


# --------------------------------------------------------------------------
# work: what a pass cannot do without
# --------------------------------------------------------------------------

# entries of a composition vector per residue, by number of residues (measured on such
# proteomes; between the points interpolated in the logarithm of the residues)
_ENTRIES = {
    ("protein", 5): ((3e3, 1.2), (1e4, 1.9), (1e5, 4.6), (4.8e5, 3.6), (1e6, 2.3), (4e6, 0.8)),
    ("protein", 6): ((3e3, 1.0), (1e4, 1.2), (1e5, 2.4), (4.8e5, 5.0), (1e6, 5.7), (4e6, 5.9)),
    ("protein", 7): ((3e3, 1.0), (1e4, 1.0), (1e5, 1.1), (4.8e5, 1.5), (1e6, 1.8), (4e6, 3.0)),
}


def _entries(residues, alphabet, k):
    if alphabet == "DNA":
        return min(4.0 ** k, 3.0 * residues)
    pts = _ENTRIES[(alphabet, k)]
    x = [math.log(a) for a, _ in pts]
    return residues * float(np.interp(math.log(max(residues, 1.0)), x, [b for _, b in pts]))


def work(case):
    c = dict(case)
    res = [_MEAN_PROTEIN * m for m in _case_counts(c)]
    nnz = [_entries(r, c["alphabet"], c["k"]) for r in res]
    space = float(len(_ALPHABET[c["alphabet"]]) ** c["k"])
    build = sum(res) + 8.0 * sum(nnz)      # residues in, keys and values out
    build_ops = 3.0 * sum(res) + 12.0 * sum(nnz)

    def products(a, b):                    # keys of both vectors, if unrelated, at least
        return a * b / space

    if c["kind"] in ("build", "batch"):
        return {"bytes": build, "flops": build_ops}
    if c["kind"] == "compare":
        return {"bytes": 8.0 * sum(nnz) + 8.0, "flops": 2.0 * products(*nnz)}
    if c["kind"] == "query":
        db, q = nnz[:c["db"]], nnz[c["db"]:]
        b = sum(res[c["db"]:]) + 16.0 * sum(q) + 8.0 * sum(db) + 8.0 * len(q) * len(db)
        return {"bytes": b, "flops": 2.0 * products(sum(q), sum(db)) + 12.0 * sum(q)}
    n = len(nnz)
    pair_ops = products(sum(nnz), sum(nnz))
    pair_bytes = 8.0 * sum(nnz) + 8.0 * n * n
    if c["kind"] == "pairs":
        return {"bytes": pair_bytes, "flops": pair_ops}
    return {"bytes": build + pair_bytes, "flops": build_ops + pair_ops}


# --------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# --------------------------------------------------------------------------

def _windows(d, k, A):
    """Codes of the windows of k valid symbols that start at each position."""
    n = d.numel() - k + 1
    if n <= 0:
        return torch.zeros(0, dtype=torch.int64, device=d.device)
    code = torch.zeros(n, dtype=torch.int64, device=d.device)
    ok = torch.ones(n, dtype=torch.bool, device=d.device)
    for j in range(k):
        x = d[j:j + n]
        code = code * A + x
        ok &= x >= 0
    return code[ok]


def _lookup(keys, counts, at):
    """counts of the codes ``at`` (0 where a code is not among the sorted ``keys``)."""
    i = torch.searchsorted(keys, at).clamp_(max=max(keys.numel() - 1, 0))
    return torch.where(keys[i] == at, counts[i], torch.zeros_like(counts[i]))


def _alpha(seq, alphabet, k):
    """(keys int64 ascending, alpha float64) of one proteome: alpha = (p - p0) / p0 with
    p0 = p(prefix) p(suffix) / p(middle), over the K-mers whose prefix and suffix occur."""
    symbols = _ALPHABET[alphabet]
    A = len(symbols)
    digit = torch.full((256,), -1, dtype=torch.int64, device=seq.device)
    for i, ch in enumerate(symbols):
        digit[ord(ch)] = i
    d = digit[seq.long()]
    c = [torch.unique(_windows(d, k - j, A), return_counts=True) for j in range(3)]
    n0, n1, n2 = (float(x[1].sum()) for x in c)
    (k0, c0), (k1, c1), (k2, c2) = c
    mid = k1 % (A ** (k - 2))
    lo = torch.searchsorted(k1, mid * A)
    num = torch.searchsorted(k1, mid * A + A) - lo
    own = torch.repeat_interleave(torch.arange(k1.numel(), device=seq.device), num)
    suf = torch.arange(own.numel(), device=seq.device) - (torch.cumsum(num, 0) - num)[own] + lo[own]
    keys = k1[own] * A + k1[suf] % A
    full = _lookup(k0, c0, keys).double()
    middle = _lookup(k2, c2, mid)[own].double()
    p0 = (c1[own].double() / n1) * (c1[suf].double() / n1) / (middle / n2)
    a = (full / n0 - p0) / p0
    keep = a.float() != 0
    return keys[keep], a[keep]


def _vector32(seq, alphabet, k):
    """The composition vector in the precision it is kept in (float values)."""
    keys, a = _alpha(seq, alphabet, k)
    a = a.float()
    return keys, (a.double() / torch.sqrt((a * a).double().sum())).float()


def _products(vectors, rows):
    """Products (64 bits) of the first ``rows`` vectors with all others (rows = 0: of
    every vector with every vector)."""
    union, rank = torch.unique(torch.cat([v[0] for v in vectors]), return_inverse=True)
    ranks = torch.split(rank, [v[0].numel() for v in vectors])
    n, U, step = len(vectors), union.numel(), 1 << 20
    del union
    out = torch.zeros((rows or n, n - rows), dtype=torch.float64, device="cuda")
    cuts = torch.arange(0, U + step, step, device="cuda")
    at = torch.stack([torch.searchsorted(r.contiguous(), cuts) for r in ranks]).cpu().numpy()
    dense = torch.empty((n, step), dtype=torch.float64, device="cuda")
    for b in range(len(cuts) - 1):
        dense.zero_()
        for v in range(n):
            i, j = int(at[v, b]), int(at[v, b + 1])
            if j > i:
                dense[v, ranks[v][i:j] - b * step] = vectors[v][1][i:j].double()
        if rows:
            out += dense[:rows] @ dense[rows:].T
        else:
            out += dense @ dense.T
    return out


def exact(case, seed):
    c = dict(case)
    alphabet, k = c["alphabet"], c["k"]
    counts = _case_counts(c)
    if sum(_entries(_MEAN_PROTEIN * m, alphabet, k) for m in counts) > 1.2e9:
        return None
    seq, off = _generate(counts, seed, alphabet)
    each = [seq[int(off[i]):int(off[i + 1])] for i in range(len(counts))]
    if c["kind"] in ("build", "batch"):
        parts = []
        for s in each:
            a = _alpha(s, alphabet, k)[1]
            a = a / torch.sqrt((a * a).sum())
            size = -(-a.numel() // 4) * 4 if c["kind"] == "batch" else _max_entries(s.numel(), alphabet, k)
            parts.append(torch.nn.functional.pad(a, (0, size - a.numel())))
        values = torch.cat(parts)
        if c["kind"] == "batch":
            size = int(np.sum(8 * np.diff(off) + 64)) + 1024
            values = torch.nn.functional.pad(values, (0, size - values.numel()))
        if c["kind"] == "build":
            return {"size": None, "keys": None, "values": values}
        return {"keys": None, "values": values, "offsets": None, "nnz": None}
    vectors = [_vector32(s, alphabet, k) for s in each]
    if c["kind"] == "query":
        return {"c": _products(vectors[c["db"]:] + vectors[:c["db"]], c["n"])}
    if c["kind"] == "compare":
        return {"c": _products(vectors, 1).reshape(-1)}
    return {"c": _products(vectors, 0)}
