"""How the work is cut: chunks of the builder's candidate passes (many or few bitmap words
per warp), segments of the survivors with and without drops, and the runs of tiles of the
pair compare."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O
from rocket_gb300 import _native
from rocket_gb300.engine import BatchBuilder

from gpu_helpers import build_gpu, ulp_diff
from test_gpu_compare import compare_gpu

pytestmark = pytest.mark.gpu

AMINO = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", np.uint8)
BASES = np.frombuffer(b"ACGT", np.uint8)


def _residues(letters, n, seed):
    """n residues with uneven frequencies, in proteins of uneven lengths, and runs of the
    first and the last letter (the first and last words of the bitmaps)."""
    rng = np.random.default_rng(seed)
    p = rng.random(len(letters)) ** 2 + 0.01
    s = letters[rng.choice(len(letters), n, p=p / p.sum())].copy()
    if n > 40:
        s[:12], s[20:32] = letters[0], letters[-1]
    s[rng.choice(n, n // 300, replace=False)] = ord("\n")
    return s.tobytes()


def _check(seq, k, alphabet, keys, vals):
    r = O.cv_native(seq, k, alphabet)
    assert np.array_equal(keys, r["keys"])
    assert ulp_diff(vals, r["values"]) <= 1  # the builder's tests' bound


# A single proteome at K = 6 keeps 32 lanes with words below 2^18 residues and takes 8 above.
@pytest.mark.parametrize("n", [1, 7, 5000, (1 << 18) - 1, 1 << 18, (1 << 18) + 1])
def test_short_and_long_single_proteomes(n):
    seq = _residues(AMINO, n, n)
    cnt, keys, vals = build_gpu(seq, 6)
    _check(seq, 6, "protein", keys[:cnt], vals[:cnt])
    assert np.all(keys[cnt:] == 0xFFFFFFFF) and np.all(vals[cnt:] == 0)


# Batches on both sides of the lines between 2, 8 and 32 lanes with words: 32 lanes from
# 1,500 chunks on, which at K = 6 (499 each) takes 4 proteomes and 8 lanes below; at K = 5
# 8 lanes from 16 proteomes (95 chunks each), over DNA at K = 10 from 12 (128 each), and 2
# lanes below; at K = 3 and 4 a few chunks in all.  K = 7: eight words per lane.
@pytest.mark.parametrize("alphabet,k,batch", [
    ("protein", 3, 1), ("protein", 4, 5), ("protein", 5, 1), ("protein", 5, 4),
    ("protein", 5, 15), ("protein", 5, 16), ("protein", 6, 1), ("protein", 6, 3),
    ("protein", 6, 4), ("protein", 7, 1), ("protein", 7, 3), ("DNA", 3, 2), ("DNA", 8, 3), ("DNA", 10, 2), ("DNA", 10, 3),
    ("DNA", 10, 12)])
def test_batches_over_every_chunk_size(alphabet, k, batch):
    letters = AMINO if alphabet == "protein" else BASES
    seqs = [_residues(letters, 1500 + 997 * i, 31 * k + i) for i in range(batch)]
    off = np.concatenate([[0], np.cumsum([len(s) for s in seqs])]).astype(np.uint64)
    d = torch.from_numpy(np.frombuffer(b"".join(seqs), np.uint8).copy()).cuda()
    arena = BatchBuilder(alphabet, k, max_batch=batch).build(d, off)
    torch.cuda.synchronize()
    for i, s in enumerate(seqs):
        _check(s, k, alphabet, *arena.host_vector(i))


# Candidates whose alpha is 0 leave the vector; segments of 256 candidates that lose none
# are moved as they are.  Repeats of one word give alpha 0 nowhere or everywhere; mixed
# with random residues, segments of both kinds stand side by side.
@pytest.mark.parametrize("repeat", [0, 1, 40, 4000])
@pytest.mark.parametrize("k", [3, 6])
def test_segments_with_and_without_drops(k, repeat):
    seq = _residues(AMINO, 60000, k) + b"\n" + b"ACDEFGHIKLMNPQRSTVWYX" * repeat + b"\n"
    cnt, keys, vals = build_gpu(seq, k)
    _check(seq, k, "protein", keys[:cnt], vals[:cnt])


def _lists(kind, n, rng):
    if kind == "below":      # every left key below every right one: whole tiles of one side
        return np.arange(n), np.arange(n) + n
    if kind == "above":
        return np.arange(n) + n, np.arange(n)
    if kind == "equal":
        return np.arange(n) * 7, np.arange(n) * 7
    if kind == "blocks":     # long stretches of one side, then of the other, some shared keys
        b = np.arange(2 * n) // 6001 % 2
        keys = np.arange(2 * n) * 3
        share = keys % 11 == 0
        return keys[(b == 0) | share], keys[(b == 1) | share]
    if kind == "few":        # one side almost empty
        a = np.arange(2 * n)
        return a, np.sort(rng.choice(a, 5, replace=False))
    a = np.flatnonzero(rng.random(4 * n) < 0.3)  # random, half of them shared or so
    return a, np.flatnonzero(rng.random(4 * n) < 0.2)


# Several tiles for each CTA (more than 456 * 4352 merged elements), where a tile's end is
# searched for from its start.  Bound: products are exact pairs of floats and a thread adds
# at most 17 per tile to a float-float sum, whose low word (at most 2^-24 of the sum) rounds
# by 2^-48 of the sum per addition: 17 * 8 tiles * 2^-48 = 5e-13 of C (all terms positive).
@pytest.mark.parametrize("kind", ["below", "above", "equal", "blocks", "few", "random"])
@pytest.mark.parametrize("n", [900, 1200000, 2500001])
def test_runs_of_tiles(kind, n):
    rng = np.random.default_rng(n)
    lk, rk = _lists(kind, n, rng)
    lv = rng.random(len(lk), dtype=np.float32)
    rv = rng.random(len(rk), dtype=np.float32)
    lk, rk = lk.astype(np.int32), rk.astype(np.int32)
    exact = O.compare_fp64(lk.view(np.uint32), lv, rk.view(np.uint32), rv)
    got = compare_gpu(lk, lv, rk, rv, slot_layout=True)
    assert abs(got - exact) <= 5e-13 * abs(exact)


# The chained launches in a graph: replays give the call's bits, also after the inputs
# have changed in place.
@pytest.mark.parametrize("n", [0, 40, 300000])
def test_compare_in_a_graph(n):
    L = _native.load()
    rng = np.random.default_rng(n)
    dev = {}
    for side in "ab":
        keys = np.sort(rng.choice(3 * n + 1, n, replace=False)).astype(np.int32)
        dev[side] = [torch.from_numpy(keys).cuda(),
                     torch.from_numpy(rng.random(n, dtype=np.float32)).cuda()]
    scratch = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    out = torch.full((1,), -1.0, dtype=torch.float64, device="cuda")

    def call():
        (ka, va), (kb, vb) = dev["a"], dev["b"]
        _native.check(L.phyloComparePairAsync(
            torch.cuda.current_stream().cuda_stream, scratch.data_ptr(), scratch.numel(),
            ka.data_ptr(), va.data_ptr(), n, kb.data_ptr(), vb.data_ptr(), n, out.data_ptr()))

    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    for _ in range(3):
        if n:
            dev["a"][1].mul_(0.5)
        call()
        want = out.item()
        out.fill_(-1.0)
        g.replay()
        torch.cuda.synchronize()
        assert out.item() == want
