"""Segments run in parts: the same FP32 runs, so the same sums, as the whole segments."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from rocket_gb300 import engine, synth
from rocket_gb300.engine import BatchBuilder, EngineConfig, PairEngine

pytestmark = pytest.mark.gpu


def _arena(alphabet, k, n, scale):
    p = synth.workload("uneven1024", n=n, scale=scale)
    data = p.data
    if alphabet == "DNA":
        data = np.frombuffer(b"ACGT", np.uint8)[data & 3].copy()
        data[p.data == 10] = 10
    return BatchBuilder(alphabet, k).build(torch.from_numpy(data).cuda(), p.offsets)


# The parts add the same FP32 run sums to float-float accumulators, in several partial
# blocks instead of one.  A lane folds at most some hundred runs at these sizes, of at
# most C = 1 in all: the low words reach 1e2 * 2^-25 and their additions round by at most
# 1e2 * (1e2 * 2^-25) * 2^-24 = 2e-11 in all, in practice far less (the sums of runs
# cut elsewhere differ by 1e-9 and more).
TOL = 2e-11


CASES = [
    ("protein", 6, 40, 0.02, dict(), 1),                    # every part a few windows
    ("protein", 6, 40, 0.02, dict(tile_cols=256, fold=8), 2),
    ("protein", 7, 33, 0.02, dict(segments=2, wshift=10), 3),
    ("protein", 5, 17, 0.05, dict(segments=1, wshift=9), 5),
    ("protein", 6, 3, 0.2, dict(segments=3, fold=16), 1),   # many lanes per column
    ("protein", 4, 21, 0.3, dict(wshift=7), 2),             # windows narrower than a table
    ("DNA", 8, 30, 0.05, dict(), 1),                        # full tables
    ("DNA", 10, 150, 0.02, dict(segments=5, compress=False), 7),
    ("DNA", 6, 9, 0.05, dict(), 1),                         # two windows in all
]


@pytest.mark.parametrize("alphabet,k,n,scale,cfg,part", CASES)
def test_parts_form_the_segments_sums(monkeypatch, alphabet, k, n, scale, cfg, part):
    arena = _arena(alphabet, k, n, scale)
    # parts as short as `part` windows, also where their tails outweigh them
    monkeypatch.setattr(engine, "split_segments",
                        lambda windows, *a: np.maximum(-(-windows // part), 1).astype(np.int64))
    monkeypatch.setattr(engine, "PART_WINDOWS", part)
    eng = PairEngine(arena, EngineConfig(**cfg))
    eng.ensure_index()
    plan = eng.plan_triangle()
    if plan.host_parts is None:  # fixed segments over columns too sparse for parts
        assert cfg.get("segments")
        pytest.skip("not cut")
    outs = [torch.zeros((n, n), dtype=torch.float64, device="cuda") for _ in range(3)]
    cycles = torch.zeros(plan.nitems, dtype=torch.int64, device="cuda")
    eng.run(plan, outs[0], item_cycles=cycles)  # whole items
    assert int(cycles.min()) > 0
    eng.run(plan, outs[1])
    eng.run(plan, outs[2])
    assert torch.equal(outs[1], outs[2])
    d = float((outs[1] - outs[0]).abs().max())
    assert d <= TOL, d


@pytest.mark.parametrize("tj,words", [(256, 4), (128, 8), (64, 4), (32, 8)])
@pytest.mark.parametrize("S", [1, 3, 5, 152])
def test_reduction_sums_every_partial(tj, words, S):
    """Partial blocks of small integers: every order of summation is exact."""
    from rocket_gb300 import _native
    L = _native.load()
    g = torch.Generator().manual_seed(tj + S)
    ncol = tj - 3
    part = torch.randint(-50, 50, (2, S, 16, tj, 2), generator=g).float().cuda()
    tiles = np.zeros((2, words), np.int32)
    for t in range(2):
        tiles[t, :4] = (16 * t, 16 - t, 5, ncol)
        if words == 8:
            tiles[t, 4:6] = (t * S, S)
    rows = torch.arange(32, dtype=torch.int32, device="cuda")
    cols = torch.arange(tj + 8, dtype=torch.int32, device="cuda")
    d_tiles = torch.from_numpy(tiles).cuda()
    out = torch.full((32, tj + 8), -1.0, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    if words == 8:
        rc = L.phyloPairsReduceParts(st, part.data_ptr(), d_tiles.data_ptr(), 2, 16, tj,
                                     rows.data_ptr(), cols.data_ptr(), out.data_ptr(), tj + 8,
                                     0, 0)
    else:
        rc = L.phyloPairsReduce(st, part.data_ptr(), d_tiles.data_ptr(), 2, S, 16, tj,
                                rows.data_ptr(), cols.data_ptr(), out.data_ptr(), tj + 8, 0, 0)
    assert rc == 0
    want = torch.full_like(out, -1.0)
    sums = part.double().sum(dim=(1, 4))
    for t in range(2):
        want[16 * t:32 - (t if t else 16), 5:5 + ncol] = sums[t, :16 - t, :ncol]
    assert torch.equal(out, want)


# Row vectors by fours, eights and sixteens: the same sums, bit for bit, whichever kernel
# takes a part (each row's products enter its own accumulators in the same order).
@pytest.mark.parametrize("rows", [1, 4, 5, 8, 9, 16, 17, 20, 24, 25])
@pytest.mark.parametrize("cols,tile_cols", [(3, 128), (37, 128), (50, 256)])
def test_few_rows(rows, cols, tile_cols):
    db = _arena("protein", 5, cols, 0.2)
    queries = _arena("protein", 5, rows, 0.05)
    cfg = EngineConfig(segments=2, compress=False, tile_cols=tile_cols)
    PairEngine(db, cfg).ensure_index()
    eng = PairEngine(queries, cfg)
    eng.ensure_index()
    plan = eng.plan_rect(np.arange(rows), np.arange(cols), ldc=cols, col_arena=db)
    assert plan.host_parts is not None
    last = rows % 16 or 16
    small = [4] if last <= 4 else [8] if last <= 8 else [16]
    assert [g[2] for g in plan.part_groups] == ([16] if rows > 16 and small != [16] else []) + small
    assert sum(g[1] for g in plan.part_groups) == len(plan.host_parts)
    outs = []
    for groups in (plan.part_groups, [(0, len(plan.host_parts), 16)]):
        plan.part_groups = groups
        out = torch.full((rows, cols), np.nan, dtype=torch.float64, device="cuda")
        eng.run(plan, out, diagonal=False, col_arena=db)
        outs.append(out.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
    assert np.isfinite(outs[0]).all()
