"""Window plans whose segments run in parts: host logic on the CPU."""
from types import SimpleNamespace

import numpy as np
import pytest

from rocket_gb300 import engine
from rocket_gb300.engine import EngineConfig, PairEngine, key_limit


def _engine(nnz, R, grid=152, **cfg):
    eng = PairEngine.__new__(PairEngine)
    eng.cfg = EngineConfig(**cfg)
    eng.arena = SimpleNamespace(n=len(nnz), nnz=np.asarray(nnz, np.int64), R=R,
                                alphabet="protein", k=6, rank_limit=key_limit("protein", 6),
                                index_on_ranks=False)
    eng.grid = grid
    eng.device = "cpu"
    return eng


def _check(plan):
    """The parts of every segment cover its windows in order; a tile's partial blocks are
    numbered from its part0, in segment and window order."""
    by_tile = {}
    for p in plan.host_parts:
        by_tile.setdefault(int(p[7]), []).append(p)
    assert sorted(int(p[6]) for p in plan.host_parts) == list(range(plan.nparts))
    for t, parts in by_tile.items():
        parts.sort(key=lambda p: int(p[6]))
        tile = plan.host_part_tiles[t]
        assert [int(p[6]) for p in parts] == list(range(tile[4], tile[4] + tile[5]))
        at = 0
        for p in parts:
            assert tuple(p[:4]) == tuple(tile[:4]) == tuple(plan.host_tiles[t][:4])
            assert p[4] == at and p[5] > p[4] and p[8] <= p[4] and p[5] <= p[9]
            at = p[5]
        whole = sorted({(int(p[8]), int(p[9])) for p in parts})
        mine = sorted((int(i[4]), int(i[5])) for i in plan.host_items[plan.item_tile == t])
        assert whole == mine


@pytest.mark.parametrize("n,R,cfg", [
    (24, 224, dict()), (30, 32, dict()), (64, 512, dict(tile_cols=256)),
    (40, 400, dict()), (90, 700, dict(segments=3)), (40, 3000, dict(segments=16))])
@pytest.mark.parametrize("spread", [1.2, 12.0])
def test_parts_cover_every_segment(n, R, cfg, spread):
    rng = np.random.default_rng(n)
    nnz = np.minimum(300 * R * spread ** rng.uniform(-0.5, 0.5, n), 2 ** 24 - 1)
    eng = _engine(nnz.astype(np.int64), R, **cfg)
    plan = eng.plan_triangle()
    _check(plan)
    assert plan.nparts > plan.nitems


def test_full_plans_and_sparse_columns_are_not_cut():
    # enough items for the grid already
    assert _engine(np.full(512, 10 ** 6), 20000, tile_cols=256).plan_triangle().host_parts is None
    # columns of a few entries per window: a lane's FP32 run reaches over many windows
    eng = _engine(np.full(24, 300), 224)
    assert eng.plan_triangle().host_parts is None
    # the other kernels have no parts
    for cfg in (dict(algorithm="postings"), dict(tile_rows=32, tile_cols=64, wshift=10),
                dict(tile_cols=64, wshift=10)):
        assert _engine(np.full(24, 10 ** 5), 224, **cfg).plan_triangle().host_parts is None


def test_parts_of_fixed_segments_do_not_depend_on_the_rows():
    """A query's sums are the same whether it runs alone or in a batch: the windows its
    parts start at depend on the columns only."""
    nnz = np.full(200, 10 ** 6)
    cuts = []
    for rows in (np.arange(3), np.arange(40)):
        eng = _engine(nnz, 41878, segments=16)
        plan = eng.plan_rect(rows, np.arange(160), ldc=160, col_arena=eng.arena)
        _check(plan)
        first = plan.host_parts[(plan.host_parts[:, 0] == 0)]
        cuts.append({tuple(int(x) for x in p[[2, 3, 4, 5, 8, 9]]) for p in first})
    assert cuts[0] == cuts[1]
    assert max(b - a for _, _, a, b, _, _ in cuts[0]) <= engine.PART_WINDOWS


@pytest.mark.parametrize("cols,nnz", [(40, 2 * 10 ** 5), (20, 10 ** 5), (5, 10 ** 6), (150, 10 ** 5)])
def test_small_databases_use_the_idle_ctas(cols, nnz):
    """Few columns of few entries: more parts than their tails alone would ask for, at most
    one per CTA, and the same whatever the rows."""
    grid, cuts = 152, []
    for rows in (np.arange(3), np.arange(40)):
        eng = _engine(np.full(200, nnz), 41878, grid=grid, segments=16)
        plan = eng.plan_rect(rows, np.arange(cols), ldc=cols, col_arena=eng.arena)
        _check(plan)
        first = plan.host_parts[(plan.host_parts[:, 0] == 0)]
        # parts whose tails are a quarter of them at most, as many as there are
        free = 0
        for c0, ncol in {(int(p[2]), int(p[3])) for p in first}:
            tail = eng.cfg.fold * -(-512 // ncol) / (nnz / 41878)
            windows = 41878 / 16
            free += 16 * max(1, int(min(-(-windows // engine.PART_WINDOWS), windows / max(4 * tail, 1))))
        assert free <= len(first) <= max(grid, free)
        cuts.append({tuple(int(x) for x in p[[2, 3, 4, 5, 8, 9]]) for p in first})
    assert cuts[0] == cuts[1]
