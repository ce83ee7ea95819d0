"""What a serving batch reserves for its partial blocks is what its plan has."""
from types import SimpleNamespace

import numpy as np
import pytest

from rocket_gb300 import serve
from rocket_gb300.engine import EngineConfig, fixed_blocks
from rocket_gb300.serve import Request, ServingEngine

from test_plan_parts_cpu import _engine

GRID = 152


def _nnz(n):
    return np.exp(np.random.default_rng(n).uniform(np.log(1e5), np.log(7e6), n)).astype(np.int64)


@pytest.mark.parametrize("R", [700, 41878, 879440])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 20), (64, 160), (17, 300), (64, 2048), (5, 20000)])
@pytest.mark.parametrize("cfg", [dict(), dict(tile_cols=256), dict(tile_cols=64, wshift=10),
                                 dict(tile_rows=32, tile_cols=64, wshift=10), dict(segments=3)])
def test_blocks_of_a_plan(R, rows, cols, cfg):
    eng = _engine(_nnz(max(rows, cols)), R, grid=GRID, **dict(dict(segments=16), **cfg))
    plan = eng.plan_rect(np.arange(rows), np.arange(cols), ldc=cols, col_arena=eng.arena)
    assert fixed_blocks(eng.cfg, R, GRID, rows, eng.arena.nnz[:cols]) == plan.nparts


def test_estimate_reserves_the_plans_blocks(monkeypatch):
    srv = ServingEngine("protein", 7, slots=1, cfg=EngineConfig(segments=16))
    srv.grid = GRID
    srv.db = SimpleNamespace(R=879440, arena=SimpleNamespace(nnz=_nnz(2060)))
    reqs = [Request(0, SimpleNamespace(lengths=lambda: np.full(64, 10 ** 6)))]
    with_blocks = srv._estimate(reqs, 2048)
    monkeypatch.setattr(serve, "fixed_blocks", lambda *a: 0)
    blocks = with_blocks - srv._estimate(reqs, 2048)
    # 64 x 2,048 vectors at K = 7, 1,024 uncut items of 16 x 128 pairs: 17 MB
    assert 1024 * 16 * 128 * 8 <= blocks <= 4 * 1024 * 16 * 128 * 8
    assert srv._estimate(reqs, 0) < with_blocks  # an empty database


def test_estimate_asks_an_engine_for_the_grid(monkeypatch):
    """A database that was not made by load(): the CTAs are those of an engine over it."""
    srv = ServingEngine("protein", 7, slots=1, cfg=EngineConfig(segments=16))
    srv.db = SimpleNamespace(R=879440, arena=SimpleNamespace(nnz=_nnz(300)))
    made = []
    monkeypatch.setattr(serve, "PairEngine",
                        lambda arena, cfg: made.append(arena) or SimpleNamespace(grid=GRID))
    reqs = [Request(0, SimpleNamespace(lengths=lambda: np.full(3, 10 ** 6)))]
    first = srv._estimate(reqs, 300)
    assert srv.grid == GRID and first == srv._estimate(reqs, 300) and made == [srv.db.arena]
