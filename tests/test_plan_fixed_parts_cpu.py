"""Parts of fixed segments against databases of many vectors: host logic on the CPU."""
import numpy as np
import pytest

from rocket_gb300 import engine

from test_plan_parts_cpu import _check, _engine

GRID, S = 152, 16


def _plan(nnz, R, rows, cols):
    eng = _engine(nnz, R, grid=GRID, segments=S)
    return eng.plan_rect(np.arange(rows), np.arange(cols), ldc=cols, col_arena=eng.arena)


def _uneven(cols, R, seed):
    """Entries of uneven vectors: 0.1 to 8 per window at K = 7, 2 to 150 at K = 6."""
    rng = np.random.default_rng(seed)
    return np.exp(rng.uniform(np.log(1e5), np.log(7e6), cols)).astype(np.int64)


@pytest.mark.parametrize("R", [41878, 879440])
@pytest.mark.parametrize("cols", [300, 512, 2048, 20000])
@pytest.mark.parametrize("uneven", [False, True])
def test_large_databases_take_no_more_parts_than_fill_the_gpu(R, cols, uneven):
    nnz = _uneven(cols, R, cols) if uneven else np.full(cols, 4 * 10 ** 6)
    tiles = -(-cols // 128)
    cuts = []
    for rows in (3, 40, 64):
        plan = _plan(nnz, R, rows, cols)
        if plan.host_parts is None:
            assert cols == 20000 and rows == 64
            continue
        _check(plan)
        blocks = -(-rows // 16)
        # the share of every tile is rounded up to whole parts
        most = engine.PARTS_PER_CTA * GRID + S * tiles
        assert plan.nparts <= blocks * most
        first = plan.host_parts[plan.host_parts[:, 0] == 0]
        assert len(first) >= GRID  # and the GPU is full with a single row tile
        cuts.append({tuple(int(x) for x in p[[2, 3, 4, 5, 8, 9]]) for p in first})
    assert all(c == cuts[0] for c in cuts)


def test_long_tiles_are_cut_before_short_ones():
    """Of a database as uneven as proteomes are, the columns of most entries take more
    parts than those of few."""
    nnz = np.sort(_uneven(2048, 41878, 1))[::-1]
    plan = _plan(nnz, 41878, 1, 2048)
    n = plan.host_part_tiles[:, 5] // S
    assert n[0] > n[-1] >= 1 and (np.diff(n) <= 0).all()


def test_whole_segments_of_few_rows_keep_their_kernels():
    """Columns enough to fill the GPU uncut: rows of a tile of at most eight still go to the
    kernels for so many; full tiles run as whole items."""
    nnz = np.full(20000, 2 * 10 ** 5)
    plan = _plan(nnz, 41878, 5, 20000)
    _check(plan)
    assert plan.nparts == plan.nitems and [g[2] for g in plan.part_groups] == [8]
    assert (plan.host_parts[:, 4:6] == plan.host_parts[:, 8:10]).all()
    assert _plan(nnz, 41878, 48, 20000).host_parts is None


@pytest.mark.parametrize("n,R", [(40, 3000), (200, 41878), (200, 8000), (24, 224), (500, 41878)])
@pytest.mark.parametrize("segments", [2, 16, 64])
def test_triangles_fill_the_gpu_together(n, R, segments):
    """All tiles of a triangle share the GPU: its fixed segments take no more parts than fill
    it, and the last rows' tiles a launch of their own only where they fill half of it."""
    eng = _engine(np.full(n, 200 * R), R, grid=GRID, segments=segments)
    plan = eng.plan_triangle()
    if plan.host_parts is None:
        return
    _check(plan)
    assert plan.nparts <= engine.PARTS_PER_CTA * GRID + plan.S * plan.ntiles
    assert sum(g[1] for g in plan.part_groups) == plan.nparts
    for first, count, rows in plan.part_groups:
        assert (plan.host_parts[first:first + count, 1] <= rows).all()
        assert rows == 16 or 2 * count >= GRID
