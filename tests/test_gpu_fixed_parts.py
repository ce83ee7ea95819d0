"""Fixed segments that are certainly cut: the same FP32 runs, so the same sums, as the whole
segments."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from rocket_gb300 import engine
from rocket_gb300.engine import EngineConfig, PairEngine

from test_gpu_parts import TOL, _arena

pytestmark = pytest.mark.gpu


# Parts as short as `part` windows whatever their tails: K = 7 (sparse columns, runs over
# many windows), K = 5, many lanes per column, and DNA.
@pytest.mark.parametrize("alphabet,k,n,scale,cfg,part", [
    ("protein", 7, 33, 0.02, dict(segments=2, wshift=10), 30),
    ("protein", 7, 5, 0.05, dict(segments=4, compress=False), 900),
    ("protein", 5, 17, 0.05, dict(segments=1, wshift=9), 5),
    ("protein", 6, 3, 0.2, dict(segments=3, fold=16), 1),
    ("protein", 6, 40, 0.02, dict(segments=2, tile_cols=256, fold=8), 2),
    ("DNA", 10, 150, 0.02, dict(segments=5, compress=False), 7)])
def test_cut_fixed_segments_form_the_whole_ones_sums(monkeypatch, alphabet, k, n, scale, cfg, part):
    arena = _arena(alphabet, k, n, scale)
    monkeypatch.setattr(engine, "fixed_parts", lambda cfg, R, grid, S, ncol, *a: np.full(
        len(ncol), -(-R // (S * part)), np.int64))
    eng = PairEngine(arena, EngineConfig(**cfg))
    eng.ensure_index()
    plan = eng.plan_triangle()
    assert plan.host_parts is not None and plan.nparts > plan.nitems
    outs = [torch.zeros((n, n), dtype=torch.float64, device="cuda") for _ in range(2)]
    eng.run(plan, outs[0])
    plan.host_parts = None  # whole items
    eng.run(plan, outs[1])
    d = float((outs[0] - outs[1]).abs().max())
    assert d <= TOL, d


@pytest.mark.parametrize("rows", [1, 4, 5, 8, 24])
def test_whole_segments_of_few_rows(rows):
    """Columns that fill the GPU uncut: whole segments through the kernels of few rows have the
    bits of whole items."""
    db = _arena("protein", 5, 300, 0.01)
    queries = _arena("protein", 5, rows, 0.05)
    cfg = EngineConfig(segments=64, compress=False)
    PairEngine(db, cfg).ensure_index()
    eng = PairEngine(queries, cfg)
    eng.ensure_index()
    plan = eng.plan_rect(np.arange(rows), np.arange(300), ldc=300, col_arena=db)
    assert plan.host_parts is not None and plan.nparts == plan.nitems
    outs = []
    for parts in (plan.host_parts, None):
        plan.host_parts = parts
        out = torch.full((rows, 300), np.nan, dtype=torch.float64, device="cuda")
        eng.run(plan, out, diagonal=False, col_arena=db)
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and bool(torch.isfinite(outs[0]).all())
