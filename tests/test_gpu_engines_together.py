"""Engines of one tile shape and different window widths in one process: the second one's
preparation leaves the first one's launches as they were."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from rocket_gb300 import synth
from rocket_gb300.engine import BatchBuilder, EngineConfig, PairEngine

pytestmark = pytest.mark.gpu


def _matrix(eng, parts):
    eng.ensure_index()
    plan = eng.plan_triangle()
    if not parts:
        plan.host_parts = None
    out = torch.zeros((eng.arena.n,) * 2, dtype=torch.float64, device="cuda")
    eng.run(plan, out)
    return out.cpu().numpy(), plan


@pytest.mark.parametrize("rows,cols,wide,narrow", [
    (16, 128, 11, 9), (16, 256, 11, 4), (16, 64, 11, 8), (16, 32, 11, 10), (32, 64, 9, 7)])
def test_narrow_windows_leave_wide_ones_running(rows, cols, wide, narrow):
    p = synth.workload("uneven1024", n=20, scale=0.02)
    seq = torch.from_numpy(p.data).cuda()
    cfg = dict(tile_rows=rows, tile_cols=cols)
    first = PairEngine(BatchBuilder("protein", 5).build(seq, p.offsets),
                       EngineConfig(wshift=wide, **cfg))
    want, _ = _matrix(first, True)
    second = PairEngine(BatchBuilder("protein", 5).build(seq, p.offsets),
                        EngineConfig(wshift=narrow, **cfg))
    _matrix(second, True)
    again, plan = _matrix(first, True)
    assert np.array_equal(again, want)
    if plan.host_parts is not None:
        _matrix(first, False)  # whole items of the same shape
