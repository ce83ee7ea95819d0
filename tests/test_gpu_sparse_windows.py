"""Windows in which most rows have no entry, or a few that share a 16-byte group with the
windows beside: the scatter that most threads skip.  Small whole numbers, so exact sums."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from rocket_gb300 import synth
from rocket_gb300.engine import BatchBuilder, EngineConfig, PairEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,wshift,rows,cols,segments", [
    (33, 4, 16, 128, 40), (20, 6, 16, 256, 9), (33, 4, 16, 64, 300), (17, 5, 16, 32, 200),
    (6, 4, 16, 128, 3), (2, 8, 16, 128, 2)])
def test_sparse_windows(n, wshift, rows, cols, segments):
    p = synth.workload("uneven1024", n=n, scale=0.01)
    arena = BatchBuilder("protein", 5).build(torch.from_numpy(p.data).cuda(), p.offsets)
    g = torch.Generator(device="cuda").manual_seed(n)
    arena.values[:arena.used] = torch.randint(-2, 3, (arena.used,), generator=g,
                                              device="cuda").float()
    eng = PairEngine(arena, EngineConfig(wshift=wshift, compress=False, tile_rows=rows,
                                         tile_cols=cols, segments=segments))
    eng.ensure_index()
    plan = eng.plan_triangle()
    dense = torch.zeros((n, 21 ** 5), dtype=torch.float64, device="cuda")
    for v in range(n):
        k, x = arena.vector(v)
        dense[v, k.long()] = x.double()
    want = dense @ dense.T
    assert float(want.abs().max()) < 2 ** 23
    out = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    eng.run(plan, out)
    assert torch.equal(out, want)
    if plan.host_parts is not None:
        plan.host_parts = None  # whole items too
        eng.run(plan, out.zero_())
        assert torch.equal(out, want)
