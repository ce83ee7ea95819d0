"""Parts that start anywhere in a long segment: every entry of a column is used by one part.

The values are small whole numbers, so every product and sum is exact in FP32 and a matrix
is right or wrong: an entry that two parts use, or none, shows."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from rocket_gb300 import engine, synth
from rocket_gb300.engine import BatchBuilder, EngineConfig, PairEngine

pytestmark = pytest.mark.gpu


# One segment of 7,977 windows in parts of `part`: the distances of their starts from it leave
# every remainder modulo the boundaries that a column's lanes load together (16 for each of
# its 512 / columns lanes), or many of them.
@pytest.mark.parametrize("cols,part,cfg", [
    (128, 61, dict()), (40, 61, dict(fold=8)), (3, 127, dict()), (1, 301, dict(fold=4)),
    (200, 97, dict(tile_cols=256)), (256, 33, dict(tile_cols=256, fold=12))])
def test_every_entry_is_in_one_part(monkeypatch, cols, part, cfg):
    p = synth.workload("uneven1024", n=cols, scale=0.02)
    arena = BatchBuilder("protein", 5).build(torch.from_numpy(p.data).cuda(), p.offsets)
    g = torch.Generator(device="cuda").manual_seed(cols)
    arena.values[:arena.used] = torch.randint(-2, 3, (arena.used,), generator=g,
                                              device="cuda").float()
    monkeypatch.setattr(engine, "split_segments",
                        lambda windows, *a: -(-windows // part).astype(np.int64))
    eng = PairEngine(arena, EngineConfig(wshift=9, compress=False, min_windows_per_item=10 ** 6,
                                         **cfg))
    eng.ensure_index()
    plan = eng.plan_triangle()
    assert plan.S == 1 and plan.nparts >= arena.R // part > 20
    out = torch.zeros((cols, cols), dtype=torch.float64, device="cuda")
    eng.run(plan, out)
    dense = torch.zeros((cols, 21 ** 5), dtype=torch.float64, device="cuda")
    for v in range(cols):
        k, x = arena.vector(v)
        dense[v, k.long()] = x.double()
    assert torch.equal(out, dense @ dense.T)
    assert float(out.abs().max()) < 2 ** 23
