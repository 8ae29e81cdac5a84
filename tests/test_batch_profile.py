"""A batch's profile across a change of its program: a tuft of one synapse a
cell leaves its layer's tail when the caller makes it read the layer's own
axons, and goes back when the whole state is written with the old sources."""
import numpy as np
import pytest

from bismit_b200 import _ffi as F, cortex, map as M
from helpers import settings_for
from test_tuft_seg import _small

pytestmark = pytest.mark.gpu


def _batch():
    src = M.TuftSourceLayer.define("iv").syn_reach(2).prevalence(1)
    tiny = M.TuftScheme.basal().proximal().dens_per_tft(1).syns_per_den(1)
    big = M.TuftScheme.basal().distal().dens_per_tft(4).syns_per_den(16).max_active_dens_l2(1)
    l2, a2 = _small(32, 1, M.CellScheme.pyramidal().tft(tiny.src_lyr(src)).tft(big.src_lyr(src)))
    ctx = cortex._Ctx(0)
    a = cortex.CorticalArea(ctx, M.area_desc("v1", l2, a2, settings_for()), 7)
    b = cortex.Batch(ctx, [a])
    b.set_profiling(True)
    return ctx, a, b


def _rows(b):
    """{(step, layer, index): launches}; a step's device time is positive."""
    rows = b.profile()
    assert all(r[5] > 0 for r in rows)
    out = {r[:3]: r[4] for r in rows}
    assert len(out) == len(rows)
    return out


@pytest.mark.parametrize("read_first", [False, True])
@pytest.mark.parametrize("back", [False, True])
def test_profile_follows_the_program(back, read_first):
    ctx, a, b = _batch()
    n = int(a.plan.layers[1].n_syns)
    keep = a.read_slab()
    own = np.full(n, int(a.plan.layers[1].base_axn_slc), np.uint8)
    steps = [("fused_tuft_batch", 0, 0), ("inhib_mtp", 0, 0), ("fused_tuft_batch", 1, 1)]
    b.cycle(3)
    if read_first:
        before = _rows(b)
        assert [before[s] for s in steps] == [3, 3, 3] and ("tuft", 1, 0) not in before
    a.write("syn_src_slc_ids", own, layer=1)
    b.cycle(2)
    if back:
        if read_first:
            _rows(b)
        a.write_slab(keep)
        b.cycle(4)
    rows = _rows(b)
    total = 9 if back else 5
    assert {s: rows[s] for s in steps} == {s: total for s in steps}
    assert [v for s, v in rows.items() if s[0] == "pyr_tail"] == [total]
    assert rows[("tuft", 1, 0)] == 2
    b.reset_profile()
    assert b.profile() == []
    b.cycle(1)
    assert (("tuft", 1, 0) in _rows(b)) == (not back)
    b.close()
    a.close()
    ctx.close()
