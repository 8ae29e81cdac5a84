"""The input filter against the oracle where its blocks of 32 x 4 cells end
inside the grid, are wider than it, or meet its sides."""
import numpy as np
import pytest

import oracle
from bismit_b200 import configs, cortex, map as M
from helpers import diff_report, frames_for, initial_slab, settings_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,n_filters,depth", [(8, 1, 1), (24, 2, 1), (40, 1, 2), (136, 2, 1)])
def test_retina_sides(side, n_filters, depth):
    ctx = cortex._Ctx(0)
    a = cortex.CorticalArea(ctx, M.area_desc("v1", *configs.retina_area(side, n_filters, depth), settings_for()), 3)
    slab = initial_slab(a.plan, 3, scramble_seed=9, clean_flags=True)
    a.write_slab(slab)
    fr = frames_for(a.plan, 3, 6, active=0.4)
    for k in range(3):
        a.write_input(fr[k])
        a.cycle(1)
        oracle.intake(a.plan, slab, 0, 0, fr[k])
        oracle.run(a.plan, slab, None, 1, start_cycle=k)
        dev = a.read_slab()
        assert np.array_equal(dev, slab), "cycle %d\n%s" % (k, diff_report(a.plan, dev, slab))
    a.close()
    ctx.close()
