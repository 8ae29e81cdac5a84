"""The activity smoother's two launches against the oracle on the whole slab
(tolerance: exact): group sides around a warp's 32 positions, layers smaller
than a hexagon, several slices, energies at both ends of their range, batched."""
import numpy as np
import pytest

import oracle
from bismit_b200 import configs, cortex, map as M
from helpers import diff_report, frames_for, initial_slab, settings_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,radius,pyr_radius", [(40, 1, 1), (33, 2, 3), (57, 3, 2), (24, 9, 7), (16, 17, 1)])
@pytest.mark.parametrize("batched", [False, True])
def test_sizes_match_oracle(side, radius, pyr_radius, batched):
    ctx = cortex._Ctx(0)
    lmaps, areas = configs.smoother_area(side, radius, pyr_radius)
    a = cortex.CorticalArea(ctx, M.area_desc("v1", lmaps, areas, settings_for()), 7)
    slab = initial_slab(a.plan, 7, scramble_seed=3, clean_flags=True)
    # Energies and activities at the ends of their ranges, where the order of
    # the six lattices shows.
    from bismit_b200 import _ffi as F
    rng = np.random.default_rng(side)
    for i in range(a.plan.n_layers):
        L = a.plan.layers[i]
        for k in ("cel_energies", "cel_activities"):
            off = int(L.buf_off[F.BUF[k]])
            slab[off:off + int(L.cells)] = rng.choice([0, 0, 1, 2, 100, 254, 255, 255], int(L.cells)).astype(np.uint8)
    a.write_slab(slab)
    b = cortex.Batch(ctx, [a]) if batched else None
    fr = frames_for(a.plan, 3, 5)
    for k in range(3):
        a.write_input(fr[k])
        (b or a).cycle(1)
        oracle.intake(a.plan, slab, 0, 0, fr[k])
        oracle.run(a.plan, slab, None, 1, start_cycle=k)
        dev = a.read_slab()
        assert np.array_equal(dev, slab), "cycle %d\n%s" % (k, diff_report(a.plan, dev, slab))
    if b:
        b.close()
    a.close()
    ctx.close()


@pytest.mark.parametrize("inhib,smooth", [(1, 2), (2, 1)])
def test_with_basket_inhibition_on_the_pyramidal_layer(inhib, smooth):
    """A basket inhibition writes the activities a smoother reads, whichever
    runs first; learning follows both."""
    ctx = cortex._Ctx(0)
    lmaps, areas = configs.smoother_area(35, 3, 2, smoothers=False)
    lm = lmaps["visual"]
    lm.layer(M.LayerScheme.define("iii_inhib").cellular(
        M.CellScheme.control(M.ControlCellKind.InhibitoryBasketSurround("iii", 3), inhib)))
    lm.layer(M.LayerScheme.define("iii_smooth").cellular(
        M.CellScheme.control(M.ControlCellKind.ActivitySmoother("iii", 2), smooth)))
    a = cortex.CorticalArea(ctx, M.area_desc("v1", lmaps, areas, settings_for()), 7)
    slab = initial_slab(a.plan, 7, scramble_seed=3, clean_flags=True)
    a.write_slab(slab)
    fr = frames_for(a.plan, 4, 5)
    for k in range(4):
        a.write_input(fr[k])
        a.cycle(1)
        oracle.intake(a.plan, slab, 0, 0, fr[k])
        oracle.run(a.plan, slab, None, 1, start_cycle=k)
        dev = a.read_slab()
        assert np.array_equal(dev, slab), "cycle %d\n%s" % (k, diff_report(a.plan, dev, slab))
    a.close()
    ctx.close()


def _with_controls(host, orders):
    """configs.smoother_area's scheme with the controls of layer `host` run in
    the order given: "basket" (a basket inhibition) or a smoother's group side."""
    lmaps, areas = configs.smoother_area(35, 3, 2, smoothers=False)
    lm = lmaps["visual"]
    lm.layers[:] = [l for l in lm.layers if l.name not in ("iv_inhib", "iii_col") or not l.name.startswith(host + "_")]
    for k, what in enumerate(orders):
        kind = (M.ControlCellKind.InhibitoryBasketSurround(host, 4) if what == "basket"
                else M.ControlCellKind.ActivitySmoother(host, what))
        lm.layer(M.LayerScheme.define("%s_c%d" % (host, k)).cellular(M.CellScheme.control(kind, k)))
    return lmaps, areas


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("kind", ["default", "bypass_inhib", "no_learning"])
@pytest.mark.parametrize("orders", [("basket", 3), (3, "basket"), (2, "basket", 3), (2, 3, "basket"), ("basket", 2, 3)],
                         ids=lambda o: "-".join(str(x) for x in o))
@pytest.mark.parametrize("host", ["iv", "iii"])
def test_smoothers_around_a_basket_inhibition(host, orders, kind, batched):
    """A basket inhibition rewrites the activities that smoothers pick by: those
    ordered before it pick by the old ones, those after it by the new ones."""
    ctx = cortex._Ctx(0)
    lmaps, areas = _with_controls(host, orders)
    a = cortex.CorticalArea(ctx, M.area_desc("v1", lmaps, areas, settings_for(kind)), 7)
    slab = initial_slab(a.plan, 7, scramble_seed=3, clean_flags=True)
    a.write_slab(slab)
    b = cortex.Batch(ctx, [a]) if batched else None
    fr = frames_for(a.plan, 4, 5)
    for k in range(4):
        a.write_input(fr[k])
        (b or a).cycle(1)
        oracle.intake(a.plan, slab, 0, 0, fr[k])
        oracle.run(a.plan, slab, None, 1, start_cycle=k)
        dev = a.read_slab()
        assert np.array_equal(dev, slab), "cycle %d\n%s" % (k, diff_report(a.plan, dev, slab))
    if b:
        b.close()
    a.close()
    ctx.close()
