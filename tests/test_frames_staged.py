"""Host frames and outputs on both sides of the sizes up to which a copy kernel
moves them over the host link (64 KB, 256 KB), in turns and without a wait
between them, against the oracle or the state slab (tolerance: exact)."""
import numpy as np
import pytest

import oracle
from bismit_b200 import configs, cortex, map as M
from helpers import diff_report, initial_slab, settings_for

pytestmark = pytest.mark.gpu

LIMIT = 64 << 10


def _two_inputs(src_side=252, src_depth=5, side=40):
    """A small area with a spatial input of src_depth slices and a nonspatial
    one (the spiny stellate layer reads the first, the apical tuft the other)."""
    lmaps, areas = M.LayerMapSchemeList(), M.AreaSchemeList()
    configs._external(lmaps, areas, "v0", src_side, nonspatial=True, depth=src_depth)
    lm = M.LayerMapScheme("visual", M.LayerMapKind.Cortical)
    lm.layer(M.LayerScheme.define("aff_in").axonal(M.AxonTopology.Spatial)
             .axon_domain(M.AxonDomain.input([(M.InputTrack.Afferent, [M.THAL_SP])])))
    lm.layer(M.LayerScheme.define("ns_in").axonal(M.AxonTopology.Nonspatial)
             .axon_domain(M.AxonDomain.input([(M.InputTrack.Afferent, [M.THAL_NSP])])))
    lm.layer(M.LayerScheme.define("iv").depth(1).tags(M.LayerTags.PSAL).axon_domain(M.AxonDomain.Local)
             .cellular(M.CellScheme.spiny_stellate()
                       .tft(M.TuftScheme.basal().proximal().syns_per_den(32)
                            .src_lyr(M.TuftSourceLayer.define("aff_in").syn_reach(6).prevalence(1)))))
    lm.layer(M.LayerScheme.define("iv_inhib").cellular(
        M.CellScheme.control(M.ControlCellKind.InhibitoryBasketSurround("iv", 4), 0)))
    lm.layer(M.LayerScheme.define("iii").depth(1).tags(M.LayerTags.PTAL)
             .axon_domain(M.AxonDomain.output([M.THAL_SP]))
             .cellular(M.CellScheme.pyramidal()
                       .tft(M.TuftScheme.basal().proximal().dens_per_tft(1).syns_per_den(1)
                            .src_lyr(M.TuftSourceLayer.define("iv").syn_reach(0).prevalence(1)))
                       .tft(M.TuftScheme.apical().distal().dens_per_tft(4).syns_per_den(16).max_active_dens_l2(1)
                            .src_lyr(M.TuftSourceLayer.define("ns_in").syn_reach(0).prevalence(1)))))
    lm.layer(M.LayerScheme.define("iii_col").cellular(
        M.CellScheme.control(M.ControlCellKind.IntraColumnInhib("iii"), 0)))
    lmaps.add(lm)
    areas.area(M.AreaScheme("v1", "visual", side).eff_areas(["v0"]))
    return lmaps, areas


# Which input each write of a cycle feeds: 0 the large one, 1 the small one.
ORDERS = [(0, 1), (1, 0, 1, 1, 0), (0, 0, 1), (1, 1, 1, 1, 1, 0, 0, 0, 1), (0, 0, 0, 0, 1)]


@pytest.mark.parametrize("src_depth", [2, 5])
def test_large_and_small_frames_in_turns(src_depth):
    ctx = cortex._Ctx(0)
    lmaps, areas = _two_inputs(src_depth=src_depth)
    a = cortex.CorticalArea(ctx, M.area_desc("v1", lmaps, areas, settings_for()), 7)
    lens = [a.input_len(i) for i in range(2)]
    assert lens[0] > LIMIT > lens[1]
    slab = initial_slab(a.plan, 7, scramble_seed=3, clean_flags=True)
    a.write_slab(slab)
    rng = np.random.default_rng(2)
    for k, order in enumerate(ORDERS + ORDERS[::-1]):
        for i in order:
            f = rng.integers(0, 256, lens[i], dtype=np.uint8)
            f[rng.random(lens[i]) < 0.8] = 0
            a.write_input(f, i)
            oracle.intake(a.plan, slab, i, 0, f)
            f[:] = 255   # the bytes are read during the call only
        a.cycle(1)
        oracle.run(a.plan, slab, None, 1, start_cycle=k)
        if k % 3 != 1:
            continue
        dev = a.read_slab()
        assert np.array_equal(dev, slab), "cycle %d\n%s" % (k, diff_report(a.plan, dev, slab))
    dev = a.read_slab()
    assert np.array_equal(dev, slab), diff_report(a.plan, dev, slab)
    a.close()
    ctx.close()


@pytest.mark.parametrize("side,depth", [(23, 1), (256, 4), (229, 5), (230, 5)])
def test_outputs_on_both_sides_of_the_limit(side, depth):
    """The output read back is the slab's, into pageable and page-locked memory."""
    import ctypes as C

    import torch

    from bismit_b200 import _ffi as F
    ctx = cortex._Ctx(0)
    a = cortex.CorticalArea(ctx, M.area_desc("v1", *configs.instance_area(side, depth, 8, 16), settings_for()), 7)
    n = a.output_len()
    assert n == side * side * depth
    rng = np.random.default_rng(side)
    pinned = torch.zeros(n, dtype=torch.uint8).pin_memory()
    for k in range(3):
        ax = rng.integers(0, 256, int(a.plan.n_axons), dtype=np.uint8)
        a.write("axon_states", ax)
        a.cycle(1)
        z = int(a.plan.axon_off) + int(a.plan.outputs[0].axn_idz)
        out = np.array(a.read_output())
        F.check(a.lib.bm_area_read_output(a.h, 0, C.c_void_p(pinned.data_ptr()), n))
        want = a.read_slab()[z:z + n]
        assert np.array_equal(out, want)
        assert np.array_equal(pinned.numpy(), want)
    a.close()
    ctx.close()
