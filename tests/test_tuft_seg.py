"""Tufts at odd sizes, against the oracle on the whole slab (tolerance: exact):
the kernel for shapes the tiled one does not take (bm_seg.cuh) -- synapse
ranges off 16-byte alignment, dendrites and cells of odd lengths, cells larger
than a block's piece, scaled and nonspatial sources, both window widths, the
batched form -- and the tiled one with dendrites and cells off alignment."""
import numpy as np
import pytest

import oracle
from bismit_b200 import _ffi as F, configs, cortex, map as M
from helpers import diff_report, frames_for, initial_slab, settings_for

pytestmark = pytest.mark.gpu

# (label, scheme, the fused kernel takes the last layer's last tuft)
SHAPES = [
    ("unaligned_512", lambda: configs.instance_area(19, 1, 16, 32), True),
    ("unaligned_1024", lambda: configs.instance_area(51, 1, 16, 64), True),
    # Every specialised shape, at odd offsets, several slices and ragged rows.
    ("unaligned_128", lambda: configs.instance_area(23, 2, 8, 16), True),
    ("unaligned_256a", lambda: configs.instance_area(21, 3, 16, 16), True),
    ("unaligned_256b", lambda: configs.instance_area(27, 1, 8, 32), True),
    ("unaligned_512b", lambda: configs.instance_area(29, 3, 8, 64), True),
    ("unaligned_512c", lambda: configs.instance_area(66, 4, 16, 32), True),
    ("unaligned_1024b", lambda: configs.instance_area(37, 3, 16, 64), True),
    # Tiles of several stages, the last round's cut into parts.
    ("split_512", lambda: configs.instance_area(100, 1, 16, 32), True),
    ("split_512_unaligned", lambda: configs.instance_area(101, 1, 16, 32), True),
    ("split_1024", lambda: configs.instance_area(96, 2, 16, 64), True),
    ("split_1024_unaligned", lambda: configs.instance_area(90, 2, 16, 64), True),
    ("split_general", lambda: configs.instance_area(100, 2, 2, 128), True),
    ("wide_16", lambda: configs.instance_area(321, 3, 1, 8), False),           # 16-byte windows
    ("unaligned_16", lambda: configs.instance_area(33, 2, 1, 16), False),
    ("odd_21", lambda: configs.instance_area(32, 2, 3, 7), False),
    ("odd_24", lambda: configs.instance_area(17, 1, 1, 24), False),
    ("single", lambda: configs.instance_area(150, 1, 1, 1), False),            # too many cells to fold into the tail
    ("pieces_4800", lambda: configs.instance_area(11, 1, 40, 120), False),     # a cell in two pieces
    ("one_piece_2520", lambda: configs.instance_area(12, 1, 21, 120), False),
    ("odd_cells", lambda: configs.benchmark_area(21, 64, 3, 16, 32, 6), True),  # dendrites and cells off alignment
    ("odd_cells_256", lambda: configs.benchmark_area(23, 32, 3, 8, 32, 3), True),
    ("testbed", lambda: configs.testbed_area(25), None),
    ("mixed", lambda: configs.mixed_area(26, 38), None),
]


def _desc(mk, settings):
    lmaps, areas = mk()
    return M.area_desc("v1", lmaps, areas, settings)


@pytest.mark.parametrize("clean_flags", [False, True])
@pytest.mark.parametrize("label,mk,fused", SHAPES, ids=[s[0] for s in SHAPES])
def test_matches_oracle(label, mk, fused, clean_flags):
    ctx = cortex._Ctx(0)
    a = cortex.CorticalArea(ctx, _desc(mk, settings_for()), 7)
    if fused is not None:
        last = a.plan.n_layers - 1
        assert bool(a.tuft_form(last, a.plan.layers[last].n_tufts - 1)["fused"]) == fused
    slab = initial_slab(a.plan, 7, scramble_seed=11, clean_flags=clean_flags)
    a.write_slab(slab)
    fr = frames_for(a.plan, 3, 5)
    for k in range(3):
        a.write_input(fr[k])
        a.cycle(1)
        oracle.intake(a.plan, slab, 0, 0, fr[k])
        oracle.run(a.plan, slab, None, 1, start_cycle=k)
        dev = a.read_slab()
        assert np.array_equal(dev, slab), "cycle %d\n%s" % (k, diff_report(a.plan, dev, slab))
    a.close()
    ctx.close()


@pytest.mark.parametrize("sides", [(19, 33, 21), (65, 71, 30), (100, 96, 40), (101, 90, 39)])
def test_batched_matches_alone(sides):
    ctx = cortex._Ctx(0)
    descs = [_desc(lambda s=s: configs.instance_area(s, 1 + s % 2, 16, 32), settings_for()) for s in sides]
    alone = [cortex.CorticalArea(ctx, d, 3 + k) for k, d in enumerate(descs)]
    batched = [cortex.CorticalArea(ctx, d, 3 + k) for k, d in enumerate(descs)]
    b = cortex.Batch(ctx, batched)
    for c in range(4):
        for k, (x, y) in enumerate(zip(alone, batched)):
            f = configs.frames(1, x.input_len(), 0.05, 10 * c + k)[0]
            x.write_input(f)
            y.write_input(f)
            x.cycle(1)
        b.cycle(1)
    for x, y in zip(alone, batched):
        assert np.array_equal(x.read_slab(), y.read_slab())
    b.close()
    for a in alone + batched:
        a.close()
    ctx.close()


@pytest.mark.parametrize("shape", [(19, 1, 16, 32), (37, 3, 16, 64), (23, 2, 8, 16)])
@pytest.mark.parametrize("batched", [False, True])
def test_unaligned_sources_moved(shape, batched):
    """Regrowth moves sources of an unaligned tuft (its compiled codes and
    offsets follow), then the caller writes sources past the pool's reach (the
    tuft takes the windowed form) and back."""
    ctx = cortex._Ctx(0)
    a = cortex.CorticalArea(ctx, _desc(lambda: configs.instance_area(*shape), settings_for("regrowth")), 7)
    slab = initial_slab(a.plan, 7, scramble_seed=11, clean_flags=True)
    a.write_slab(slab)
    a.set_cycle(199)
    b = cortex.Batch(ctx, [a]) if batched else None
    fr = frames_for(a.plan, 5, 5)

    def step(k):
        a.write_input(fr[k])
        (b or a).cycle(1)
        oracle.intake(a.plan, slab, 0, 0, fr[k])
        oracle.run(a.plan, slab, None, 1, start_cycle=199 + k)
        dev = a.read_slab()
        assert np.array_equal(dev, slab), "cycle %d\n%s" % (199 + k, diff_report(a.plan, dev, slab))

    for k in range(3):   # fires in the cycle numbered 200
        step(k)
    last = a.plan.n_layers - 1
    off = int(a.plan.layers[last].buf_off[F.BUF["syn_src_col_v_offs"]])
    n = int(a.plan.layers[last].n_syns)
    keep = slab[off:off + n].copy()
    slab[off + n - 700:off + n:3] = 100
    a.write("syn_src_col_v_offs", slab[off:off + n].view(np.int8), layer=last)
    step(3)
    slab[off:off + n] = keep
    a.write("syn_src_col_v_offs", keep.view(np.int8), layer=last)
    step(4)
    if b:
        b.close()
    a.close()
    ctx.close()


def _small(side, depth, pyr):
    """configs.instance_area with the pyramidal cells given."""
    lmaps, areas = M.LayerMapSchemeList(), M.AreaSchemeList()
    ext = M.LayerMapScheme("v0_lm", M.LayerMapKind.Subcortical)
    ext.layer(M.LayerScheme.define("ganglion").depth(1).axonal(M.AxonTopology.Spatial)
              .axon_domain(M.AxonDomain.output([M.THAL_SP])))
    lmaps.add(ext)
    areas.area(M.AreaScheme("v0", "v0_lm", side))
    lm = M.LayerMapScheme("visual", M.LayerMapKind.Cortical)
    lm.layer(M.LayerScheme.define("aff_in").axonal(M.AxonTopology.Spatial)
             .axon_domain(M.AxonDomain.input([(M.InputTrack.Afferent, [M.THAL_SP])])))
    lm.layer(M.LayerScheme.define("iv").depth(1).tags(M.LayerTags.PSAL).axon_domain(M.AxonDomain.Local)
             .cellular(M.CellScheme.spiny_stellate()
                       .tft(M.TuftScheme.basal().proximal().syns_per_den(32)
                            .src_lyr(M.TuftSourceLayer.define("aff_in").syn_reach(6).prevalence(1)))))
    lm.layer(M.LayerScheme.define("iv_inhib").cellular(
        M.CellScheme.control(M.ControlCellKind.InhibitoryBasketSurround("iv", 4), 0)))
    lm.layer(M.LayerScheme.define("iii").depth(depth).tags(M.LayerTags.PTAL)
             .axon_domain(M.AxonDomain.output([M.THAL_SP])).cellular(pyr))
    lm.layer(M.LayerScheme.define("iii_col").cellular(
        M.CellScheme.control(M.ControlCellKind.IntraColumnInhib("iii"), 0)))
    lmaps.add(lm)
    areas.area(M.AreaScheme("v1", "visual", side).eff_areas(["v0"]))
    return lmaps, areas


@pytest.mark.parametrize("dens,syns,mad", [(1, 1, 0), (1, 1, 3), (2, 1, 1), (1, 3, 0), (2, 2, 0)])
@pytest.mark.parametrize("kind", ["proximal", "distal"])
@pytest.mark.parametrize("side,depth,batched", [(17, 1, False), (40, 3, True), (19, 9, False), (132, 1, False)])
def test_tufts_of_a_few_synapses(dens, syns, mad, kind, side, depth, batched):
    """Tufts of up to four synapses a cell: folded into the tail (one-synapse
    ones with every input loaded first), in columns deeper than a warp's
    group, as a distal tuft that learns, and too many to fold."""
    src = M.TuftSourceLayer.define("iv").syn_reach(2).prevalence(1)
    tiny = getattr(M.TuftScheme.basal(), kind)().dens_per_tft(dens).syns_per_den(syns).max_active_dens_l2(mad)
    other = "distal" if kind == "proximal" else "proximal"
    big = getattr(M.TuftScheme.basal(), other)().dens_per_tft(4).syns_per_den(16).max_active_dens_l2(1)
    l2, a2 = _small(side, depth, M.CellScheme.pyramidal().tft(tiny.src_lyr(src)).tft(big.src_lyr(src)))
    ctx = cortex._Ctx(0)
    a = cortex.CorticalArea(ctx, M.area_desc("v1", l2, a2, settings_for()), 7)
    slab = initial_slab(a.plan, 7, scramble_seed=11, clean_flags=True)
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


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("syns", [1, 2])
def test_few_synapses_from_the_layers_own_axons(syns, batched):
    """A tuft of a few synapses that reads the axons its layer's tail writes, by
    its pool or because the caller wrote such sources, does not run inside that
    tail."""
    own = M.TuftSourceLayer.define("iii").syn_reach(5).prevalence(1)
    iv = M.TuftSourceLayer.define("iv").syn_reach(5).prevalence(1)

    def tuft(kind, src):
        return getattr(M.TuftScheme.basal(), kind)().dens_per_tft(1).syns_per_den(syns).max_active_dens_l2(0).src_lyr(src)

    for srcs in ((iv, own), (iv, iv)):
        l2, a2 = _small(70, 2, M.CellScheme.pyramidal().tft(tuft("proximal", srcs[0])).tft(tuft("distal", srcs[1])))
        ctx = cortex._Ctx(0)
        a = cortex.CorticalArea(ctx, M.area_desc("v1", l2, a2, settings_for()), 7)
        slab = initial_slab(a.plan, 7, scramble_seed=11, clean_flags=True)
        a.write_slab(slab)
        b = cortex.Batch(ctx, [a]) if batched else None
        fr = frames_for(a.plan, 12, 5, active=0.2)
        for k in range(12):
            if k == 4 and srcs[1] is iv:   # the layer's own slices, from here on
                last = a.plan.layers[1]
                off = int(last.buf_off[F.BUF["syn_src_slc_ids"]])
                slab[off:off + int(last.n_syns)] = int(last.base_axn_slc) + np.arange(int(last.n_syns)) % 2
                a.write("syn_src_slc_ids", slab[off:off + int(last.n_syns)], layer=1)
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


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("mk", [
    lambda: configs.benchmark_area(48, 64, 4, 16, 32, 6), lambda: configs.benchmark_area(33, 32, 1, 8, 32, 3),
    lambda: configs.instance_area(100, 1, 16, 32), lambda: configs.instance_area(96, 2, 16, 64),
    lambda: configs.instance_area(64, 3, 8, 16), lambda: configs.instance_area(80, 5, 8, 64),
    lambda: configs.smoother_area(35, 3, 2)],
    ids=["bench48", "bench33", "split_512", "split_1024", "three_slices", "five_slices", "smoother35"])
def test_foreign_flags_come_and_go(mk, batched):
    """Flag bytes with bits besides SYN_PREV_ACTIVE, in one synapse and in all:
    the tuft's flags are streamed through, its compiled sources stay in use."""
    ctx = cortex._Ctx(0)
    a = cortex.CorticalArea(ctx, _desc(mk, settings_for()), 7)
    slab = initial_slab(a.plan, 7, scramble_seed=11, clean_flags=True)
    a.write_slab(slab)
    b = cortex.Batch(ctx, [a]) if batched else None
    fr = frames_for(a.plan, 4, 5)
    rng = np.random.default_rng(4)
    for k in range(4):
        for l in range(a.plan.n_layers):
            n = int(a.plan.layers[l].n_syns)
            off = int(a.plan.layers[l].buf_off[F.BUF["syn_flag_sets"]])
            flags = slab[off:off + n]
            if k == 1:
                flags[n - 1] |= 0x40
            elif k == 2:
                flags |= rng.integers(0, 256, n, dtype=np.uint8) & 0xEF
            elif k == 3:
                flags &= 0x10
            if k:
                a.write("syn_flag_sets", flags, layer=l)
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


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("dens,syns", [(1, 1), (1, 4), (2, 1), (2, 2), (4, 1), (2, 4)])
def test_spiny_stellate_cells_of_a_few_synapses(dens, syns, batched):
    """Spiny stellate cells have no cell-tuft arrays: one dendrite a cell (with
    the folded soma step) and several."""
    src = M.TuftSourceLayer.define("iv").syn_reach(2).prevalence(1)
    l2, a2 = _small(21, 2, M.CellScheme.pyramidal().tft(
        M.TuftScheme.basal().proximal().dens_per_tft(2).syns_per_den(2).src_lyr(src)))
    for layer in l2["visual"].layers:
        if layer.name == "iv":
            layer.cellular(M.CellScheme.spiny_stellate().tft(
                M.TuftScheme.basal().proximal().dens_per_tft(dens).syns_per_den(syns)
                .src_lyr(M.TuftSourceLayer.define("aff_in").syn_reach(3).prevalence(1))))
    ctx = cortex._Ctx(0)
    a = cortex.CorticalArea(ctx, M.area_desc("v1", l2, a2, settings_for()), 7)
    assert int(a.plan.layers[0].tufts[0].syns_per_tft) == dens * syns
    slab = initial_slab(a.plan, 7, scramble_seed=11, clean_flags=True)
    a.write_slab(slab)
    b = cortex.Batch(ctx, [a]) if batched else None
    fr = frames_for(a.plan, 3, 5, active=0.2)
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
