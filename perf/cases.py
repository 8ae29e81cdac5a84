"""The cases that performance work on this framework is measured by.

A case is the work a program has the framework do through its public entry
points: an area that takes one host frame and gives its output back every
cycle, an area that cycles through a block of frames already on the device,
several areas of uneven size in one batch, a hierarchy joined by tracts, a
serving tick, and the encoders that fill frame blocks. Area schemes are the
package's own (``bismit_b200.configs``); sizes run from the 24 x 24 grids of the
reference's test bed to the 256 x 256 area, on sides that are and are not
multiples of a tile, and over the shapes a tuft takes: dendrites of 1 to 64
synapses, cells of 1 to 1024, one to four source slices, scaled and nonspatial
sources.

Every output is a byte of an integer method (states, strengths, frames), so
results are compared for equality.
"""
import math

import numpy as np
import torch

from bismit_b200 import CorticalAreaSettings, area_desc, configs, plan_of
from bismit_b200 import _ffi as F
from bismit_b200.cortex import Batch, CorticalArea, Cortex, Server, _Ctx
from bismit_b200.encode import encode_2d_image

WARM_CYCLES = 6       # cycles run before the state is handed over: activity and learning have started
HOST_FRAMES = 8       # frames a host loop goes round
NO_BUF = 2 ** 64 - 1


def listed():
    return [
        # One 64 x 64 area in a sense-act loop: a host frame in, one cycle, the
        # output axons back on the host. The smallest call; latency is all of it.
        {"name": "live_64", "kind": "live", "scheme": "benchmark", "side": 64, "ssc": 32, "depth": 1, "prox": 1,
         "prox_syns": 1, "prox_reach": 0, "active": 0.02},
        # The same area left to learn through a block of frames on the device, with
        # synapse regrowth on (bismit's default), which fires once in 201 cycles.
        {"name": "area_64_regrow", "kind": "area", "scheme": "benchmark", "side": 64, "ssc": 32, "depth": 1,
         "prox": 1, "prox_syns": 1, "prox_reach": 0, "active": 0.02, "cycles": 201, "regrow": True},
        # The 256 x 256 area (272.6 M synapses), a training run's steady state:
        # frames resident, bandwidth-bound.
        {"name": "area_256", "kind": "area", "scheme": "benchmark", "side": 256, "ssc": 64, "depth": 4, "prox": 16,
         "prox_syns": 32, "prox_reach": 6, "active": 0.03, "cycles": 8, "regrow": False},
        # The same area driven live from the host, one frame at a time.
        {"name": "live_256", "kind": "live", "scheme": "benchmark", "side": 256, "ssc": 64, "depth": 4, "prox": 16,
         "prox_syns": 32, "prox_reach": 6, "active": 0.03},
        # A ragged side and the largest cells (16 dendrites of 64 synapses).
        {"name": "instance_150", "kind": "area", "scheme": "instance", "side": 150, "depth": 3, "dens": 16,
         "syns": 64, "active": 0.03, "cycles": 12, "regrow": False},
        # A population of independent instances of uneven size, cycled together
        # and replayed from a CUDA graph (a parameter study, an ensemble).
        {"name": "batch_24", "kind": "batch", "n": 24, "draw_seed": 0, "cycles": 6},
        # Three areas joined by feed-forward and feedback tracts.
        {"name": "hierarchy_3", "kind": "cortex", "side_a": 128, "side_b": 192, "side_c": 96, "depth": 2,
         "active": 0.02, "cycles": 12},
        # The reference's test bed layer map with its retina filter: small
        # dendrites (4 x 8 and 2 x 32), three source slices, reach 16.
        {"name": "testbed_96", "kind": "area", "scheme": "testbed", "side": 96, "retina": True, "active": 0.05,
         "cycles": 24, "regrow": False},
        # Scaled and nonspatial sources, dendrites of 12, 16 and 24 synapses,
        # two distal tufts that learn in turn, several controls on one layer.
        {"name": "mixed_100", "kind": "area", "scheme": "mixed", "side": 100, "src_side": 148, "active": 0.05,
         "cycles": 16, "regrow": False},
        # Activity smoothers on both layers, a side no tile divides.
        {"name": "smoother_120", "kind": "area", "scheme": "smoother", "side": 120, "radius": 3, "pyr_radius": 2,
         "active": 0.03, "cycles": 24, "regrow": False},
        # A server's steady state: every resident session has frames queued;
        # a pass submits them, ticks until they are cycled and reads the outputs.
        {"name": "serve_12", "kind": "serve", "n": 12, "draw_seed": 7, "frames": 4},
        # An image set resampled into hexagonal tract frames for a later run.
        {"name": "encode_images", "kind": "encode", "n": 2000, "x": 28, "y": 28, "v": 128, "u": 128, "scale": 1.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# The shapes of an instance's distal tuft, and the whole range of its layers.
_DENS, _SYNS = (8, 16), (16, 32, 64)
_MOST_BYTES = 15e9   # just below the 256 x 256 block: no drawn case costs more


def draw(rng):
    kind = rng.choice(("live", "area", "area", "instance", "instance", "batch", "cortex", "testbed", "mixed", "smoother",
                       "serve", "encode"))
    active = round(rng.uniform(0.01, 0.06), 4)
    if kind in ("live", "area"):
        side = _log_int(rng, 24, 256)
        deep = rng.random() < 0.5
        c = {"kind": kind, "scheme": "benchmark", "side": side, "ssc": rng.choice((32, 64)),
             "depth": rng.randint(1, 4) if deep else rng.randint(1, 2), "prox": 16 if deep else 1,
             "prox_syns": 32 if deep else 1, "prox_reach": rng.choice((3, 6)) if deep else 0, "active": active}
        if kind == "area":
            c["regrow"] = side <= 96 and rng.random() < 0.5
            c["cycles"] = 201 if c["regrow"] else rng.randint(4, 48)
    elif kind == "instance":
        c = {"kind": "area", "scheme": "instance", "side": _log_int(rng, 32, 192), "depth": rng.randint(1, 4),
             "dens": rng.choice(_DENS), "syns": rng.choice(_SYNS), "active": active, "cycles": rng.randint(4, 48),
             "regrow": False}
    elif kind == "batch":
        c = {"kind": "batch", "n": rng.randint(2, 24), "draw_seed": rng.randrange(1000), "cycles": rng.randint(2, 12)}
    elif kind == "cortex":
        a = _log_int(rng, 48, 128)
        b = int(a * rng.uniform(0.75, 1.5))   # a tuft's pool needs 32 offsets after scaling
        c = {"kind": "cortex", "side_a": a, "side_b": b, "side_c": int(b * rng.uniform(0.6, 1.2)),
             "depth": rng.randint(1, 2), "active": active, "cycles": rng.randint(4, 24)}
    elif kind == "testbed":
        retina = rng.random() < 0.5   # the filter takes sides that are multiples of 8
        c = {"kind": "area", "scheme": "testbed", "side": 8 * rng.randint(3, 16) if retina else rng.randint(24, 128),
             "retina": retina, "active": active, "cycles": rng.randint(8, 48), "regrow": False}
    elif kind == "mixed":
        side = rng.randint(24, 128)
        c = {"kind": "area", "scheme": "mixed", "side": side, "src_side": 2 * int(side * rng.uniform(0.4, 0.8)),
             "active": active, "cycles": rng.randint(6, 32), "regrow": False}
    elif kind == "smoother":
        c = {"kind": "area", "scheme": "smoother", "side": rng.randint(32, 160), "radius": rng.randint(2, 4),
             "pyr_radius": rng.randint(1, 3), "active": active, "cycles": rng.randint(8, 40), "regrow": False}
    elif kind == "serve":
        c = {"kind": "serve", "n": rng.randint(2, 14), "draw_seed": rng.randrange(1000), "frames": rng.randint(1, 6)}
    else:
        c = {"kind": "encode", "n": _log_int(rng, 8, 4000), "x": rng.randint(16, 64), "y": rng.randint(16, 64),
             "v": rng.randint(24, 256), "u": rng.randint(24, 256), "scale": round(rng.uniform(0.8, 1.2), 3)}
        c["n"] = max(1, min(c["n"], int(200e6 / (c["v"] * c["u"]))))
    while "cycles" in c and c["cycles"] > 2 and work(c)["bytes"] > _MOST_BYTES:
        c["cycles"] //= 2
        if c.get("regrow"):
            c["regrow"] = False   # too short a block for regrowth to fire in
    return c


# ------------------------------------------------------------- descriptors --
def _settings(regrow=False):
    s = CorticalAreaSettings()
    if not regrow:
        s.disable_regrowth()
    return s


def _area(case):
    k = case["scheme"]
    if k == "benchmark":
        lm = configs.benchmark_area(case["side"], case["ssc"], case["depth"], case["prox"], case["prox_syns"],
                                    case["prox_reach"])
    elif k == "instance":
        lm = configs.instance_area(case["side"], case["depth"], case["dens"], case["syns"])
    elif k == "testbed":
        lm = configs.testbed_area(case["side"], retina=case["retina"])
    elif k == "mixed":
        lm = configs.mixed_area(case["side"], case["src_side"])
    else:
        lm = configs.smoother_area(case["side"], case["radius"], case["pyr_radius"])
    return area_desc("v1", lm[0], lm[1], _settings(case.get("regrow", False)))


def _instances(case):
    return [(area_desc("v1", *configs.instance_area(side, depth, dens, syns), _settings()), act)
            for side, depth, dens, syns, act in configs.batch_instances(case["n"], case["draw_seed"])]


def _hierarchy(case):
    return configs.hierarchy((case["side_a"], case["side_b"], case["side_c"]), case["depth"])


def _cycle_bytes(p):
    """Bytes one cycle of the planned area cannot do without: a synapse's
    source (3), strength and state read, its state and flags written; a
    dendrite's activity read and written, its two states written; the eight
    cell-tuft bytes, four of them read too; 4 a cell; the input frame."""
    b = int(p.inputs[0].len) if p.n_inputs else 0
    for i in range(p.n_layers):
        L = p.layers[i]
        tufts = int(L.n_celtfts) if L.kind == F.BM_LYR_PYRAMIDAL else 0
        b += 7 * int(L.n_syns) + 4 * int(L.n_dens) + 12 * tufts + 4 * int(L.cells)
    return b


def work(case):
    k = case["kind"]
    if k == "encode":
        return {"bytes": case["n"] * (case["x"] * case["y"] + case["v"] * case["u"]), "flops": 0}
    if k in ("live", "area"):
        b = _cycle_bytes(plan_of(_area(case)))
    elif k == "cortex":
        lmaps, areas, names = _hierarchy(case)
        b = sum(_cycle_bytes(plan_of(area_desc(n, lmaps, areas, _settings()))) for n in names)
    else:
        b = sum(_cycle_bytes(plan_of(d)) for d, _ in _instances(case))
    return {"bytes": b * case.get("cycles", case.get("frames", 1)), "flops": 0}


# ------------------------------------------------------------------ states --
class _DeviceBytes:
    """n bytes of an area's slab; a tensor over it keeps the area (`owner`) alive."""

    def __init__(self, ptr, n, owner, signed=False):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": "|i1" if signed else "|u1",
                                         "data": (int(ptr), False), "version": 3, "strides": None}


def _view(ptr, n, owner, signed=False):
    return torch.as_tensor(_DeviceBytes(ptr, n, owner, signed), device="cuda:0")


def _slab(area):
    return _view(area.slab_ptr(), area.slab_bytes, area)


def _buffers(area):
    """{name: the area's own device buffer}: the axons and every buffer of every layer."""
    p, base = area.plan, area.slab_ptr()
    out = {"axons": _view(base + int(p.axon_off), p.n_axons, area)}
    for i in range(p.n_layers):
        L = p.layers[i]
        for k, name in enumerate(F.BUF_NAMES):
            if int(L.buf_off[k]) != NO_BUF and int(L.buf_len[k]):
                out["%d.%s" % (i, name)] = _view(base + int(L.buf_off[k]), L.buf_len[k], area,
                                                name in F.SIGNED_BUFS)
    return out


def _device_frames(n, length, active, seed):
    """n frames of input bytes: an axon is active with probability `active`, at 1..255."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    on = torch.rand(n, length, generator=g, device="cuda") < active
    v = torch.randint(1, 256, (n, length), generator=g, device="cuda", dtype=torch.uint8)
    out = torch.where(on, v, torch.zeros_like(v)).contiguous()
    torch.cuda.synchronize()
    return out


def _prepare_area(case, seed):
    ctx = _Ctx(0)
    a = CorticalArea(ctx, _area(case), seed, "v1")
    n = case.get("cycles", 1)
    length = a.input_len()
    if case.get("regrow"):
        # A state after a long run: strengths spread to and below the level
        # at which a synapse is given a new source.
        g = np.random.default_rng([seed, 1])
        for i in range(a.plan.n_layers):
            a.write("syn_strengths", g.integers(-40, 41, int(a.plan.layers[i].n_syns)).astype(np.int8), layer=i)
    for k in range(1, int(a.plan.n_inputs)):   # inputs that stay as they are through the pass
        a.write_input(configs.frames(1, a.input_len(k), case["active"], seed + k)[0], idx=k)
    warm = _device_frames(WARM_CYCLES, length, case["active"], seed + 1)
    a.cycle_frames_device(warm.data_ptr(), length, WARM_CYCLES)
    ctx.synchronize()
    s = {"kind": case["kind"], "ctx": ctx, "area": a, "len": length, "n": n, "out": _buffers(a)}
    if case["kind"] == "live":
        s["frames"] = configs.frames(HOST_FRAMES, length, case["active"], seed)
        s["at"] = 0
    else:
        s["frames"] = _device_frames(n, length, case["active"], seed)
    return s


def _prepare_batch(case, seed):
    ctx = _Ctx(0)
    ins = _instances(case)
    areas = [CorticalArea(ctx, d, seed + k, "v%d" % k) for k, (d, _) in enumerate(ins)]
    b = Batch(ctx, areas)

    def block(n, sd):
        return torch.cat([_device_frames(n, a.input_len(), act, sd + 100 * k)
                          for k, (a, (_, act)) in enumerate(zip(areas, ins))], dim=1).contiguous()

    warm, frames = block(WARM_CYCLES, seed + 1), block(case["cycles"], seed)
    torch.cuda.synchronize()
    b.cycle_frames_device(warm.data_ptr(), WARM_CYCLES)
    ctx.synchronize()
    return {"kind": "batch", "ctx": ctx, "areas": areas, "batch": b, "frames": frames, "n": case["cycles"],
            "out": [_slab(a) for a in areas]}


def _prepare_cortex(case, seed):
    lmaps, areas, names = _hierarchy(case)
    cx = Cortex.builder(lmaps, areas).ca_settings(_settings()).seed(seed).build()
    length = cx.batch.frame_bytes()
    warm = _device_frames(WARM_CYCLES, length, case["active"], seed + 1)
    cx.batch.cycle_frames_device(warm.data_ptr(), WARM_CYCLES)
    cx.synchronize()
    return {"kind": "cortex", "cortex": cx, "frames": _device_frames(case["cycles"], length, case["active"], seed),
            "n": case["cycles"], "out": [_slab(cx.area(n)) for n in names]}


def _prepare_serve(case, seed):
    ctx = _Ctx(0)
    ins = _instances(case)
    plans = [plan_of(d) for d, _ in ins]
    srv = Server(ctx, 32 << 30)
    sids = [srv.open(d, seed + k) for k, (d, _) in enumerate(ins)]
    frames = [configs.frames(case["frames"], int(p.inputs[0].len), act, seed + 100 * k)
              for k, (p, (_, act)) in enumerate(zip(plans, ins))]
    lens = [int(p.outputs[0].len) for p in plans]
    # Every session admitted, built and past its first frames; the resident set
    # is then stable and its tick settled.
    warm = 0
    while warm < 3:
        for sid, f in zip(sids, frames):
            srv.submit(sid, f)
        left = len(sids) * case["frames"]
        while left:
            left -= srv.tick()
        warm += 1
    srv.drain()
    return {"kind": "serve", "ctx": ctx, "server": srv, "sids": sids, "frames": frames, "lens": lens,
            "n": case["frames"]}


def _prepare_encode(case, seed):
    ctx = _Ctx(0)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    images = torch.randint(0, 256, (case["n"], case["y"], case["x"]), generator=g, device="cuda", dtype=torch.uint8)
    frames = torch.zeros(case["n"], case["v"] * case["u"], device="cuda", dtype=torch.uint8)
    torch.cuda.synchronize()
    return {"kind": "encode", "ctx": ctx, "images": images, "frames": frames, "src": (case["x"], case["y"]),
            "tar": (case["v"], case["u"]), "scale": case["scale"]}


def prepare(case, seed):
    k = case["kind"]
    if k in ("live", "area"):
        return _prepare_area(case, seed)
    return {"batch": _prepare_batch, "cortex": _prepare_cortex, "serve": _prepare_serve,
            "encode": _prepare_encode}[k](case, seed)


def run(s):
    k = s["kind"]
    if k == "area":
        s["area"].cycle_frames_device(s["frames"].data_ptr(), s["len"], s["n"])
        return s["out"]
    if k == "live":
        s["area"].write_input(s["frames"][s["at"]])
        s["at"] = (s["at"] + 1) % HOST_FRAMES
        s["area"].cycle(1)
        return {"output": s["area"].read_output(), **s["out"]}
    if k == "batch":
        s["batch"].cycle_frames_device(s["frames"].data_ptr(), s["n"])
        return s["out"]
    if k == "cortex":
        s["cortex"].batch.cycle_frames_device(s["frames"].data_ptr(), s["n"])
        return s["out"]
    if k == "serve":
        srv = s["server"]
        for sid, f in zip(s["sids"], s["frames"]):
            srv.submit(sid, f)
        for _ in range(s["n"]):
            srv.tick()
        srv.drain()
        return [srv.read_output(sid, n)[0] for sid, n in zip(s["sids"], s["lens"])]
    encode_2d_image(s["ctx"], s["images"], s["src"], s["tar"], s["scale"], s["frames"])
    return s["frames"]


def exact(case, seed):
    """No output is a computed number with a value in 64 bits: every one is a
    byte of an integer method (the image encoder's is a byte of the image that
    the reference's f32 geometry picks), held equal."""
    return None
