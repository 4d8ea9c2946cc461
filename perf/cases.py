"""Performance cases of the out-of-core volume path.

Every case is one call sequence that a program using this library makes, over
the range of volumes, bricks, images and options the library is used with:

  frame   one frame of a camera whose bricks are resident: restart the
          progressive buffers, ray-cast, cache update (LRU + request scan)
  loop    a few views rendered to convergence one after the other through a
          pool too small for all of them: ray-cast / request / load / install
          until the update reports an empty miss list
  batch   uneven views submitted to the continuous batch and ticked until
          all have retired
  mip     the mip pyramid of a volume
  prep    ingesting a volume: mip pyramid, bricking of every level, empty
          flags and value bins of every brick
  miss    the allocation-free miss list of a recorded request buffer

A case is a dict of plain values; prepare() makes what the program holds before
the call, run() is the call, work() its compulsory bytes and operations and
exact() the ray caster's (and the float pyramid's) values in 64 bits.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "gpu-out-of-core-volume-data_gb300")
for _p in (_ROOT, _PKG):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import gcgb300 as gc  # noqa: E402

DIAG = 2.0 * math.sqrt(3.0)  # diagonal of the view box [-1, 1]^3
TSTEP = 2.0 / 256.0
MAX_ITERATIONS = 200         # render / update iterations of one view of a loop
MAX_TICKS = 20000


def _frame(name, size, eb, ch, B, c, bb, W, H, dist, dvr, tri, fast, pt):
    return {"name": name, "kind": "frame", "x": size[0], "y": size[1], "z": size[2], "eb": eb, "ch": ch, "B": B,
            "c": c, "bb": bb, "W": W, "H": H, "dist": dist, "dvr": dvr, "tri": tri, "fast": fast, "pt": pt}


def listed():
    return [
        # the smallest interactive frame (a thumbnail): launches and host latency
        _frame("frame_thumb_u8", (64, 64, 64), 1, 1, 16, 1, 1, 128, 128, 1.0, True, False, False, 0),
        # the in-core orbit: 256^3 u8, 512^2 at twice the diagonal
        _frame("frame_orbit_u8", (256, 256, 256), 1, 1, 16, 1, 1, 512, 512, 2.0, True, False, False, 0),
        # a full-window view of a 16-bit volume with the fast arithmetic
        _frame("frame_u16_fast", (512, 512, 512), 2, 1, 16, 1, 1, 1024, 1024, 0.9, True, False, True, 0),
        # maximum intensity, trilinear, large bricks, a wide image, a volume of uneven sides
        _frame("frame_mop_hd", (512, 448, 288), 1, 1, 32, 1, 1, 1920, 1080, 0.8, False, True, False, 0),
        # two interleaved channels, 2D transfer function, covering 2, big bricks, two-level directory, odd image
        _frame("frame_two_channel", (256, 256, 256), 2, 2, 16, 2, 2, 777, 555, 0.7, True, False, False, 8),
        # paging: three views of a 16-bit volume from a page-locked host store through a small pool
        {"name": "loop_host_u16", "kind": "loop", "x": 512, "y": 512, "z": 512, "eb": 2, "B": 16, "W": 1024,
         "H": 1024, "views": 3, "far": 1.6, "near": 0.6, "pool_mib": 256, "requests": 8192, "source": "host",
         "fast": True},
        # paging of a large volume whose pyramid stays on the device, the reference-sized image
        {"name": "loop_device_u8", "kind": "loop", "x": 1024, "y": 1024, "z": 1024, "eb": 1, "B": 16, "W": 512,
         "H": 512, "views": 3, "far": 2.0, "near": 0.5, "pool_mib": 128, "requests": 4096, "source": "device",
         "fast": False},
        # the batched form: uneven images in one persistent launch, overlapped loads, bricks resident
        {"name": "batch_mixed_u16", "kind": "batch", "x": 512, "y": 512, "z": 512, "eb": 2, "B": 32, "views": 24,
         "overlap": True, "pool_mib": 1024, "fast": True},
        # the pyramid of a large 16-bit volume
        {"name": "mip_u16", "kind": "mip", "x": 1024, "y": 1024, "z": 1024, "eb": 2, "ch": 1, "float": False},
        # ingesting a scan with odd sides: rows of no whole 16 bytes, odd levels
        {"name": "prep_odd_u8", "kind": "prep", "x": 381, "y": 347, "z": 291, "eb": 1, "ch": 1, "B": 16, "c": 1,
         "bb": 1},
        # ingesting a large 16-bit volume
        {"name": "prep_u16", "kind": "prep", "x": 768, "y": 768, "z": 768, "eb": 2, "ch": 1, "B": 16, "c": 1,
         "bb": 1},
        # the request buffer of a 2048^3 volume in 16^3 bricks: 6.4 M entries
        {"name": "miss_2048", "kind": "miss", "x": 2048, "y": 2048, "z": 2048, "B": 16, "c": 1, "requests": 8192,
         "missing": 5000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "loop", "batch", "mip", "prep", "prep", "miss"))
    if kind == "frame":
        ch = rng.choice((1, 1, 1, 2))
        eb = 2 if ch == 2 else rng.choice((1, 2))
        size = [_log(rng, 64, 512 if eb == 1 else 448) for _ in range(3)]
        W, H = _log(rng, 100, 1600), _log(rng, 100, 1000)
        return {"kind": kind, "x": size[0], "y": size[1], "z": size[2], "eb": eb, "ch": ch,
                "B": rng.choice((8, 16, 16, 32)) if min(size) >= 128 else 16, "c": rng.choice((1, 1, 2)),
                "bb": rng.choice((1, 1, 2)), "W": W, "H": H, "dist": round(rng.uniform(0.5, 2.0), 3),
                "dvr": rng.choice((True, True, False)), "tri": rng.choice((True, False)),
                "fast": rng.choice((True, False)), "pt": rng.choice((0, 0, 0, 4, 8))}
    if kind == "loop":
        n = _log(rng, 192, 512)
        return {"kind": kind, "x": n, "y": _log(rng, 192, 512), "z": _log(rng, 192, 512), "eb": rng.choice((1, 2)),
                "B": rng.choice((16, 16, 32)), "W": _log(rng, 200, 1024), "H": _log(rng, 200, 1024),
                "views": rng.randint(2, 3), "far": round(rng.uniform(1.2, 2.0), 3),
                "near": round(rng.uniform(0.5, 0.9), 3), "pool_mib": _log(rng, 64, 256),
                "requests": rng.choice((50, 1024, 1024)), "source": rng.choice(("host", "device")),
                "fast": rng.choice((True, False))}
    if kind == "batch":
        return {"kind": kind, "x": _log(rng, 128, 512), "y": _log(rng, 128, 512), "z": _log(rng, 128, 512),
                "eb": rng.choice((1, 2)), "B": rng.choice((16, 32)), "views": rng.randint(3, 24),
                "overlap": rng.choice((True, False)), "pool_mib": 1024, "fast": rng.choice((True, False))}
    if kind == "mip":
        real = rng.choice((False, False, True))
        ch = 1 if real else rng.choice((1, 1, 2))
        eb = 4 if real else ch * rng.choice((1, 2))
        odd = rng.choice((0, 0, 1))
        size = [_log(rng, 64, 800) // 16 * 16 + (odd * rng.randint(1, 15)) for _ in range(3)]
        return {"kind": kind, "x": size[0], "y": size[1], "z": size[2], "eb": eb, "ch": ch, "float": real}
    if kind == "prep":
        ch = rng.choice((1, 1, 1, 2))
        eb = ch * rng.choice((1, 2)) if ch == 1 else 2
        odd, B = rng.choice((0, 1)), rng.choice((8, 16, 16, 32))
        size = [_log(rng, 128 if B == 8 else 64, 600) // 16 * 16 + (odd * rng.randint(1, 15)) for _ in range(3)]
        return {"kind": kind, "x": size[0], "y": size[1], "z": size[2], "eb": eb, "ch": ch, "B": B, "c": rng.choice((1, 1, 2)), "bb": rng.choice((1, 1, 2))}
    n = _log(rng, 256, 2048)
    return {"kind": "miss", "x": n, "y": _log(rng, 256, 2048), "z": _log(rng, 256, 2048), "B": rng.choice((16, 32)),
            "c": rng.choice((1, 2)), "requests": rng.choice((50, 1024, 8192)), "missing": _log(rng, 10, 100000)}


# ---------------------------------------------------------------------------
# Inputs: seeded volumes, transfer functions and cameras.

def _field(size, gen, blobs):
    """Sum of anisotropic Gaussian blobs and smooth value noise in [0, 1], (z, y, x)."""
    x, y, z = size
    f = torch.nn.functional.interpolate(
        torch.rand((1, 1) + tuple(max(2, n // 24) for n in (z, y, x)), generator=gen, device="cuda"),
        size=(z, y, x), mode="trilinear", align_corners=False)[0, 0] * 0.1
    p = torch.rand((blobs, 7), generator=gen, device="cuda").cpu().numpy()
    for b in p:
        g = []
        for a, n in enumerate((x, y, z)):
            at = torch.arange(n, device="cuda", dtype=torch.float32)
            s = n * (0.04 + 0.12 * float(b[3 + a]))
            g.append(torch.exp(-0.5 * ((at - float(b[a]) * n) / s) ** 2))
        g[0] *= 0.25 + 0.55 * float(b[6])
        f += g[2][:, None, None] * (g[1][:, None] * g[0][None, :])
    return f.clamp_(0.0, 1.0)


def _volume(case, seed):
    """Level 0 as bytes: (z, y, x, channel) voxels of the case's width."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000003 * seed + 17)
    size, ch = (case["x"], case["y"], case["z"]), case.get("ch", 1)
    cb = case["eb"] // ch
    parts = []
    for k in range(ch):
        f = _field(size, gen, 10 if k == 0 else 3)
        if case.get("float"):
            parts.append(f.mul_(4095.0))
            continue
        f.mul_(255.0 if cb == 1 else 65535.0).add_(0.5)
        parts.append(f.to(torch.uint8) if cb == 1 else f.to(torch.int32).to(torch.int16))
        del f
    v = parts[0] if ch == 1 else torch.stack(parts, -1)
    return v.contiguous().reshape(-1).view(torch.uint8)


def _tf(case, seed):
    """Transfer function: three seeded Gaussian bumps of opacity (one channel),
    or a 2D table (two channels)."""
    rng = np.random.default_rng(seed + 101)
    w = 256 if case.get("ch", 1) == 1 else 64
    x = np.linspace(0.0, 1.0, w)
    a = np.zeros(w)
    for k in range(3):
        a += rng.uniform(0.2, 0.7) * np.exp(-0.5 * ((x - rng.uniform(0.25 + 0.2 * k, 0.4 + 0.2 * k)) /
                                                    rng.uniform(0.03, 0.08)) ** 2)
    tf = np.stack([np.clip(0.3 + x, 0, 1), np.clip(1.2 - x, 0, 1), 0.5 + 0.5 * np.sin(6 * x), np.clip(a, 0, 1)], 1)
    if case.get("ch", 1) == 2:
        y = np.linspace(0.0, 1.0, 48)[:, None, None]
        tf = tf[None] * np.concatenate([np.ones((48, 1, 3)), 0.3 + 0.7 * y], 2)
    return tf.astype(np.float32)


def _camera(rng, dist):
    """A camera on a sphere of `dist` diagonals, looking near the centre."""
    v = rng.standard_normal(3)
    v[1] *= 0.4
    v /= np.linalg.norm(v)
    return gc.look_at(tuple(float(q) * dist * DIAG for q in v), tuple(float(q) for q in rng.uniform(-0.1, 0.1, 3)))


FOCAL = 1.0 / math.tan(math.radians(45.0) / 2)


class _Image:
    """One view's buffers on the device and its gc_view."""

    def __init__(self, case, cam, W, H, tf, tf_dev):
        self.rgba = torch.zeros(W * H, dtype=torch.int32, device="cuda")
        self.t = torch.zeros(W * H, dtype=torch.float32, device="cuda")
        self.state = torch.zeros(W * H * 4, dtype=torch.float32, device="cuda")
        self.cam = cam
        two = tf.ndim == 3
        self.view = gc.make_view(
            cam, W, H, tf_dev.data_ptr(), tf.shape[-2], self.rgba.data_ptr(), self.t.data_ptr(),
            self.state.data_ptr(), tstep=TSTEP, focal=FOCAL, early_alpha=0.99,
            mode=gc.MODE_DVR if case.get("dvr", True) else gc.MODE_MOP,
            sampler=gc.SAMPLER_TRILINEAR if case.get("tri") else gc.SAMPLER_REFERENCE,
            tf_height=tf.shape[0] if two else 0)

    def restart(self):
        self.t.zero_()
        self.state.zero_()

    def outputs(self):
        return {"rgba": self.rgba, "t": self.t, "state": self.state}


def _desc(case):
    bb = case.get("bb", 1)
    vol = gc.volume_desc((case["x"], case["y"], case["z"]), case["B"], case.get("c", 1), case.get("eb", 1),
                         case.get("ch", 1), (bb, bb, bb))
    return vol, gc.compute_layout(vol)


def _precision(case):
    gc.render_precision(gc.RENDER_FAST if case.get("fast") else gc.RENDER_EXACT)


def _pyramid(case, vol, layout, seed):
    """Level 0 in a pyramid buffer (the other levels not built yet)."""
    offs, total = gc.pyramid_offsets(layout, case["eb"])
    pyr = torch.zeros(total, dtype=torch.uint8, device="cuda")
    v = _volume(case, seed)
    pyr[: v.numel()].copy_(v)
    return pyr, offs


def _cache(case, vol, layout, slots, requests, seed, source="device", sync=True, pt=0, pt_slots=0):
    """A cache over the case's volume, its bricks cut from a device pyramid or
    read from a page-locked host store."""
    cm = gc.CacheManager(vol, layout, slots, max_requests=requests, sync_loader=sync, pt_block=pt,
                         pt_slots=pt_slots)
    if source == "host":
        store, offs, _ = gc.pre_process(vol, layout, _volume(case, seed), pin=True)
        cm.set_source_host(store, offs)
    else:
        pyr, offs = _pyramid(case, vol, layout, seed)
        gc.Mipmapper.process(pyr.data_ptr(), layout, offs, case["eb"], case.get("ch", 1))
        cm.set_source_device(pyr.data_ptr(), offs, keep=pyr)
    return cm


def _bricks(layout):
    return [layout.nb_bricks[l][0] * layout.nb_bricks[l][1] * layout.nb_bricks[l][2] for l in range(layout.nb_levels)]


# ---------------------------------------------------------------------------

def _prepare_frame(case, seed):
    vol, layout = _desc(case)
    edge = math.ceil(max(sum(_bricks(layout)), 64) ** (1.0 / 3.0))  # room for every brick
    pt, pt_slots = case["pt"], 0
    if pt:
        pt_slots = sum((-(-layout.nb_bricks[l][0] // pt)) * (-(-layout.nb_bricks[l][1] // pt)) *
                       (-(-layout.nb_bricks[l][2] // pt)) for l in range(layout.nb_levels))
    cm = _cache(case, vol, layout, (edge, edge, edge), min(8192, edge ** 3), seed, pt=pt, pt_slots=pt_slots)
    tf = _tf(case, seed)
    tf_dev = torch.from_numpy(tf.reshape(-1)).cuda()
    im = _Image(case, _camera(np.random.default_rng(seed), case["dist"]), case["W"], case["H"], tf, tf_dev)
    _precision(case)
    for _ in range(8):  # until a frame from its start meets no missing brick
        im.restart()
        for frame in range(2000):
            cm.render(im.view)
            if cm.update():
                break
        if frame == 0:
            break
    return {"kind": "frame", "cm": cm, "image": im, "tf": tf_dev}


def _prepare_loop(case, seed):
    vol, layout = _desc(case)
    slots = gc.pool_dims(vol, case["pool_mib"] << 20)
    requests = min(case["requests"], slots[0] * slots[1] * slots[2])
    cm = _cache(case, vol, layout, slots, requests, seed, source=case["source"])
    tf = _tf(case, seed)
    tf_dev = torch.from_numpy(tf.reshape(-1)).cuda()
    rng = np.random.default_rng(seed)
    ims = []
    for k in range(case["views"]):
        d = case["far"] + (case["near"] - case["far"]) * k / max(1, case["views"] - 1)
        ims.append(_Image(case, _camera(rng, d), case["W"], case["H"], tf, tf_dev))
    _precision(case)
    return {"kind": "loop", "cm": cm, "images": ims, "tf": tf_dev}


def _prepare_batch(case, seed):
    vol, layout = _desc(case)
    slots = gc.pool_dims(vol, case["pool_mib"] << 20)
    cm = _cache(case, vol, layout, slots, 4096, seed, sync=not case["overlap"])
    tf = _tf(case, seed)
    tf_dev = torch.from_numpy(tf.reshape(-1)).cuda()
    rng = np.random.default_rng(seed)
    sizes = ((256, 256), (512, 512), (1024, 1024), (1920, 1080))
    ims = [_Image(case, _camera(rng, rng.uniform(0.5, 3.0)), *sizes[k % 4], tf, tf_dev) for k in range(case["views"])]
    _precision(case)
    batch = gc.Batch(cm, max_views=16, max_pixels=8 << 20, max_occupancy=0.5, reorder_window=8,
                     overlap_loads=case["overlap"])
    state = {"kind": "batch", "cm": cm, "images": ims, "batch": batch, "tf": tf_dev}
    run(state)  # the bricks of the views are resident from here on
    return state


def _prepare_mip(case, seed):
    vol, layout = _desc(dict(case, B=16))
    pyr, offs = _pyramid(case, vol, layout, seed)
    n0 = case["x"] * case["y"] * case["z"] * case["eb"]
    levels = [pyr[offs[l]: offs[l] + int(np.prod(list(layout.mip[l]))) * case["eb"]]
              for l in range(1, layout.nb_levels)]
    if case["float"]:
        levels = [v.view(torch.float32) for v in levels]
    return {"kind": "mip", "pyramid": pyr, "layout": layout, "offs": offs, "eb": case["eb"], "ch": case["ch"],
            "levels": levels, "n0": n0}


def _prepare_prep(case, seed):
    vol, layout = _desc(case)
    pyr, offs = _pyramid(case, vol, layout, seed)
    soffs, total, _ = gc.brick_store_offsets(layout, vol)
    store = torch.zeros(total, dtype=torch.uint8, device="cuda")
    nbig = [layout.nb_big_bricks[l][0] * layout.nb_big_bricks[l][1] * layout.nb_big_bricks[l][2]
            for l in range(layout.nb_levels)]
    flags = [torch.zeros(n, dtype=torch.uint8, device="cuda") for n in nbig]
    bins = [torch.zeros(n, dtype=torch.int64, device="cuda") for n in _bricks(layout)]
    return {"kind": "prep", "vol": vol, "layout": layout, "pyramid": pyr, "offs": offs, "store": store,
            "soffs": soffs, "nbig": nbig, "flags": flags, "bins": bins, "eb": case["eb"], "ch": case["ch"],
            # a threshold of 5 % of the range: the empty space around the blobs
            "threshold": 0.05 * (255.0 if case["eb"] // case["ch"] == 1 else 65535.0)}


def _prepare_miss(case, seed):
    vol, layout = _desc(case)
    mx = sum(layout.nb_bricks[l][0] for l in range(layout.nb_levels))
    my = max(layout.nb_bricks[l][1] for l in range(layout.nb_levels))
    mz = max(layout.nb_bricks[l][2] for l in range(layout.nb_levels))
    n = mx * my * mz
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    # stamps of earlier frames everywhere a ray has been, this frame's on the missing bricks
    req = torch.randint(0, 100, (n,), generator=gen, device="cuda", dtype=torch.int32)
    at = torch.randint(0, n - 1, (case["missing"],), generator=gen, device="cuda")
    req[at] = 100
    return {"kind": "miss", "req": req, "n": n, "layout": layout, "requests": case["requests"],
            "list": torch.zeros(case["requests"] * 4, dtype=torch.int32, device="cuda"),
            "total": torch.zeros(1, dtype=torch.int32, device="cuda")}


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


# ---------------------------------------------------------------------------

def _run_frame(s):
    im, cm = s["image"], s["cm"]
    im.restart()
    cm.render(im.view)
    cm.update()
    return im.outputs()


def _run_loop(s):
    cm = s["cm"]
    for im in s["images"]:
        im.restart()
        for _ in range(MAX_ITERATIONS):
            cm.render(im.view)
            if cm.update():
                break
    return [im.outputs() for im in s["images"]]


def _run_batch(s):
    batch, left = s["batch"], len(s["images"])
    for k, im in enumerate(s["images"]):
        batch.submit(im.view, k)
    for _ in range(MAX_TICKS):
        batch.tick()
        left -= len(batch.poll(64))
        if left <= 0:
            break
    return [im.rgba for im in s["images"]]


def _run_mip(s):
    gc.Mipmapper.process(s["pyramid"].data_ptr(), s["layout"], s["offs"], s["eb"], s["ch"])
    return s["levels"]


def _run_prep(s):
    vol, layout, pyr, store = s["vol"], s["layout"], s["pyramid"].data_ptr(), s["store"].data_ptr()
    gc.Mipmapper.process(pyr, layout, s["offs"], s["eb"], s["ch"])
    for l in range(layout.nb_levels):
        at = store + s["soffs"][l]
        gc.process_bricking(pyr + s["offs"][l], layout.initial[l], vol, layout.nb_big_bricks[l], at)
        gc.process_empty(at, s["nbig"][l], vol, s["threshold"], s["flags"][l].data_ptr())
        gc.brick_value_bins(vol, layout, l, at, s["bins"][l].data_ptr())
    return {"store": s["store"], "flags": s["flags"], "bins": s["bins"]}


def _run_miss(s):
    gc.miss_list_noalloc(s["req"].data_ptr(), s["n"], 100, s["layout"], s["requests"], s["list"].data_ptr(),
                         s["total"].data_ptr())
    return {"list": s["list"], "total": s["total"]}


def run(state):
    return globals()["_run_" + state["kind"]](state)


# ---------------------------------------------------------------------------

def _pixels(case):
    if case["kind"] == "frame":
        return [(case["W"] * case["H"], case["dist"])]
    if case["kind"] == "loop":
        n = case["views"]
        return [(case["W"] * case["H"], case["far"] + (case["near"] - case["far"]) * k / max(1, n - 1))
                for k in range(n)]
    sizes = (256 * 256, 512 * 512, 1024 * 1024, 1920 * 1080)
    return [(sizes[k % 4], 1.75) for k in range(case["views"])]


def work(case):
    """Ray casting: 44 bytes a pixel (RGBA out; t and colour state in and out)
    and the voxels of the level of detail that the rays through the box see,
    each read once, with about 60 operations a sample.  Preprocessing: the
    level-0 voxels read, levels, bricks, flags and bins written."""
    kind = case["kind"]
    if kind == "miss":
        _, layout = _desc(case)
        n = (sum(layout.nb_bricks[l][0] for l in range(layout.nb_levels)) *
             max(layout.nb_bricks[l][1] for l in range(layout.nb_levels)) *
             max(layout.nb_bricks[l][2] for l in range(layout.nb_levels)))
        return {"bytes": 4 * n + 16 * min(case["requests"], case["missing"]) + 4, "flops": 0}
    n0 = case["x"] * case["y"] * case["z"] * case["eb"]
    if kind in ("mip", "prep"):
        vol, layout = _desc(dict(case, B=case.get("B", 16), bb=case.get("bb", 1)))
        out = sum(layout.mip[l][0] * layout.mip[l][1] * layout.mip[l][2] for l in range(1, layout.nb_levels))
        if kind == "mip":
            return {"bytes": n0 + out * case["eb"], "flops": 8 * n0 // case["eb"] // 7}
        _, store, big = gc.brick_store_offsets(layout, vol)
        return {"bytes": n0 + out * case["eb"] + store + store // big + 8 * sum(_bricks(layout)),
                "flops": 8 * n0 // case["eb"] // 7}
    total_bytes = total_flops = 0
    for px, dist in _pixels(case):
        # share of the image that the box covers, and voxels along a ray at the level the pixel size selects
        cover = min(1.0, (FOCAL / (dist * DIAG)) ** 2)
        along = min(max(case["x"], case["y"], case["z"]), math.sqrt(px))
        rays = px * cover
        total_bytes += 44 * px + min(n0, int(rays * along * case["eb"] / 4))
        total_flops += int(rays * along * 60)
    return {"bytes": int(total_bytes), "flops": int(total_flops)}


# ---------------------------------------------------------------------------
# 64-bit values.  The ray caster as plain tensor arithmetic on whole levels.

def _levels64(case, layout, v):
    """Every level as (z, y, x, channel) float64 values with a border of zeros."""
    ch = case.get("ch", 1)
    cb = case["eb"] // ch
    a = v if cb == 1 else v.view(torch.int16)
    a = a.reshape(case["z"], case["y"], case["x"], ch).to(torch.int32)
    if cb == 2:
        a = a & 0xFFFF
    out = []
    for l in range(layout.nb_levels):
        if l:
            z, y, x = (n // 2 * 2 for n in a.shape[:3])
            a = a[:z, :y, :x].reshape(z // 2, 2, y // 2, 2, x // 2, 2, ch).sum(dim=(1, 3, 5)) // 8
        out.append(torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1, 1, 1)).double())
    return out


def _march64(case, layout, levels, tf, cam, W, H):
    f64 = torch.float64
    dev = levels[0].device
    m = torch.tensor(cam, dtype=torch.float32).double().reshape(3, 4).to(dev)
    dvr, ch = case.get("dvr", True), case.get("ch", 1)
    tstep, early = float(np.float32(TSTEP)), float(np.float32(0.99))
    focal = float(np.float32(FOCAL))
    py, px = torch.meshgrid(torch.arange(H, device=dev), torch.arange(W, device=dev), indexing="ij")
    px, py = px.reshape(-1).to(f64), py.reshape(-1).to(f64)
    qx, qy = torch.where(px + 1 > W, px - 1, px + 1), torch.where(py + 1 > H, py - 1, py + 1)

    def ray(x, y):
        d = torch.stack([(x + 0.5) / W * 2 - 1, (y + 0.5) / H * 2 - 1, torch.full_like(x, -focal)], -1)
        return (d / d.norm(dim=-1, keepdim=True)) @ m[:, :3].T

    def unit(v):
        return v / v.norm(dim=-1, keepdim=True)

    d, dx, dy = ray(px, py), ray(qx, py), ray(px, qy)
    left, up = unit(torch.linalg.cross(d, dy)), unit(torch.linalg.cross(d, dx))
    o = m[:, 3]
    a, b = (-1.0 - o) / d, (1.0 - o) / d
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    tnear, tfar = lo.amax(-1), hi.amin(-1)
    rays = torch.nonzero(tfar > tnear).reshape(-1)
    t_out = torch.zeros(W * H, dtype=f64, device=dev)
    s_out = torch.zeros(W * H, 4, dtype=f64, device=dev)
    d, dx, dy, left, up = d[rays], dx[rays], dy[rays], left[rays], up[rays]
    t, tfar = tnear[rays].clamp(min=0.0), tfar[rays]
    pos = o + d * t[:, None]
    ex, ey = ((d - dx) * left).sum(-1).abs() * tfar, ((d - dy) * up).sum(-1).abs() * tfar
    nl = layout.nb_levels
    dims = torch.tensor([list(layout.initial[l]) for l in range(nl)], dtype=f64, device=dev)
    inv = 2.0 / dims
    step = (2.0 / dims.amin(-1)) / 2.0
    sl = torch.stack([(left * inv[l]).norm(dim=-1) for l in range(nl)], -1)
    su = torch.stack([(up * inv[l]).norm(dim=-1) for l in range(nl)], -1)
    flat = torch.cat([v.reshape(-1, ch) for v in levels])
    base = torch.tensor([0] + [v[..., 0].numel() for v in levels], device=dev).cumsum(0)[:-1]
    sx = torch.tensor([v.shape[2] for v in levels], device=dev)
    sxy = torch.tensor([v.shape[2] * v.shape[1] for v in levels], device=dev)
    vmax = 255.0 if case["eb"] // ch == 1 else 65535.0
    tab = torch.from_numpy(tf).to(dev).double()
    lod = torch.zeros(rays.numel(), dtype=torch.long, device=dev)
    col = torch.zeros(rays.numel(), 4, dtype=f64, device=dev)

    def axis(s, n):
        x = s * n - 0.5
        i = x.floor()
        return i.long().clamp(0, n - 1), (i.long() + 1).clamp(0, n - 1), (x - i)[:, None]

    def classify(s):
        i0, i1, ax = axis(s[:, 0], tab.shape[-2])
        if ch == 1:
            return tab[i0] + (tab[i1] - tab[i0]) * ax
        j0, j1, ay = axis(s[:, 1], tab.shape[0])
        r0 = tab[j0, i0] + (tab[j0, i1] - tab[j0, i0]) * ax
        r1 = tab[j1, i0] + (tab[j1, i1] - tab[j1, i0]) * ax
        return r0 + (r1 - r0) * ay

    while rays.numel():
        live = (t < tfar) & ((col[:, 3] < early) if dvr else torch.ones_like(t, dtype=torch.bool))
        if not bool(live.all()):
            gone = ~live
            t_out[rays[gone]] = t[gone]
            s_out[rays[gone]] = col[gone]
            rays, t, tfar, pos, d, ex, ey, sl, su, lod, col = (
                q[live] for q in (rays, t, tfar, pos, d, ex, ey, sl, su, lod, col))
            if not rays.numel():
                break
        al = t / tfar
        for _ in range(nl - 1):
            nxt = (lod + 1).clamp(max=nl - 1)[:, None]
            keep = (sl.gather(1, nxt)[:, 0] >= ex * al) | (su.gather(1, nxt)[:, 0] >= ey * al) | (lod + 1 >= nl)
            if bool(keep.all()):
                break
            lod = torch.where(keep, lod, lod + 1)
        np_ = pos * 0.495 + 0.495
        np_ = torch.stack([np_[:, 0], np_[:, 1], 1.0 - np_[:, 2]], -1).clamp(0.0, 0.99)
        f = np_ * dims[lod]
        if case.get("tri"):
            i = (f - 0.5).floor()
            w = f - 0.5 - i
        else:
            i = f.floor() - 1
            w = torch.full_like(f, 0.5)
        i = i.long() + 1
        at = base[lod] + i[:, 2] * sxy[lod] + i[:, 1] * sx[lod] + i[:, 0]
        s = 0
        for k in range(8):
            c = [(w if (k >> q) & 1 else 1 - w)[:, q] for q in range(3)]
            s = s + flat[at + (k & 1) + ((k >> 1) & 1) * sx[lod] + (k >> 2) * sxy[lod]] * (c[0] * c[1] * c[2])[:, None]
        s = s / vmax
        h = step[lod]
        if dvr:
            q = classify(s)
            q[:, 3] = 1.0 - (1.0 - q[:, 3]) ** (h / tstep)
            r = torch.where(q[:, 3] > 0.001, 1.0 - col[:, 3], torch.zeros_like(h))
            col = torch.cat([q[:, :3] * q[:, 3:], q[:, 3:]], -1) * r[:, None] + col
        else:
            col = torch.cat([torch.maximum(col[:, :1], s[:, :1]), col[:, 1:]], -1)
        t = t + h
        pos = pos + d * h[:, None]
    return t_out, s_out.reshape(-1)


def exact(case, seed):
    if case["kind"] == "mip" and case["float"]:
        _, layout = _desc(dict(case, B=16))
        a = _volume(case, seed).view(torch.float32).reshape(case["z"], case["y"], case["x"])
        out = []
        for _ in range(1, layout.nb_levels):
            z, y, x = (n // 2 * 2 for n in a.shape)
            a = a[:z, :y, :x].double().reshape(z // 2, 2, y // 2, 2, x // 2, 2).mean(dim=(1, 3, 5))
            out.append(a.reshape(-1))
        return out
    # preprocessing, miss lists and batched images are whole numbers; the rays
    # of a loop resume where they paused and a view whose bricks do not fit the
    # pool ends unfinished, so its values follow from what was resident
    if case["kind"] != "frame":
        return None
    vol, layout = _desc(case)
    levels = _levels64(case, layout, _volume(case, seed))
    tf = _tf(case, seed)
    rng = np.random.default_rng(seed)
    t, s = _march64(case, layout, levels, tf, _camera(rng, case["dist"]), case["W"], case["H"])
    return {"rgba": None, "t": t, "state": s}
