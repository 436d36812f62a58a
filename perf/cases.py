"""The work a user of this framework has it do, as timed cases.

Every case goes through the public entry points (``barney_b200.VolumeRenderer``,
``Context.render_batch``, ``Server``: thin mirrors of the C API) the way an
application does: volumes, transfer functions and frame buffers are set up once
(``prepare``), and one pass (``run``) is what the application repeats.

Kinds of case
  edit     the user drags the transfer function: new table, majorants mapped
           again, accumulation restarted, one preview frame read back
  frame    camera moved, accumulation restarted, a frame of `spp` paths per
           pixel, colour read back; `form` is the precision form: "plain" (the
           drop-in default) or "compensated" (majorants rounded up and
           compensated sums, for 16- and 8-bit storage)
  paths    the same frame in the multi-scatter build (volume bounces)
  surface  the same frame with a matte isosurface inside the volume
  load     a volume that is already in device memory is opened: field, volume,
           macrocell and majorant build, first preview frame
  batch    frames of many small volumes in one launch
  serve    a burst of requests through the continuous-batching server

A Monte-Carlo frame is a sum over paths whose every decision (which collision,
which light) is taken by an integer random stream against binary32 quantities, so
there is no 64-bit value of the same frame to compare with; the kernels are bit-
reproducible instead, and their frames are compared exactly.  Macrocell ranges and
majorants do have one (`exact`).  The fast-math form is left out for the same reason:
a path's random streams are seeded by the bits of its collision distance, so two
correct fast-math kernels share no path, only expectations.
"""
import math
import random

import torch

import barney_b200 as bn
from barney_b200 import synth

EDGE_MIN, EDGE_MAX = 48, 1024   # volume edges of the frame cases
PIXELS_MIN, PIXELS_MAX = 160 * 120, 1920 * 1080


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(name, kind, dims, dtype, field, width, height, spp, **kw):
    c = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "dtype": dtype, "field": field,
         "width": width, "height": height, "spp": spp, "form": "plain", "look": "scatter", "azimuth": 45.0,
         "elevation": 28.0, "color": "float4"}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # interactive transfer-function editing on a small 8-bit scan
        _case("edit_128_u8", "edit", (128, 128, 128), "u8", "blobs", 320, 240, 1, look="ambient", color="rgba8"),
        # the small workload: 64^3 blobs, 256 x 256, 16 paths per pixel
        _case("small_64_f32", "frame", (64, 64, 64), "f32", "blobs", 256, 256, 16, look="ambient"),
        # interactive orbit: one preview path per pixel on a ragged 16-bit volume
        _case("orbit_ragged_u16", "frame", (251, 187, 313), "u16", "noise", 1279, 719, 1, color="rgba8",
              azimuth=200.0, elevation=-10.0),
        # the main workload: 512^3 noise, 1080p, 64 paths per pixel, one light + ambient
        _case("full_512_f32", "frame", (512, 512, 512), "f32", "noise", 1920, 1080, 64),
        # the large one in 16-bit storage, compensated sums, anisotropic scattering
        _case("large_1024_f16", "frame", (1024, 1024, 1024), "f16", "noise", 1920, 1080, 16, form="compensated",
              anisotropy=0.4),
        # a square frame of an 8-bit scan, as a server renders it
        _case("square_512_u8", "frame", (512, 512, 512), "u8", "noise", 1024, 1024, 4, form="compensated",
              color="rgba8", azimuth=120.0, elevation=50.0),
        # multi-scatter build: up to 8 volume bounces
        _case("paths_512_f32", "paths", (512, 512, 512), "f32", "noise", 1280, 720, 16, bounces=8),
        # an isosurface inside the volume
        _case("surface_256_f32", "surface", (256, 256, 256), "f32", "noise", 1280, 720, 8, iso=0.5),
        # opening a 512^3 volume that a simulation left in device memory
        _case("load_512_f32", "load", (512, 512, 512), "f32", "noise", 640, 360, 1, color="rgba8"),
        # the batching workload: 64 mixed jobs (edges 32-256, sides 128-1024, 1-32 paths)
        _case("batch_64_mixed", "batch", (256, 256, 256), "mixed", "mixed", 1024, 1024, 32, jobs=64, mix=0),
        # the serving workload: a burst of requests over resident volumes
        _case("serve_64_mixed", "serve", (256, 256, 256), "f16", "mixed", 1024, 1024, 16, jobs=64, mix=7, volumes=6,
              form="compensated", color="rgba8"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["edit", "frame", "frame", "frame", "paths", "surface", "load", "batch", "serve"])
    pixels = _log_int(rng, PIXELS_MIN, PIXELS_MAX)
    aspect = rng.choice([1.0, 4 / 3, 16 / 9])
    height = max(16, int(math.sqrt(pixels / aspect)))
    width = max(16, pixels // height)
    edge = _log_int(rng, EDGE_MIN, EDGE_MAX)
    dims = (edge, edge, edge)
    if rng.random() < 0.5:
        dims = tuple(max(9, int(edge * rng.uniform(0.4, 1.0))) for _ in range(3))
    dtype = rng.choice(["f32", "f32", "f16", "bf16", "u8", "u16"])
    field = rng.choice(["noise", "noise", "blobs"])
    kw = {"look": rng.choice(["scatter", "scatter", "ambient"]), "azimuth": round(rng.uniform(0.0, 360.0), 1),
          "elevation": round(rng.uniform(-30.0, 60.0), 1), "color": rng.choice(["float4", "rgba8"])}
    spp = rng.choice([1, 2, 4, 7, 16, 32, 64])
    if kind == "frame":
        kw["form"] = "plain" if dtype == "f32" else rng.choice(["plain", "compensated"])
        kw["anisotropy"] = rng.choice([0.0, 0.0, 0.4, -0.3])
    elif kind == "paths":
        spp, kw["bounces"], kw["look"] = min(spp, 8), rng.choice([1, 2, 8]), "scatter"
    elif kind == "surface":
        spp, kw["iso"] = min(spp, 4), rng.choice([0.4, 0.5, 0.6])
        dims = tuple(min(d, 320) for d in dims)
    elif kind in ("edit", "load"):
        spp = 1
    elif kind == "batch":
        kw.update(jobs=rng.randint(2, 64), mix=rng.randint(1, 10**6))
        dims, width, height, spp, dtype, field = (256, 256, 256), 1024, 1024, 32, "mixed", "mixed"
    else:
        kw.update(jobs=rng.randint(4, 64), mix=rng.randint(1, 10**6), volumes=rng.randint(2, 8), color="rgba8",
                  form=rng.choice(["plain", "compensated"]))
        dims, width, height, spp, dtype, field = (256, 256, 256), 1024, 1024, 16, rng.choice(["f32", "f16", "u8"]), "mixed"
    return _case(None, kind, dims, dtype, field, width, height, spp, **kw)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _axis(n, device):
    return torch.linspace(0.0, 1.0, n, dtype=torch.float32, device=device)


def _lerp_axis(lattice, coord, dim):
    """The lattice along `dim` at lattice coordinates `coord`, quintic fade."""
    i = coord.floor().clamp(max=lattice.shape[dim] - 2).long()
    t = coord - i
    t = t * t * t * (t * (t * 6.0 - 15.0) + 10.0)
    shape = [1, 1, 1]
    shape[dim] = -1
    t = t.view(shape)
    a, b = lattice.index_select(dim, i), lattice.index_select(dim, i + 1)
    return a.add_((b - a).mul_(t))


def _noise(nx, ny, nz, seed):
    """6-octave value noise in [0, 1] (base frequency 4, lacunarity 2, gain 0.5)."""
    gen = torch.Generator().manual_seed(seed)
    out = torch.zeros((nz, ny, nx), dtype=torch.float32, device="cuda")
    for k in range(6):
        f = 4 << k
        lat = torch.rand((f + 1, f + 1, f + 1), generator=gen).cuda()
        part = _lerp_axis(lat, _axis(nz, "cuda") * f, 0)
        part = _lerp_axis(part, _axis(ny, "cuda") * f, 1)
        x = _axis(nx, "cuda") * f
        for z0 in range(0, nz, 64):  # slabs: bounded temporary memory
            out[z0:z0 + 64].add_(_lerp_axis(part[z0:z0 + 64], x, 2), alpha=0.5 ** k / 1.96875)
    return out.clamp_(0.0, 1.0)


def _blobs(nx, ny, nz, seed):
    """Sum of 8 isotropic Gaussians, as synth.blobs."""
    centres, sigma, amp = synth.blob_params(seed)
    out = torch.zeros((nz, ny, nx), dtype=torch.float32, device="cuda")
    for c, s, a in zip(centres, sigma, amp):
        gx, gy, gz = (torch.exp(-(_axis(n, "cuda") - float(p)) ** 2 / float(2 * s * s)) for n, p in
                      ((nx, c[0]), (ny, c[1]), (nz, c[2])))
        out.addcmul_((gz * float(a)).view(-1, 1, 1) * gy.view(1, -1, 1), gx.view(1, 1, -1))
    return out


def _stored(vol, dtype):
    if dtype == "u8":
        return vol.clamp(0.0, 1.0).mul_(255.0).round_().to(torch.uint8)
    if dtype == "u16":
        return vol.clamp(0.0, 1.0).mul_(65535.0).round_().to(torch.int32).to(torch.int16)
    if dtype == "f16":
        return vol.half().view(torch.int16)
    if dtype == "bf16":
        return vol.bfloat16().view(torch.int16)
    return vol


def _volume(field, nx, ny, nz, dtype, seed):
    vox = _stored((_blobs if field == "blobs" else _noise)(nx, ny, nz, seed), dtype)
    torch.cuda.synchronize()  # the library copies it on its own stream
    return vox


def _camera(case):
    az, el = math.radians(case["azimuth"]), math.radians(case["elevation"])
    r = 2.345  # the distance of the workloads' camera (2, 1.5, 2) from the cube's centre
    return synth.look_at((0.5 + r * math.cos(el) * math.cos(az), 0.5 + r * math.sin(el),
                          0.5 + r * math.cos(el) * math.sin(az)))


def _scene(case, voxels):
    kw = {"spp": case["spp"]}
    if case["look"] == "ambient":  # linear ramp, ambient 1, the default build
        tf, kw["ambient"] = synth.tf_linear_ramp(128), 1.0
    else:  # knot TF, directional light + ambient, HG phase
        tf = synth.tf_knots(256, 1)
        kw.update(ambient=0.25, dir_lights=synth.CONFIG2_LIGHTS, phase="hg", anisotropy=case.get("anisotropy", 0.0),
                  scattering_albedo=0.8)
    if case["form"] != "plain":
        kw.update(majorant_round_up=True, compensated_accum=True)
    if case["kind"] == "paths":
        kw["max_volume_bounces"] = case["bounces"]
    if case["kind"] == "surface":
        kw["iso"] = {"value": case["iso"], "color": (0.9, 0.5, 0.2)}
    return synth.scene(voxels, case["dtype"], case["width"], case["height"], tf, 50.0, _camera(case), **kw)


def _jobs(case, seed):
    """The batching workload's jobs: edge log-uniform in [32, 256], blobs or
    noise, mixed storage, side log-uniform in [128, 1024], spp {1, 4, 16, 32}.
    The mix (sizes, types) is the case's; the fields are the seed's."""
    rng = random.Random(case["mix"])
    out = []
    for i in range(case["jobs"]):
        edge, side = _log_int(rng, 32, 256), _log_int(rng, 128, 1024)
        field = rng.choice(["blobs", "noise"])
        dtype = rng.choice(["u8", "f16", "f32"])
        sub = _case(None, "frame", (edge, edge, edge), dtype, field, side, side, rng.choice([1, 4, 16, 32]),
                    look="ambient" if field == "blobs" else "scatter", azimuth=rng.uniform(0.0, 360.0),
                    elevation=rng.uniform(-30.0, 60.0), color="rgba8")
        out.append((sub, seed * 1000 + i))
    return out


def _requests(case):
    """The serving workload's requests: (volume, side, spp, camera)."""
    rng = random.Random(case["mix"])
    vols = []
    for v in range(case["volumes"]):
        edge = _log_int(rng, 128, 320)
        field = rng.choice(["blobs", "noise"])
        vols.append(_case(None, "frame", (edge, edge, edge), case["dtype"], field, 16, 16, 1,
                          look="ambient" if field == "blobs" else "scatter", form=case["form"], color="rgba8"))
    reqs = []
    for _ in range(case["jobs"]):
        cam = dict(case, azimuth=rng.uniform(0.0, 360.0), elevation=rng.uniform(-30.0, 60.0))
        reqs.append((rng.randrange(case["volumes"]), rng.choice([256, 512, 1024]), rng.choice([1, 4, 16]),
                     _camera(cam)))
    return vols, reqs


def _frame_buffer(height, width, color):
    """Pinned host memory for a frame, as an application reads into."""
    if color == "float4":
        return torch.empty((height, width, 4), dtype=torch.float32, pin_memory=True)
    return torch.empty((height, width), dtype=torch.int32, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind}
    if kind == "batch":
        st["ctx"] = bn.Context()
        st["renderers"] = [bn.VolumeRenderer(_scene(c, _volume(c["field"], c["nx"], c["ny"], c["nz"], c["dtype"], s)),
                                             color_format=c["color"], context=st["ctx"])
                           for c, s in _jobs(case, seed)]
        st["out"] = [_frame_buffer(r.height, r.width, "rgba8") for r in st["renderers"]]
        return st
    if kind == "serve":
        vols, reqs = _requests(case)
        st["ctx"] = bn.Context()
        st["volumes"] = [bn.VolumeRenderer(_scene(c, _volume(c["field"], c["nx"], c["ny"], c["nz"], c["dtype"],
                                                             seed * 1000 + i)), context=st["ctx"])
                         for i, c in enumerate(vols)]
        st["server"] = bn.Server(st["ctx"], hbm_budget_bytes=16 << 30, slice_waves=16, slice_pixel_waves=64 << 20)
        st["server"].reserve(2 << 30)
        st["requests"] = reqs
        st["out"] = [_frame_buffer(side, side, "rgba8") for _, side, _, _ in reqs]
        return st
    voxels = _volume(case["field"], case["nx"], case["ny"], case["nz"], case["dtype"], seed)
    st["scene"] = _scene(case, voxels)
    st["out"] = _frame_buffer(case["height"], case["width"], case["color"])
    if kind == "load":
        st["ctx"] = bn.Context()
    else:
        st["renderer"] = bn.VolumeRenderer(st["scene"], color_format=case["color"])
    return st


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "batch":
        for r in state["renderers"]:
            r.accum_reset()
        state["ctx"].render_batch(state["renderers"])
        for r, o in zip(state["renderers"], state["out"]):
            r.read(o)
        return state["out"]
    if kind == "serve":
        ids = [state["server"].submit(state["volumes"][v], cam, side, side, spp)
               for v, side, spp, cam in state["requests"]]
        for i, o in zip(ids, state["out"]):
            state["server"].wait(i, o)
        return state["out"]
    if kind == "load":
        r = bn.VolumeRenderer(state["scene"], color_format=case["color"], context=state["ctx"])
        ranges, majorants = r.macrocells()
        r.render()
        r.read(state["out"])
        r.close()
        return [ranges, majorants, state["out"]]
    r = state["renderer"]
    if kind == "edit":
        d = state["scene"]
        r.set_transfer_function(d["tf"], d["domain"], d["density"])
    else:
        r.set_camera(state["scene"]["camera"])
    r.accum_reset()
    r.render()
    r.read(state["out"])
    return state["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
_VOXEL_BYTES = {"f32": 4, "f16": 2, "bf16": 2, "u16": 2, "u8": 1}
_COLOR_BYTES = {"float4": 16, "rgba8": 4}
# Arithmetic of the estimator per path that enters the volume: ray generation and
# its random numbers (~80), two box tests and DDA set-ups (~2 x 70), about 10
# macrocell steps (~10 each), two Woodcock steps with a trilinear sample and a TF
# lookup (~2 x 70), light sampling, phase function and accumulation (~120).
_FLOPS_PER_PATH = 580
_FLOPS_PER_BOUNCE = 300     # a further generation: scatter, its ray and shadow ray
_FLOPS_PER_SURFACE = 1500   # eleven samples in each candidate macrocell of three rays


def _frame_work(c):
    paths = c["width"] * c["height"] * c["spp"] * min(1.0, 0.43 * c["height"] / c["width"])  # rays that meet the cube
    per = _FLOPS_PER_PATH + (_FLOPS_PER_BOUNCE * c["bounces"] if c["kind"] == "paths" else 0)
    per += _FLOPS_PER_SURFACE if c["kind"] == "surface" else 0
    voxels = c["nx"] * c["ny"] * c["nz"]
    # the volume is opaque: rays read a shell of it, at most 16 voxels a path
    touched = min(0.25 * voxels, 16.0 * paths)
    pixels = c["width"] * c["height"]
    return touched * _VOXEL_BYTES[c["dtype"]] + pixels * (16 + _COLOR_BYTES[c["color"]]), paths * per


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_frame_work(c) for c, _ in _jobs(case, 0)]
    elif kind == "serve":
        vols, reqs = _requests(case)
        parts = [_frame_work(dict(vols[v], width=side, height=side, spp=spp)) for v, side, spp, _ in reqs]
    else:
        parts = [_frame_work(case)]
    total, flops = sum(p[0] for p in parts), sum(p[1] for p in parts)
    if kind == "load":  # the library's own copy of the voxels (read + write), from which the macrocells are built
        total += 2.0 * case["nx"] * case["ny"] * case["nz"] * _VOXEL_BYTES[case["dtype"]]
    return {"bytes": float(total), "flops": float(flops)}


def tolerance(case):
    """Every form here is bit-reproducible: the kernels evaluate each binary32
    expression as the reference source writes it, and sum in its order."""
    return "exact"


# ---------------------------------------------------------------------------
# 64-bit values where an output has one
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] != "load":
        return None
    vox = _volume(case["field"], case["nx"], case["ny"], case["nz"], case["dtype"], seed)
    if case["dtype"] == "u8":
        v = vox.double() / 255.0
    elif case["dtype"] == "u16":
        v = (vox.int() & 0xffff).double() / 65535.0
    elif case["dtype"] == "f16":
        v = vox.view(torch.float16).double()
    elif case["dtype"] == "bf16":
        v = vox.view(torch.bfloat16).double()
    else:
        v = vox.double()
    v = v[None, None]
    # macrocell i covers scalars 8 i .. 8 i + 8 of each axis
    pad = [p for n in reversed(v.shape[2:]) for p in (0, 8 * math.ceil((n - 1) / 8) + 1 - n)]
    hi = torch.nn.functional.max_pool3d(torch.nn.functional.pad(v, pad, value=-math.inf), 9, 8)[0, 0]
    lo = -torch.nn.functional.max_pool3d(torch.nn.functional.pad(-v, pad, value=-math.inf), 9, 8)[0, 0]
    tf = torch.tensor(_scene(case, vox)["tf"][:, 3], dtype=torch.float64, device="cuda")
    n = tf.numel()
    best = torch.stack([torch.cat([tf.new_full((i,), -math.inf), tf[i:].cummax(0).values]) for i in range(n)])

    def at(x):
        x = x.clamp(0.0, 1.0) * (n - 1)
        i = x.long().clamp(0, n - 2)
        return i, torch.lerp(tf[i], tf[i + 1], x - i)

    i_lo, w_lo = at(lo)
    i_hi, w_hi = at(hi)
    inner = torch.where(i_lo < i_hi, best[(i_lo + 1).clamp(max=n - 1), i_hi], torch.zeros_like(w_lo))
    maj = torch.maximum(torch.maximum(w_lo, w_hi), inner) * 50.0
    return [torch.stack([lo, hi], dim=-1).cpu().numpy(), maj.cpu().numpy(), None]
