"""What is timed of this framework: its calls as a user's program makes them, over their real range.

A case is a dict of plain values; `call` names the entry point it goes through:

  render   vt_render: one frame of hit records into device memory
  rays     vt_trace_rays: a buffer of rays on the device
  views    vt_batch_run: many cameras over several grids, one graph replay
  path     vt_path_trace: a path-traced frame (float radiance)
  scene    vt_grid_create_u8_device, then the first frame of the new grid, then vt_grid_destroy
  texture  vt_grid_create from host memory, a preview frame, vt_grid_destroy
  page     vt_grid_update: a chunk paged in, a frame, and the chunk paged out again
  world    start/end_update_instances, render_tick and the read-back of its frame
  serve    vt_serve_submit and vt_serve_poll: a burst of requests to a running service

Scenes are the three kinds of this repository's workloads (heightfield terrain, scattered boxes
and spheres, noise caves), made on the GPU from the seed.
"""
import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

import vtrace_gb300 as vt
from vtrace_gb300 import workloads


def listed():
    return [
        # the smallest frame: a thumbnail of a model-sized grid, where launch and latency count
        {"name": "render_thumb", "call": "render", "scene": "terrain", "nx": 64, "ny": 64, "nz": 64,
         "rgba": False, "width": 96, "height": 64, "light": True, "shadows": False},
        # an ordinary frame of a heightfield world, lit without shadows
        {"name": "render_terrain", "call": "render", "scene": "terrain", "nx": 256, "ny": 256, "nz": 256,
         "rgba": False, "width": 640, "height": 480, "light": True, "shadows": False},
        # the large frame: full HD over a big scattered scene, one shadow ray per lit hit
        {"name": "render_hd_shadow", "call": "render", "scene": "shapes", "nx": 1024, "ny": 1024, "nz": 1024,
         "rgba": False, "width": 1920, "height": 1080, "light": True, "shadows": True},
        # picking and line-of-sight queries: a few thousand rays, axis-parallel ones among them, in
        # a ragged RGBA8 grid
        {"name": "rays_few", "call": "rays", "scene": "cave", "nx": 61, "ny": 90, "nz": 37,
         "rgba": True, "rays": 4099},
        # sensor or lighting simulation: millions of incoherent rays inside a cave
        {"name": "rays_cave", "call": "rays", "scene": "cave", "nx": 512, "ny": 512, "nz": 512,
         "rgba": False, "rays": 1 << 24},
        # data generation: many cameras of uneven size and sample count over several scenes
        {"name": "views_batch", "call": "views", "scenes": 8, "views": 16, "low": 128, "high": 512,
         "min_px": 320 * 240, "max_px": 1920 * 1080, "max_spp": 4},
        # an offline-quality frame: jittered samples, bounces and a sun
        {"name": "path_hd", "call": "path", "scene": "shapes", "nx": 1024, "ny": 1024, "nz": 1024,
         "rgba": False, "width": 1920, "height": 1080, "spp": 2, "bounces": 3},
        # loading a large scene that is already on the device and showing its first frame
        {"name": "scene_load", "call": "scene", "scene": "shapes", "nx": 1024, "ny": 1024, "nz": 1024,
         "width": 640, "height": 480},
        # loading one chunk texture of the streaming world from host memory, with a preview
        {"name": "texture_chunk", "call": "texture", "scene": "terrain", "nx": 16, "ny": 16, "nz": 16,
         "rgba": True, "z_fastest": False, "width": 160, "height": 120},
        # streaming a world: a 16^3 chunk written into the resident grid, drawn, taken out again
        {"name": "page_chunk", "call": "page", "scene": "shapes", "nx": 1024, "ny": 1024, "nz": 1024,
         "chunk": 16, "z_fastest": True, "width": 640, "height": 480},
        # one frame of the chunked world through the reference's C entry points
        {"name": "world_tick", "call": "world", "reach": 6},
        # a render service under a burst of requests of mixed sizes
        {"name": "serve_burst", "call": "serve", "scenes": 4, "requests": 24, "low": 128, "high": 512,
         "min_px": 320 * 240, "max_px": 1280 * 720, "max_spp": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["render", "render", "rays", "rays", "views", "path", "scene", "texture",
                       "page", "world", "serve"])
    case = {"call": call}
    if call in ("render", "rays", "path"):
        n = _log(rng, 32, 1024)
        side = [max(8, int(n * rng.uniform(0.5, 1.0))) for _ in range(3)]
        if rng.random() < 0.4:
            side = [n, n, n]
        case.update(scene=rng.choice(["terrain", "shapes", "cave"] if n <= 512 else ["terrain", "shapes"]),
                    nx=side[0], ny=side[1], nz=side[2], rgba=n <= 256 and rng.random() < 0.3)
    if call in ("render", "path"):
        h = _log(rng, 48, 1080 if call == "render" else 720)
        case.update(width=int(h * rng.choice([1.0, 4.0 / 3.0, 16.0 / 9.0])), height=h)
    if call == "render":
        case.update(light=rng.random() < 0.85, shadows=rng.random() < 0.6)
    elif call == "rays":
        case.update(rays=_log(rng, 1000, 1 << 24))
    elif call == "path":
        case.update(spp=rng.randint(1, 4), bounces=rng.randint(0, 3))
    elif call == "views":
        low = rng.randrange(64, 256, 8)
        case.update(scenes=rng.randint(1, 6), views=_log(rng, 2, 24), low=low, high=low + rng.randrange(0, 257, 8),
                    min_px=160 * 120, max_px=_log(rng, 320 * 240, 1280 * 720), max_spp=rng.randint(1, 4))
    elif call == "scene":
        case.update(scene=rng.choice(["terrain", "shapes"]), nx=_log(rng, 72, 1024), ny=_log(rng, 72, 1024),
                    nz=_log(rng, 72, 1024), width=_log(rng, 160, 960), height=_log(rng, 120, 540))
    elif call == "texture":
        case.update(scene=rng.choice(["terrain", "shapes"]), nx=_log(rng, 8, 160), ny=_log(rng, 8, 160),
                    nz=_log(rng, 8, 160), rgba=rng.random() < 0.7, z_fastest=rng.random() < 0.5, width=160, height=120)
    elif call == "page":
        n = _log(rng, 96, 1024)
        case.update(scene=rng.choice(["terrain", "shapes"]), nx=n, ny=max(64, int(n * rng.uniform(0.5, 1.0))), nz=n,
                    chunk=rng.choice([5, 8, 16, 16, 32, 61]), z_fastest=rng.random() < 0.5, width=640, height=480)
    elif call == "world":
        case.update(reach=rng.randint(2, 6))
    elif call == "serve":
        low = rng.randrange(64, 256, 8)
        case.update(scenes=rng.randint(1, 4), requests=_log(rng, 1, 32), low=low, high=low + rng.randrange(0, 257, 8),
                    min_px=160 * 120, max_px=_log(rng, 320 * 240, 1280 * 720), max_spp=rng.randint(1, 4))
    return case


# ---------------------------------------------------------------- content

def _ball(r, cache):
    """Mask of the voxels whose centres lie within r of a voxel's centre."""
    if r not in cache:
        a = torch.arange(-r, r + 1, device="cuda")
        cache[r] = (a[:, None, None] ** 2 + a[None, :, None] ** 2 + a[None, None, :] ** 2) <= r * r
    return cache[r]


def _shapes(nx, ny, nz, g):
    n = (nx * ny * nz) ** (1.0 / 3.0)
    count, rmin, rmax = max(50, int(n * n / 100.0)), 2.0, max(4.0, n / 25.0)
    vox = torch.zeros((nz, ny, nx), dtype=torch.uint8, device="cuda")
    u = torch.rand((count, 10), generator=g, device="cuda").cpu().numpy().astype(np.float64)
    cache = {}
    for s in u:
        r = rmin + (rmax - rmin) * s[0] * s[1] * s[2]  # many small shapes, few large ones
        sphere = s[3] < 0.5
        half = [int(round(r))] * 3 if sphere else [max(1, int(round(r * (0.5 + 0.5 * k)))) for k in s[7:10]]
        c = [int(s[4] * nz), int(s[5] * ny), int(s[6] * nx)]
        lo = [max(0, c[a] - half[a]) for a in range(3)]
        hi = [min(vox.shape[a], c[a] + half[a] + 1) for a in range(3)]
        part = vox[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]]
        value = 1 + int(s[9] * 1e6) % 255
        if sphere:
            cut = tuple(slice(lo[a] - c[a] + half[a], hi[a] - c[a] + half[a]) for a in range(3))
            part.masked_fill_(_ball(half[0], cache)[cut], value)
        else:
            part.fill_(value)
    return vox


def _colours(shape, g):
    return torch.randint(1, 256, shape, generator=g, device="cuda", dtype=torch.uint8)


def _terrain(nx, ny, nz, g):
    height = torch.full((nz, nx), 0.3, device="cuda")
    for octave in range(5):  # a few hills across the grid, each octave half as high
        k = 5 << octave
        noise = torch.rand((1, 1, k, k), generator=g, device="cuda") - 0.5
        height += 0.45 * 0.5 ** octave * F.interpolate(noise, size=(nz, nx), mode="bicubic", align_corners=True)[0, 0]
    level = (height.clamp(0.0, 1.0) * ny).to(torch.int32)
    solid = torch.arange(ny, device="cuda")[None, :, None] < level[:, None, :]
    return _colours((nz, ny, nx), g) * solid


def _cave(nx, ny, nz, g):
    field = torch.zeros((nz, ny, nx), device="cuda")
    for k, amplitude in ((8, 1.0), (14, 0.5)):
        noise = torch.randn((1, 1, k, k, k), generator=g, device="cuda")
        field += amplitude * F.interpolate(noise, size=(nz, ny, nx), mode="trilinear", align_corners=True)[0, 0]
    step = max(1, field.numel() // 100000)
    some = field.reshape(-1)[::step]
    level = some.kthvalue(max(1, int(0.55 * some.numel()))).values
    return _colours((nz, ny, nx), g) * (field > level)


def _scene(kind, nx, ny, nz, seed):
    """A u8 grid [z, y, x] on the device and its palette."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    vox = {"shapes": _shapes, "terrain": _terrain, "cave": _cave}[kind](nx, ny, nz, g)
    return vox, vt.gen_palette(seed & 0x7FFFFFFF)


def _texels(vox, palette):
    """The same scene as RGBA8 texels [z, y, x] in host memory."""
    return palette[vox.cpu().numpy()]


def _grid(case, seed):
    vox, palette = _scene(case["scene"], case["nx"], case["ny"], case["nz"], seed)
    if case.get("rgba"):
        return vt.Grid.from_rgba8(_texels(vox, palette)), vox, palette
    torch.cuda.synchronize()
    return vt.Grid.from_u8_device(vox, (case["nx"], case["ny"], case["nz"]), palette), vox, palette


def _camera(kind, dims, seed, width, height):
    rng = np.random.default_rng(seed)
    n = max(dims)
    if kind == "cave":  # seen from inside
        eye = [float(d * rng.uniform(0.3, 0.7)) for d in dims]
        target = [float(d * rng.uniform(0.0, 1.0)) + 0.25 for d in dims]
    else:
        eye, target = workloads.seeded_pose(dims, seed, (1.1 if kind == "terrain" else 0.9) * n)
    return vt.camera_look_at(eye, target, (0.0, 1.0, 0.0), 60.0, width, height)


def _records(count):
    return torch.empty((count, 4), dtype=torch.int32, device="cuda")


class _Held:
    """The library objects of one state, closed when the state goes, as a user's program closes
    them at its end."""

    def __init__(self, *objects):
        self.objects = objects

    def __del__(self):
        torch.cuda.synchronize()
        for x in self.objects:
            x.stop() if isinstance(x, vt.Service) else x.destroy()


def _views(case, seed):
    """Scenes (kind, size, voxels, palette) and view specs of a batch or of a burst of requests."""
    scenes, specs = [], []
    for i in range(case["scenes"]):
        n = case["low"] // 8 * 8 + (i * 5 + 1) % 8 * (case["high"] - case["low"]) // 7 // 8 * 8
        kind = ("terrain", "shapes", "cave")[i % 3]
        scenes.append((kind, n) + _scene(kind, n, n, n, seed * 16 + i))
    for v in range(case.get("views") or case["requests"]):
        # areas spread evenly over the range by their logarithm
        count = case.get("views") or case["requests"]
        area = case["min_px"] * (case["max_px"] / case["min_px"]) ** ((v + 0.5) / count)
        aspect = 16.0 / 9.0 if v % 2 else 4.0 / 3.0
        h = max(1, int(math.sqrt(area / aspect)))
        si = v % len(scenes)
        kind, n = scenes[si][:2]
        specs.append({"scene": si, "camera": _camera(kind, (n, n, n), seed * 64 + v, max(1, int(h * aspect)), h),
                      "spp": 1 + (v * 7 + 3) % case["max_spp"], "seed": v, "view_id": v,
                      "light": workloads.seeded_light(seed * 64 + v, shadows=v % 2 == 0)})
    return scenes, specs


# ---------------------------------------------------------------- the calls

def prepare(case, seed):
    call = case["call"]
    s = {"call": call}
    if call in ("render", "rays", "path", "page"):
        grid, vox, palette = _grid(case, seed)
        s.update(grid=grid, held=_Held(grid))
        dims = (case["nx"], case["ny"], case["nz"])
    if call in ("render", "path", "page"):
        s["camera"] = _camera(case["scene"], dims, seed + 1, case["width"], case["height"])
        pixels = case["width"] * case["height"]
    if call == "render":
        s["light"] = workloads.seeded_light(seed, shadows=case["shadows"]) if case["light"] else None
        s["hits"] = _records(pixels)
    elif call == "rays":
        g = torch.Generator(device="cuda").manual_seed(seed + 7)
        n = case["rays"]
        o = torch.rand((n, 3), generator=g, device="cuda") * torch.tensor(dims, device="cuda", dtype=torch.float32)
        d = F.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
        if n < 100000:  # queries along the axes and in axis planes among the others
            d[::16, 0] = 0.0
            d[::32, 1] = 0.0
            d[::32, 2] = torch.where(d[::32, 2] < 0.0, -1.0, 1.0)
        s.update(rays=torch.cat((o, d), 1).contiguous(), n=n, hits=_records(n))
    elif call == "path":
        s["params"] = vt.make_path_params(spp=case["spp"], max_bounces=case["bounces"], seed=seed & 0xFFFF)
        s["image"] = torch.empty((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
    elif call == "page":
        rng = np.random.default_rng(seed + 3)
        c = case["chunk"]
        x, y, z = (int(rng.integers(0, (d - c) // 8 + 1)) * 8 if c % 8 == 0 else int(rng.integers(0, d - c + 1))
                   for d in dims)
        before = vox[z:z + c, y:y + c, x:x + c].cpu().numpy()
        k = np.arange(c)
        ground = (0.5 + 0.3 * np.sin(k[None, :] * 0.4 + rng.uniform(0, 6)) * np.cos(k[:, None] * 0.3)) * c
        after = np.where(k[None, :, None] < ground[:, None, :], rng.integers(1, 256, (c, c, c)), 0).astype(np.uint8)
        order = vt.ORDER_Z_FASTEST if case["z_fastest"] else vt.ORDER_X_FASTEST
        if case["z_fastest"]:
            before, after = (np.ascontiguousarray(a.transpose(2, 1, 0)) for a in (before, after))
        s.update(origin=(x, y, z), before=np.ascontiguousarray(before), after=after, order=order, hits=_records(pixels))
    elif call == "scene":
        vox, palette = _scene(case["scene"], case["nx"], case["ny"], case["nz"], seed)
        dims = (case["nx"], case["ny"], case["nz"])
        s.update(vox=vox, palette=palette, dims=dims, hits=_records(case["width"] * case["height"]),
                 camera=_camera(case["scene"], dims, seed + 1, case["width"], case["height"]))
    elif call == "texture":
        vox, palette = _scene(case["scene"], case["nx"], case["ny"], case["nz"], seed)
        data = _texels(vox, palette) if case["rgba"] else vox.cpu().numpy()
        if case["z_fastest"]:
            data = np.ascontiguousarray(data.transpose(2, 1, 0))
        dims = (case["nx"], case["ny"], case["nz"])
        s.update(data=data, palette=None if case["rgba"] else palette, z_fastest=case["z_fastest"],
                 hits=_records(case["width"] * case["height"]),
                 camera=_camera(case["scene"], dims, seed + 1, case["width"], case["height"]))
    elif call == "views":
        scenes, specs = _views(case, seed)
        torch.cuda.synchronize()
        grids = [vt.Grid.from_u8_device(v, (n, n, n), pal) for _, n, v, pal in scenes]
        s["hits"] = [_records(p["camera"].width * p["camera"].height * p["spp"]) for p in specs]
        batch = vt.Batch([vt.make_view(grids[p["scene"]], p["camera"], h, p["spp"], p["seed"], p["view_id"], p["light"])
                          for p, h in zip(specs, s["hits"])])
        s.update(batch=batch, held=_Held(batch, *grids))
    elif call == "world":
        world = workloads.pager_world(load_dist=case["reach"], seed=seed & 0xFFFF)
        lib = vt.lib()
        if lib.entry() != 0:
            raise RuntimeError("entry() failed")
        ids = []
        for t in world["textures"]:
            nz, ny, nx = t.shape
            ids.append(lib.add_texture(t.ctypes.data, nx, ny, nz))
        if min(ids) < 0:
            raise RuntimeError("add_texture() failed: " + vt.last_error())
        inst = world["instances"]
        inst[:, 15] = np.array(ids, np.int32)[inst[:, 15].view(np.int32)].view(np.float32)
        s.update(lib=lib, instances=inst, P=world["P"], C=world["C"], width=ctypes.c_int32(0), height=ctypes.c_int32(0),
                 frame=torch.empty((world["height"], world["width"], 4), dtype=torch.uint8, pin_memory=True),
                 info=vt.RenderTickInfo(world["P"].ctypes.data, world["C"].ctypes.data))
    elif call == "serve":
        scenes, specs = _views(case, seed)
        service = vt.Service()
        ids = [service.add_scene(v.cpu().numpy(), pal) for _, _, v, pal in scenes]
        images = [torch.empty((p["camera"].height, p["camera"].width, 4), dtype=torch.uint8, pin_memory=True)
                  for p in specs]
        s.update(service=service, requests=[dict(p, scene=ids[p["scene"]]) for p in specs], images=images,
                 held=_Held(service))
    return s


def run(s):
    call = s["call"]
    if call == "render":
        vt.render(s["grid"], s["camera"], s["light"], s["hits"], torch.cuda.current_stream())
        return s["hits"]
    if call == "rays":
        vt.trace_rays(s["grid"], s["rays"], s["n"], s["hits"], torch.cuda.current_stream())
        return s["hits"]
    if call == "path":
        vt.path_trace(s["grid"], s["camera"], s["params"], s["image"], stream=torch.cuda.current_stream())
        return s["image"]
    if call == "views":
        s["batch"].run(torch.cuda.current_stream())
        return s["hits"]
    if call == "scene":
        stream = torch.cuda.current_stream()
        grid = vt.Grid.from_u8_device(s["vox"], s["dims"], s["palette"], stream)
        info = grid.info()
        vt.render(grid, s["camera"], None, s["hits"], stream)
        grid.destroy()
        return {"hits": s["hits"], "occupied": info["voxels_occupied"], "bricks": info["bricks_nonempty"]}
    if call == "texture":
        if s["z_fastest"]:
            grid = vt.Grid.from_chunk(s["data"], s["palette"])
        elif s["palette"] is None:
            grid = vt.Grid.from_rgba8(s["data"])
        else:
            grid = vt.Grid.from_u8(s["data"], s["palette"])
        info = grid.info()
        vt.render(grid, s["camera"], None, s["hits"], torch.cuda.current_stream())
        grid.destroy()
        return {"hits": s["hits"], "occupied": info["voxels_occupied"], "bricks": info["bricks_nonempty"]}
    if call == "page":  # the updates and the frame are ordered by the library's own stream
        s["grid"].update(s["origin"], s["after"], s["order"])
        vt.render(s["grid"], s["camera"], None, s["hits"], None)
        s["grid"].update(s["origin"], s["before"], s["order"])
        return s["hits"]
    if call == "world":
        lib, inst = s["lib"], s["instances"]
        ctypes.memmove(lib.start_update_instances(len(inst)), inst.ctypes.data, inst.nbytes)
        lib.end_update_instances(len(inst))
        lib.render_tick(ctypes.byref(s["width"]), ctypes.byref(s["height"]), ctypes.byref(s["info"]))
        lib.vt_framebuffer_download(s["frame"].data_ptr(), s["frame"].numel())
        return s["frame"]
    sent = [s["service"].submit(r["scene"], r["camera"], image, r["spp"], r["seed"], r["view_id"], r["light"])
            for r, image in zip(s["requests"], s["images"])]
    for request in sent:
        s["service"].wait(request)
    return s["images"]


# ---------------------------------------------------------------- what a pass cannot do without

def _bricks(case):
    return math.prod((case[k] + 7) // 8 for k in ("nx", "ny", "nz"))


def work(case):
    """Bytes: what comes in and goes out, once: hit records (16 B), rays (24 B), pixels, voxels, and
    4 B per brick of the traversed grid.  Operations: three per voxel step, with half the grid's
    mean side stepped per ray (the recurrence of the traversal: a comparison, an addition and an
    index)."""
    call = case["call"]
    if call in ("views", "serve"):
        count = case.get("views") or case["requests"]
        lo, hi = case["min_px"], max(case["max_px"], case["min_px"] + 1)
        samples = count * (hi - lo) / math.log(hi / lo) * (case["max_spp"] + 1) / 2.0
        side = (case["low"] + case["high"]) / 2.0
        out = samples * 16 if call == "views" else samples / ((case["max_spp"] + 1) / 2.0) * 4
        return {"bytes": out + case["scenes"] * (side / 8) ** 3 * 4, "flops": samples * 1.5 * side}
    if call == "world":
        chunks = (2 * case["reach"] + 1) ** 3 // 2 + 121
        return {"bytes": 1e6 * 4 + chunks * (64 + 8 * 4), "flops": 1e6 * 3 * 16}
    voxels = case["nx"] * case["ny"] * case["nz"]
    side = (case["nx"] + case["ny"] + case["nz"]) / 3.0
    if call == "rays":
        return {"bytes": case["rays"] * 40 + _bricks(case) * 4, "flops": case["rays"] * 1.5 * side}
    pixels = case["width"] * case["height"]
    if call == "path":
        rays = pixels * case["spp"] * (1 + case["bounces"]) * 1.5
        return {"bytes": pixels * 16 + _bricks(case) * 4, "flops": rays * 1.5 * side}
    rays = pixels * (2 if case.get("shadows") else 1)
    total = {"bytes": pixels * 16 + _bricks(case) * 4, "flops": rays * 1.5 * side}
    if call in ("scene", "texture"):  # the dense voxels in, the tables of the bricks out
        total["bytes"] += voxels * (4 if case.get("rgba") else 1) + _bricks(case) * 20
    elif call == "page":  # two chunks in, their bricks out
        total["bytes"] += 2 * 2 * case["chunk"] ** 3
    return total


def exact(case, seed):
    """Every output is whole numbers (packed hit records, pixels, counts) but the radiance of a path
    frame, whose binary64 restatement without this framework would take minutes (and takes other
    ways at voxel edges, so that single pixels differ by whole bounces)."""
    return None
