"""Performance cases of the path tracer: what a program that uses it has it render.

A case is a Renderer fed through set_scene / set_camera / render_frames as a viewer or an offline
renderer does it ("render"), a Batch of resident scenes rendered together ("batch"), or a Server that
is handed jobs and waited for ("serve").  Sizes follow the workloads of bench.py and the scenes of
ataraxia_gb300/scenes.py: 3 to 65,536 spheres, 1 to 64 samples per pixel and call, viewports from
256x256 to 3840x2160 and odd ones between, 2 to 15 bounces, 1 to 16 lights, with and without sky
light, accumulating under a still camera and restarting under a moving one, the scene resident or
uploaded again for every render, images read back at once, one render later, or left on the device.
"""
import math

import numpy as np
import torch

from ataraxia_gb300 import Batch, Camera, Renderer, Server, Settings, scenes
from ataraxia_gb300 import _native

# A "render" case:
#   spheres, clustered   sphere count; uniform in a box of the medium scene's density, on a ground sphere
#                        of radius 1000 (up to 24 spheres), or in 32 Gaussian clusters
#   materials, lights, emissive   table sizes; the share of the materials that emit
#   width, height, bounces, spp, sky
#   camera   "still": accumulates; "orbit": moves before every render and restarts the accumulation
#   upload   the scene is handed over again before every render (an animated scene)
#   overlap  the renderer is created with overlapped renders
#   read     "device": accumulator and image stay device buffers; "image": the RGBA8 image is read into
#            page-locked memory; "async": the same, waited for one render later


def _render(name, spheres, width, height, bounces, spp, *, lights=8, materials=64, clustered=False, emissive=0.0,
            sky=False, camera="still", upload=False, overlap=False, read="device"):
    c = {"kind": "render", "spheres": spheres, "clustered": clustered, "materials": materials, "lights": lights,
         "emissive": emissive, "width": width, "height": height, "bounces": bounces, "spp": spp, "sky": sky,
         "camera": camera, "upload": upload, "overlap": overlap, "read": read}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a material thumbnail refined one frame per call: the smallest call, all launch and latency
        _render("thumbnail", 9, 256, 256, 5, 1, lights=1, materials=8),
        # the interactive viewer on the small scene while its camera moves: one frame, shown at once
        _render("viewer_small_orbit", 9, 1280, 720, 5, 1, lights=1, materials=8, camera="orbit", read="image"),
        # the small scene rendered offline: its 64 frames in one call
        _render("small_64spp", 9, 1280, 720, 5, 64, lights=1, materials=8),
        # an outdoor scene with sky light and a few lamps, the default bounce depth, an odd viewport
        _render("sky_odd", 48, 1001, 563, 15, 4, lights=3, materials=16, emissive=0.2, sky=True),
        # the medium scene, progressive, every image read one render later: the steady state of a viewer
        # whose camera rests (bench.py's workload)
        _render("medium_16spp", 256, 1920, 1080, 8, 16, overlap=True, read="async"),
        # the medium scene while the camera moves: one sample per pixel, the accumulation restarted
        _render("medium_orbit", 256, 1920, 1080, 8, 1, camera="orbit", read="image"),
        # the medium scene animated: its spheres handed over again for every frame
        _render("medium_animated", 256, 1280, 720, 8, 16, upload=True),
        # the most spheres that go without a BVH, at an odd viewport, a default renderer
        _render("packed_1000", 1000, 1279, 719, 6, 8, lights=12),
        # the first sizes that go through the BVH, many samples in a call
        _render("bvh_4096", 4096, 1280, 720, 8, 16, materials=16),
        # the large clustered scene at 4K (bench.py's large scene)
        _render("large_4k", 65536, 3840, 2160, 8, 4, lights=16, materials=256, clustered=True),
        # sixteen scenes of the batched mix in one pass, their images read
        {"name": "batch_16", "kind": "batch", "scenes": 16, "spp": 0},
        # a render server that gets a burst of twelve small jobs and returns their images
        {"name": "serve_12", "kind": "serve", "jobs": 12},
    ]


_SIZES = ((256, 256), (320, 180), (511, 383), (640, 480), (853, 479), (1280, 720), (1281, 721), (1600, 900),
          (1920, 1080), (2560, 1440))


def draw(rng):
    kind = rng.choices(("render", "batch", "serve"), (10, 1, 1))[0]
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(2, 16), "spp": rng.randint(4, 32)}
    if kind == "serve":
        return {"kind": "serve", "jobs": rng.randint(2, 12)}
    n = int(round(math.exp(rng.uniform(math.log(3), math.log(40000)))))
    w, h = rng.choice(_SIZES)
    if rng.random() < 0.3:
        w, h = w - rng.randint(0, 37), h - rng.randint(0, 37)
    spp = int(round(math.exp(rng.uniform(0.0, math.log(64)))))
    if n > 1024:   # a walk costs several times a listed lookup: stay below the large scene's cost
        spp = max(1, min(spp, 16 * 1280 * 720 // (w * h)))
    while w * h * spp > 34_000_000:
        spp = max(1, spp // 2)
    camera = rng.choice(("still", "still", "orbit"))
    overlap = rng.random() < 0.3
    return _render(None, n, w, h, rng.randint(2, 15), spp, lights=rng.randint(1, 16),
                   materials=rng.choice((8, 16, 64, 256)), clustered=n > 1024 and rng.random() < 0.5,
                   emissive=rng.choice((0.0, 0.0, 0.2)), sky=rng.random() < 0.3, camera=camera,
                   upload=rng.random() < 0.15, overlap=overlap,
                   read="async" if overlap else rng.choice(("device", "image")))


# ------------------------------------------------------------------ inputs


def _scene(case, seed):
    """Spheres, materials, lights, and the camera's distance and height over its target."""
    st = scenes.Stream(int(seed), "case")
    n, nm, nl = case["spheres"], case["materials"], case["lights"]
    mats = scenes.draw_materials(st, nm)
    glow = st.uniform(nm) < case["emissive"]
    mats["emission_color"] = np.where(glow[:, None], st.uniform(3 * nm, 0.2, 1.0).reshape(nm, 3), 0.0)
    mats["emission_intensity"] = np.where(glow, 2.0, 0.0)
    if n <= 24 and not case.get("open"):   # the small scene: a handful of spheres on a ground sphere
        m = n - 1
        c = np.stack([st.uniform(m, -5, 5), st.uniform(m, 0, 3), st.uniform(m, -5, 5)], axis=1)
        c = np.vstack([c, [[0.0, -1000.0, 0.0]]])
        r = np.append(st.lognormal(0.0, 0.4, m), 1000.0)
        lights = scenes.draw_lights(st, nl, 8.0)
        lights["position"][:, 1] = np.abs(lights["position"][:, 1]) + 4.0
        dist, height = 10.0, 2.0
    elif case["clustered"]:
        k = 32
        at = st.uniform(3 * k, -100, 100).reshape(k, 3)
        c = at[st.integers(0, k, n)] + 5.0 * st.normal(3 * n).reshape(n, 3)
        r = st.lognormal(-1.5, 0.5, n)
        lights = scenes.draw_lights(st, nl, 30.0)
        dist, height = 320.0, 40.0
    else:
        half = 20.0 * (n / 256.0) ** (1.0 / 3.0)
        c = st.uniform(3 * n, -half, half).reshape(n, 3)
        r = st.lognormal(-0.5, 0.5, n)
        lights = scenes.draw_lights(st, nl, 1.5 * half)
        dist, height = 3.0 * half, 0.6 * half
    s = np.zeros(n, dtype=scenes.SPHERE_DTYPE)
    s["center"], s["radius"], s["material"] = c, r, st.integers(0, nm, n)
    return s, mats, lights, dist, height


def _mix(case):
    """The scenes of a "batch" or "serve" case: counts, viewports, depths and samples of the batched mix
    (scenes.batch_scene), the served jobs at most 640x480 and 16 or 64 samples per pixel."""
    st, parts = scenes.Stream(3, case["kind"]), []
    for i in range(case["jobs"] if case["kind"] == "serve" else case["scenes"]):
        sc = scenes.batch_scene(st, i)
        q = {"spheres": len(sc.spheres), "open": True, "clustered": False, "materials": 16, "lights": len(sc.lights),
             "emissive": 0.0, "width": sc.width, "height": sc.height, "bounces": sc.max_bounces,
             "spp": case.get("spp") or sc.spp}
        if case["kind"] == "serve":
            if sc.pixels > 640 * 480:
                q["width"], q["height"] = 640, 480
            q["spp"] = (16, 64)[i % 2]
        parts.append(q)
    return parts


def _camera(dist, height, step):
    """The camera after `step` moves around the target."""
    a = 0.01 * step
    p = np.array([dist * math.sin(a), height, dist * math.cos(a)])
    d = -p / np.linalg.norm(p)
    return Camera(45.0, 0.1, max(100.0, 4.0 * dist), tuple(p), tuple(d))


class _DeviceArray:
    """A device buffer for torch.as_tensor; the tensor keeps this object, and with it the renderer that owns the buffer."""

    def __init__(self, owner, pointer, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (pointer, False), "version": 2}


def prepare(case, seed):
    if case["kind"] != "render":
        parts = []
        for i, q in enumerate(_mix(case)):
            *arrays, dist, height = _scene(q, int(seed) * 64 + i)
            parts.append((*arrays, _camera(dist, height, 0), q["width"], q["height"],
                          Settings(accumulation=True, skyLight=False, maxBounces=q["bounces"])))
        if case["kind"] == "serve":
            jobs = [(*p, q["spp"]) for p, q in zip(parts, _mix(case))]
            return {"case": case, "server": Server(max_active_jobs=16), "jobs": jobs}
        b = Batch()
        ids = [b.add_scene(*p) for p in parts]
        for i, q in zip(ids, _mix(case)):
            b.set_spp(i, q["spp"])
        return {"case": case, "batch": b, "ids": ids}
    s, mats, lights, dist, height = _scene(case, seed)
    w, h = case["width"], case["height"]
    r = Renderer(flags=_native.FLAG_OVERLAP_RENDERS if case["overlap"] else 0)
    r.on_resize(w, h)
    r.set_settings(Settings(accumulation=True, skyLight=case["sky"], maxBounces=case["bounces"]))
    r.set_scene(s, mats, lights)
    r.set_camera(_camera(dist, height, 0))
    state = {"case": case, "r": r, "scene": (s, mats, lights), "view": (dist, height), "step": 0, "ticket": None}
    if case["read"] != "device":
        state["host"] = [torch.empty((h, w), dtype=torch.int32, pin_memory=True) for _ in range(2)]
        state["words"] = [x.numpy().view(np.uint32) for x in state["host"]]
    else:
        a, i = r.device_buffers()
        state["out"] = {"accumulation": torch.as_tensor(_DeviceArray(r, a, (h, w, 4), "<f4"), device="cuda"),
                        "image": torch.as_tensor(_DeviceArray(r, i, (h, w), "<i4"), device="cuda")}
        for x in state["out"].values():
            x.renderer = r
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.run()
        return [b.get_image(i).view(np.int32) for i in state["ids"]]
    if case["kind"] == "serve":
        srv = state["server"]
        ids = [srv.submit_scene(*job) for job in state["jobs"]]
        images = []
        for j in ids:
            srv.wait(j)
            images.append(srv.image(j).view(np.int32))
            srv.release(j)
        return images
    r = state["r"]
    state["step"] += 1
    if case["upload"]:
        r.set_scene(*state["scene"])
    if case["camera"] == "orbit":
        r.set_camera(_camera(*state["view"], state["step"]))
        r.reset_frame_index()
    r.render_frames(case["spp"])
    if case["read"] == "device":
        return state["out"]
    k = state["step"] & 1
    if case["read"] == "image":
        r.get_image(state["words"][k])
    else:
        ticket = r.read_image_async(state["words"][k])
        if state["ticket"] is not None:
            r.wait_read(state["ticket"])
        state["ticket"] = ticket
    return {"image": state["host"][k]}


# -------------------------------------------------------------------- work

# Shaded hits per path, as the renderer's ray statistics show for such scenes: most primary rays of the
# open scenes leave them; the ground sphere fills the small scene's lower half.
_HITS = {"small": 1.6, "open": 0.14}
_SHADE_FLOPS = 300   # position, normal, one Cook-Torrance term, shadow ray, roulette, the next direction


def _pass_work(n, pixels, paths, small, read_back):
    hits = paths * _HITS["small" if small else "open"]
    # the accumulator read and written and the image written once, the scene read once; a primary ray and
    # its nearest hit for every pixel, the shading of every hit, four additions per path
    return {"bytes": pixels * (16 + 16 + 4 + (4 if read_back else 0)) + 24 * n,
            "flops": 80 * pixels + _SHADE_FLOPS * hits + 4 * paths}


def work(case):
    if case["kind"] == "render":
        px = case["width"] * case["height"]
        return _pass_work(case["spheres"], px, px * case["spp"], case["spheres"] <= 24, case["read"] != "device")
    total = {"bytes": 0.0, "flops": 0.0}
    for q in _mix(case):
        px = q["width"] * q["height"]
        w = _pass_work(q["spheres"], px, px * q["spp"], False, True)
        total = {k: total[k] + w[k] for k in total}
    return total


# ------------------------------------------------------------ 64-bit result

_M32 = 0xFFFFFFFF


def _hash(x):
    s = (x * 747796405 + 2891336453) & _M32
    w = (((s >> ((s >> 28) + 4)) ^ s) * 277803737) & _M32
    return (w >> 22) ^ w


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _unit(a):
    return a / _dot(a, a).sqrt()


def _nearest(o, d, centre, r2):
    """Distance (inf: none) and index of the nearest sphere in front of each ray."""
    t, k = [], []
    step = max(1, (1 << 25) // len(r2))
    for i in range(0, len(o), step):
        p, v = o[i:i + step], d[i:i + step]
        a = _dot(v, v)
        b = _dot(p, v) - v @ centre.T
        c = _dot(p, p) - 2.0 * (p @ centre.T) + ((centre * centre).sum(-1) - r2)
        disc = b * b - a * c
        x = -(b + disc.clamp(min=0.0).sqrt()) / a
        x = torch.where((disc >= 0.0) & (x > 0.0), x, math.inf)
        m = x.min(dim=1)
        t.append(m.values)
        k.append(m.indices)
    if not t:
        return o[:, 0], torch.empty(0, dtype=torch.int64, device=o.device)
    return torch.cat(t), torch.cat(k)


def _trace(case, arrays, camera, frames):
    """The accumulator after the given frames: the reference's per-pixel loop in double precision."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def f64(x):
        return torch.from_numpy(np.array(x, dtype=np.float64)).to(dev)

    s, mats, lts = arrays
    centre, r2 = f64(s["center"]), f64(s["radius"]) ** 2
    smat = torch.from_numpy(s["material"].astype(np.int64)).to(dev)
    albedo, rough, metal, f0 = f64(mats["albedo"]), f64(mats["roughness"]), f64(mats["metallic"]), f64(mats["f0"])
    glow = f64(mats["emission_color"]) * f64(mats["emission_intensity"])[:, None]
    emits = f64(mats["emission_intensity"]) > 0.0
    lpos, le = f64(lts["position"]), f64(lts["color"]) * f64(lts["intensity"])[:, None]
    sky = torch.tensor([0.6, 0.7, 0.9], dtype=torch.float64, device=dev)
    w, h = case["width"], case["height"]
    eye, fwd = f64(np.float32(camera.position)), f64(np.float32(camera.direction))
    fwd = _unit(fwd)
    up = torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64, device=dev)
    right = _unit(torch.linalg.cross(fwd, up))
    top = torch.linalg.cross(right, fwd)
    th = math.tan(math.radians(camera.fov) / 2.0)
    pix = torch.arange(w * h, device=dev)
    cx = (pix % w).double() / w * 2.0 - 1.0
    cy = (pix // w).double() / h * 2.0 - 1.0
    prim = _unit(right * (cx * th * w / h)[:, None] + top * (cy * th)[:, None] + fwd)
    t0, k0 = _nearest(eye.expand_as(prim), prim, centre, r2)
    acc = torch.zeros(w * h, 4, dtype=torch.float64, device=dev)
    for frame in frames:
        path = pix
        seed = (pix * frame) & _M32
        o, d, thr = eye.expand_as(prim), prim, torch.ones_like(prim)
        t, k = t0, k0
        for bounce in range(case["bounces"]):
            if bounce:
                t, k = _nearest(o, d, centre, r2)
            miss = torch.isinf(t)
            if case["sky"]:
                acc[path[miss], :3] += sky * thr[miss]
            on = ~miss
            path, seed, o, d, thr, t, k = (x[on] for x in (path, seed, o, d, thr, t, k))
            if not len(path):
                break
            seed = (seed + bounce) & _M32
            pos = o + d * t[:, None]
            n = _unit(pos - centre[k])
            m = smat[k]
            alb, ro, me = albedo[m], rough[m][:, None], metal[m][:, None]
            lit = emits[m]
            acc[path[lit], :3] += glow[m][lit] * thr[lit]
            li = _hash(seed) % len(lpos)
            to = lpos[li] - pos
            dist2 = _dot(to, to)
            l = to / dist2.sqrt()
            hv = _unit(l - d)
            nl, nv = _dot(n, l).clamp(min=1e-7), -_dot(n, d).clamp(max=-1e-7)
            nh, vh = _dot(n, hv).clamp(min=0.0), (-_dot(d, hv)).clamp(0.0, 1.0)
            base = f0[m] * (1.0 - me) + alb * me
            fr = base + (1.0 - base) * (1.0 - vh) ** 5
            a2 = ro ** 4
            dn = math.pi * (nh * nh * (a2 - 1.0) + 1.0) ** 2
            kk = (ro + 1.0) ** 2 / 8.0
            g = nv / (nv * (1.0 - kk) + kk) * nl / (nl * (1.0 - kk) + kk)
            spec = fr * (a2 / dn * g) / (4.0 * nl * nv + 0.001)
            f = ((1.0 - fr) * (1.0 - me) * ((1.0 - fr) * alb / math.pi) + spec) * nl
            so = pos + 1e-4 * n
            ts, _ = _nearest(so, l, centre, r2)
            seen = ~(ts * ts < dist2[:, 0])
            acc[path[seen], :3] += (le[li] * f * thr)[seen]
            if bounce + 1 >= case["bounces"]:
                break
            thr = thr * alb
            p = _dot(thr, thr).sqrt().clamp(0.1, 1.0)
            seed = _hash(seed)
            on = ~(seed.double() / 4294967296.0 > p[:, 0])
            path, seed, n, thr, o, ro, me = (x[on] for x in (path, seed, n, thr / p, so, ro, me))
            seed = _hash(seed)
            u1 = (seed.double() / 4294967296.0)[:, None]
            seed = _hash(seed)
            u2 = (seed.double() / 4294967296.0)[:, None]
            ct = ((1.0 - u1) / (1.0 + (ro ** 4 - 1.0) * u1)).sqrt()
            z = torch.where(me > 0.0, ct, (1.0 - u1).sqrt())
            rad = torch.where(me > 0.0, (1.0 - ct * ct).clamp(min=0.0).sqrt(), u1.sqrt())
            zero = torch.zeros_like(n[:, 0])
            tx = torch.stack([-n[:, 2], zero, n[:, 0]], 1)
            ty = torch.stack([zero, -n[:, 2], n[:, 1]], 1)
            tan = _unit(torch.where((n[:, 0].abs() > n[:, 1].abs())[:, None], tx, ty))
            bit = torch.linalg.cross(n, tan)
            d = tan * (rad * torch.cos(2.0 * math.pi * u2)) + bit * (rad * torch.sin(2.0 * math.pi * u2)) + n * z
        acc[:, 3] += 1.0
    return acc.reshape(h, w, 4)


def exact(case, seed):
    if case["kind"] != "render" or case["read"] != "device":
        return None   # images only: whole numbers
    # where many small spheres graze one another a path in single precision takes another branch now and
    # then, and its pixel is off by a whole contribution: a frame in 64 bits says nothing about such scenes
    # (it is a tenth off at 1,000 spheres, a quarter at 4,096)
    if case["spheres"] > 64:
        return None
    *arrays, dist, height = _scene(case, seed)
    step = 1 if case["camera"] == "orbit" else 0
    acc = _trace(case, arrays, _camera(dist, height, step), range(1, case["spp"] + 1))
    return {"accumulation": acc, "image": None}
