"""Workloads that performance work on the tracer is measured on.

Every case is one call sequence a host program makes through the public entry points:
a frame into a host film, a frame accumulated into a caller's device film, a render without
device allocation, a multi-camera session, a batch of animation frames with refits, a
stream of jobs through the render server, or a scene baked, rendered and freed in one call
(what the drop-in `renderForwardCuda` does).  Scenes are the repository's own synthetic
ones (Cornell box, dispersive glass, fog + strands) and a showroom that holds every
supported material; sizes span preview renders to production frames.

All outputs are whole numbers (64-bit fixed-point films and energy tallies): a film does not
depend on the order in which photons land, so another correct implementation gives the
same integers and cases are compared exactly.
"""
import ctypes
import math

import numpy as np
import torch

from goodphotons_b200 import abi, lib, scenes

FAMILIES = {"cornell": 8, "glass": 16, "fog_strands": 32, "showroom": 16}   # bounce caps


def _case(name, entry, scene, size, res_x, res_y, photons, hero=1, band=False, parts=1, bounces=0):
    c = {"entry": entry, "scene": scene, "size": size, "res_x": res_x, "res_y": res_y, "photons": photons,
         "hero": hero, "band": band, "parts": parts, "bounces": bounces or FAMILIES[scene]}
    return dict(c, name=name) if name else c


def listed():
    return [
        # an interactive preview: a small film, few photons, launch and call latency count
        _case("preview_cornell", "frame", "cornell", 0, 128, 128, 1 << 16),
        # a plug-in host that forbids device allocation while it renders, one progressive step
        _case("noalloc_steps", "noalloc", "glass", 16, 200, 120, 70_001, parts=3),
        # the Cornell configuration: 256^2, 2^24 photons, wavelengths uniform over 380-780 nm
        _case("cornell_frame", "frame", "cornell", 0, 256, 256, 1 << 24, band=True),
        # the reference's command line default, bundles of 4 wavelengths, on an odd film
        _case("cornell_hero4", "device", "cornell", 0, 301, 199, 3_000_001, hero=4),
        # the dispersive-caustics configuration: 327,680 triangles, 1024^2, half its photons
        _case("glass_frame", "frame", "glass", 128, 1024, 1024, 1 << 27),
        # bundles over glass: most paths lose their secondary wavelengths on the way
        _case("glass_hero4", "device", "glass", 64, 777, 555, 9_999_991, hero=4),
        # the fog + strands configuration (250k strands, 1M curve segments), half its photons
        _case("fog_strands_frame", "frame", "fog_strands", 250_000, 512, 512, 1 << 25),
        # every material, nested glass, planar mirrors and two lights
        _case("showroom_frame", "frame", "showroom", 24, 640, 360, 5_000_000),
        # animation: frames of one shared mesh, refit and rendered as one batch
        _case("animation_batch", "batch", "glass", 128, 512, 512, 1 << 25, parts=8),
        # four cameras connected to one set of paths, in two batches
        _case("session_4_views", "session", "glass", 64, 512, 288, 6_000_000, parts=4),
        # jobs of mixed scene, film and budget through the render server
        _case("served_jobs", "serve", "glass", 100, 512, 512, 1 << 25, parts=24),
        # the drop-in call: bake (device build), render, free
        _case("bake_and_render", "bake", "glass", 64, 512, 512, 1 << 22),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["frame", "frame", "frame", "device", "device", "noalloc", "batch", "session", "serve", "bake"])
    scene = rng.choice(["cornell", "glass", "fog_strands", "showroom"])
    if entry in ("batch", "serve"):
        scene = "glass"
    if entry == "noalloc" and scene == "showroom":   # its planar mirrors leave fewer photons a call
        scene = "cornell"
    size = {"cornell": 0, "glass": _log(rng, 7, 180), "fog_strands": _log(rng, 250, 250_000),
            "showroom": _log(rng, 7, 48)}[scene]
    res_x = _log(rng, 64, 1024)
    res_y = max(48, min(1024, int(res_x * rng.choice([1.0, 9 / 16, 3 / 4, 1.21]))))
    most = {"cornell": 1 << 26, "glass": 1 << 26, "fog_strands": 1 << 24, "showroom": 1 << 24}[scene]
    parts = 1
    if entry == "noalloc":
        most, parts = 32768 * 4, 4
    elif entry == "batch":
        most, parts = 1 << 25, rng.randint(2, 12)
    elif entry == "session":
        most, parts = most >> 2, rng.randint(2, 4)
    elif entry == "serve":
        most, parts = 1 << 25, rng.randint(4, 32)
    photons = _log(rng, 1 << 14, most)
    plain = entry in ("frame", "device", "bake")   # entry points where callers vary these
    hero = rng.choice([1, 1, 2, 4]) if plain and scene != "fog_strands" else 1
    band = rng.random() < 0.3 if plain else False
    return _case("", entry, scene, size, res_x, res_y, photons, hero=hero, band=band, parts=parts)


# ---- scenes -----------------------------------------------------------------------------
def _showroom(L, size, seed):
    sb = scenes.SceneBuilder()
    white = scenes.cornell_box(sb, boxes=False)
    mirror = sb.material(abi.MAT_MIRROR, reflect=sb.const(0.9))
    sb.quad((0.3, 0.3, 0.02), (1.4, 0, 0), (0, 1.4, 0), mirror)
    half = sb.material(abi.MAT_HALF_MIRROR, reflect=sb.table([(400, 0.3), (700, 0.7)]))
    sb.quad((1.35, 0.0, 1.3), (0.4, 0, -0.2), (0, 0.9, 0), half)
    sb.box((1.45, 0.5), (0.5, 0.5), 0.5, 25.0, sb.material(abi.MAT_GLOSSY, reflect=sb.const(0.8), roughness=0.3))
    sb.quad((0.2, 0.1, 1.6), (0.5, 0, 0), (0, 0.8, 0),
            sb.material(abi.MAT_FILTER, transmit=sb.table([(400, 0.2), (550, 0.9), (700, 0.3)])))
    sb.quad((1.3, 0.2, 1.7), (0.5, 0, 0.05), (0, 0.7, 0),
            sb.material(abi.MAT_DIFFUSE_TRANSMIT, reflect=sb.const(0.4), transmit=sb.const(0.35)))
    outer = sb.material(abi.MAT_DIELECTRIC, ior=sb.cauchy(1.5, 0.0042), absorb=sb.const(0.3), roughness=0.05,
                        priority=1)
    scenes.glass_blob(sb, center=(0.7, 0.5, 0.9), radius=0.35, amp=0.04, seed=seed, mat=outer, freq=size)
    inner = sb.material(abi.MAT_DIELECTRIC, ior=sb.sellmeier(1.03961212, 0.231792344, 1.01046945, 0.00600069867,
                                                             0.0200179144, 103.560653), priority=2)
    scenes.glass_blob(sb, center=(0.7, 0.5, 0.9), radius=0.15, amp=0.0, seed=seed, mat=inner, freq=8)
    v, f = scenes.geodesic_sphere(12)   # smooth-shaded, exact vertex normals
    tri = v[f]
    sb.tris((tri * 0.2 + np.array([1.2, 1.5, 0.7])).reshape(-1, 9), white, normals=tri.reshape(-1, 9))
    sb.sphere((1.5, 1.2, 0.6), 0.15, sb.diffuse(sb.const(0.6)))
    sb.sphere_light((0.4, 1.5, 1.4), 0.08, sb.blackbody(3000.0, 0.5))
    return sb.build(L)


def _desc(L, scene, size, seed):
    if scene == "glass":
        return scenes.make_glass(L, seed=seed, freq=size)
    if scene == "fog_strands":
        return scenes.make_fog_strands(L, n_strands=size, seed=seed)
    if scene == "showroom":
        return _showroom(L, size, seed)
    return scenes.make_cornell(L)


def _camera(L, res_x, res_y, eye_x=1.0):
    return L.look_at((eye_x, 1.0, 5.4), (1.0, 1.0, 1.0), (0.0, 1.0, 0.0), 40.0, res_x, res_y)


def _host_film(res_x, res_y):
    return torch.zeros(res_y, res_x, 4, dtype=torch.int64).pin_memory().numpy()


def _device_film(res_x, res_y):
    return torch.zeros(res_y, res_x, 4, dtype=torch.int64, device="cuda")


# ---- state and pass ---------------------------------------------------------------------
def prepare(case, seed):
    L = lib.load()
    rng = np.random.default_rng(seed)
    plan = np.random.default_rng(case["parts"])   # film sizes and budgets: the case's, not the seed's
    c, entry, n = dict(case), case["entry"], case["photons"]
    s = {"lib": L, "case": c, "base": int(rng.integers(0, 1 << 40)), "cam": _camera(L, c["res_x"], c["res_y"]),
         "mode": abi.LAMBDA_UNIFORM_380_780 if c["band"] else abi.LAMBDA_SPD}
    if entry == "batch":
        s["blas"] = lib.Blas(scenes.blob_tris(seed=seed, freq=c["size"]), 4, lib=L)   # the room's materials are 0-3
        desc = scenes.make_glass_instanced(L, handle=s["blas"])
        s["scene"] = lib.Scene(desc, 0, L)
        s["jobs"], s["films"], s["maps"] = [], [], []
        weights = np.exp2(plan.uniform(0.0, 5.0, c["parts"]))   # budgets 32 : 1, log-uniform
        counts = np.maximum(1, (n * weights / weights.sum()).astype(np.int64))
        base = s["base"]
        for i in range(c["parts"]):
            axis, angle, shift = rng.normal(size=3), rng.uniform(0, 360), rng.uniform(-0.2, 0.2, 3)
            m = scenes.affine(axis, angle, np.asarray(scenes.GLASS_CENTER) + shift)
            k = int(plan.integers(1, 5))   # a quarter to the whole of the largest film
            rx, ry = max(1, c["res_x"] * k // 4), max(1, c["res_y"] * k // 4)
            film = _device_film(rx, ry)
            s["maps"].append(m)
            s["films"].append(film)
            s["jobs"].append(dict(scene=s["scene"].clone_instances(m), cam=_camera(L, rx, ry), d_film=film.data_ptr(),
                                  n=int(counts[i]), seed_base=base, max_bounce=c["bounces"]))
            base += int(counts[i])
        return s
    if entry == "serve":
        library = {f: lib.Scene(_desc(L, f, size, seed), 0, L)
                   for f, size in (("cornell", 0), ("glass", c["size"]), ("fog_strands", 250 * c["size"]))}
        s["server"] = lib.Server(max_active=64, lib=L)
        weights = np.exp2(plan.uniform(0.0, 6.0, c["parts"]))
        counts = np.maximum(1, (n * weights / weights.sum()).astype(np.int64))
        base = s["base"]
        s["jobs"] = []
        for i in range(c["parts"]):
            fam = ("cornell", "glass", "fog_strands")[int(plan.integers(0, 3))]
            k = int(plan.integers(1, 5))
            rx, ry = max(1, c["res_x"] * k // 4), max(1, c["res_y"] * k // 4)
            s["jobs"].append(dict(scene=library[fam], cam=_camera(L, rx, ry), n=int(counts[i]), seed_base=base,
                                  max_bounce=FAMILIES[fam], host_film=_host_film(rx, ry)))
            base += int(counts[i])
        return s
    s["desc"] = _desc(L, c["scene"], c["size"], seed)
    if entry != "bake":
        s["scene"] = lib.Scene(s["desc"], 0, L)
    if entry in ("frame", "bake"):
        s["film"] = _host_film(c["res_x"], c["res_y"])
    elif entry in ("device", "noalloc"):
        s["film"] = _device_film(c["res_x"], c["res_y"])
    elif entry == "session":
        s["cams"] = (abi.Camera * c["parts"])(*[_camera(L, c["res_x"], c["res_y"], 0.7 + 0.2 * i)
                                               for i in range(c["parts"])])
        s["film"] = [_host_film(c["res_x"], c["res_y"]) for _ in range(c["parts"])]
    return s


def _tallies(energy):
    return np.array(list(energy.fx), dtype=np.int64)


def run(s):
    c, L, n = s["case"], s["lib"], s["case"]["photons"]
    entry, kw = c["entry"], dict(seed_base=s["base"], max_bounce=c["bounces"])
    if entry == "frame":
        film, _, en = s["scene"].render(s["cam"], n, out=s["film"], hero_c=c["hero"], lambda_mode=s["mode"], **kw)
        return film, _tallies(en)
    if entry == "device":
        stream = torch.cuda.current_stream().cuda_stream
        s["film"].zero_()
        s["scene"].render_device(s["cam"], n, s["film"].data_ptr(), stream=stream, hero_c=c["hero"],
                                 lambda_mode=s["mode"], **kw)
        return s["film"]
    if entry == "noalloc":
        stream = torch.cuda.current_stream().cuda_stream
        s["film"].zero_()
        per = -(-n // c["parts"])
        for first in range(0, n, per):
            p = abi.RenderParams(min(per, n - first), s["base"] + first, c["bounces"], 22, 1, s["mode"])
            L.check(L.L.ftb_render_forward_noalloc(s["scene"].h, ctypes.byref(s["cam"]), ctypes.byref(p),
                                                   ctypes.c_void_p(s["film"].data_ptr()), None, None,
                                                   ctypes.c_void_p(stream)))
        return s["film"]
    if entry == "batch":
        stream = torch.cuda.current_stream().cuda_stream
        for job, film, m in zip(s["jobs"], s["films"], s["maps"]):
            film.zero_()
            job["scene"].set_instance_transforms(m)
        _, ens = L.render_batch(s["jobs"], stream=stream)
        return s["films"], [_tallies(e) for e in ens]
    if entry == "session":
        h, en, info = ctypes.c_void_p(), abi.Energy(), abi.FilmInfo()
        L.check(L.L.ftb_session_begin(s["scene"].h, s["cams"], len(s["cams"]), c["bounces"], 20, c["hero"],
                                      ctypes.byref(h)))
        try:
            half = n // 2
            L.check(L.L.ftb_session_batch(h, half, s["base"]))
            L.check(L.L.ftb_session_batch(h, n - half, s["base"] + half))
            for i, film in enumerate(s["film"]):
                L.check(L.L.ftb_session_download(h, i, film.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)),
                                                 ctypes.byref(info), ctypes.byref(en)))
        finally:
            L.check(L.L.ftb_session_end(h))
        return s["film"], _tallies(en)
    if entry == "serve":
        ids = [s["server"].submit(j["scene"], j["cam"], j["n"], j["seed_base"], j["max_bounce"],
                                  host_film=j["host_film"]) for j in s["jobs"]]
        ens = [s["server"].wait(i) for i in ids]
        for r in ens:
            L.check(r.status)
        return [j["host_film"] for j in s["jobs"]], [_tallies(r.energy) for r in ens[:8]]
    scene = lib.Scene(s["desc"], 0, L, build=abi.BUILD_DEVICE)
    try:
        film, _, en = scene.render(s["cam"], n, out=s["film"], hero_c=c["hero"], lambda_mode=s["mode"], **kw)
    finally:
        scene.close()
    return film, _tallies(en)


# ---- the work and what results may differ by ----------------------------------------------
def work(case):
    """Bytes: the scene's primitives read once and the films written once.  Operations: per
    path vertex a closest-hit and an occlusion query -- one 8-wide node per level of the
    hierarchy (8 boxes of 6 planes, a multiply-add and a comparison each) and one exact
    primitive test (~100) -- and ~150 for the interaction, ~3 vertices per photon."""
    prims = {"cornell": 36, "glass": 20 * case["size"] ** 2 + 12, "fog_strands": 4 * case["size"] + 36,
             "showroom": 20 * case["size"] ** 2 + 4200}[case["scene"]]
    films = case["parts"] if case["entry"] in ("batch", "session", "serve") else 1
    share = 0.47 if case["entry"] in ("batch", "serve") else 1.0   # mean area of k/4-sized films
    levels = max(1.0, math.log(prims / 2.0, 8.0))
    vertex = 2 * (levels * 8 * 6 * 3 + 100) + 150
    return {"bytes": prims * 76 + films * share * case["res_x"] * case["res_y"] * 32,
            "flops": case["photons"] * 3 * vertex}


def tolerance(case):
    return "exact"


def exact(case, seed):
    """The outputs are whole numbers, compared as they are: there is no floating-point value
    that a 64-bit evaluation could be nearer to."""
    return None
