"""Performance cases of the path tracer: what a program that uses it has it do, over the sizes it does it at.

Scenes, frames, cameras and parameters have the shapes of the benchmark configurations (vktrace.configs) and of the
GPU tests; contents are random from the case's seed.  Every case goes through the C ABI's Python binding (vktrace.abi,
vktrace.autograd).  A program renders on one CUDA stream of its own; all states here share one.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "vk-renderer_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "vk-renderer_gb300"))

from vktrace import abi, autograd  # noqa: E402
from vktrace import scene as S  # noqa: E402

SKY = (1.0, 1.0, 1.0)
#: Most pixel x sample x depth steps of a drawn case: a third of what the largest listed frame has, as paths in a
#: closed scene, or with shadow rays, cost more a step than that frame's.
MOST_BOUNCES = 1920 * 1080 * 16 * 8 // 3


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # One small frame with a fixed time budget, for a program that may not allocate while it renders (a probe, a
        # thumbnail, a picture in a tool window): the smallest call, all latency and launches.
        {"name": "noalloc_96", "kind": "noalloc", "geometry": "soup", "tris": 2000, "extent": 10.0, "width": 96,
         "height": 96, "spp": 2, "depth": 4},
        # A quick look at a scene of spheres: 512^2, one sample, two bounces, median BVH (the c0 configuration).
        {"name": "spheres_512", "kind": "frame", "geometry": "spheres", "spheres": 64, "width": 512, "height": 512,
         "spp": 1, "depth": 2, "aov": "rgba8"},
        # The reference program's own frame: its scene of ten primitives (linear scan, light sphere, shadow rays)
        # at 1024^2 x 4 samples, then its present pass into its 1024 x 768 window.
        {"name": "draw_ref_1024", "kind": "draw", "geometry": "ref", "width": 1024, "height": 1024, "spp": 4,
         "depth": 4, "mode": "pingpong", "fb_width": 1024, "fb_height": 768, "fb": "rgba8"},
        # An interactive viewer that refines a still picture: a small ragged frame of one sample a pass, added to
        # the running mean and scaled up into a float framebuffer.
        {"name": "draw_preview_333x187", "kind": "draw", "geometry": "soup", "tris": 10_000, "extent": 10.0,
         "width": 333, "height": 187, "spp": 1, "depth": 4, "mode": "accumulate", "fb_width": 641, "fb_height": 359,
         "fb": "rgba32f"},
        # A scene of everything: triangles, spheres (some of them lights, so shadow rays at every diffuse hit) and
        # planes, with float output for a compositor.
        {"name": "mixed_640x360", "kind": "frame", "geometry": "mixed", "tris": 5000, "spheres": 48, "lights": 2,
         "extent": 10.0, "width": 640, "height": 360, "spp": 4, "depth": 6, "aov": "rgba8+rgba32f"},
        # A closed surface mesh (a terrain), as a modelled scene is: neighbouring triangles, most rays hit.
        {"name": "mesh_1280x720", "kind": "frame", "geometry": "mesh", "tris": 80_000, "width": 1280, "height": 720,
         "spp": 8, "depth": 8, "aov": "rgba8+linear"},
        # The flagship frame (the c1 configuration): 1920x1080, 16 samples, depth 8, 100k triangles, the picture
        # read back to the host.
        {"name": "soup_1080p", "kind": "frame", "geometry": "soup", "tris": 100_000, "extent": 50.0, "width": 1920,
         "height": 1080, "spp": 16, "depth": 8, "aov": "rgba8", "readback": True},
        # Many scenes of uneven size and resolution at once (a quarter of the c2 configuration), every picture read
        # back: data generation, thumbnails of a library of assets.
        {"name": "batch_16", "kind": "batch", "scenes": 16, "tris_lo": 1000, "tris_hi": 100_000, "res_lo": 128,
         "res_hi": 1024, "spp": 4, "depth": 6},
        # One backward pass alone (the c3 configuration): gradients of a 256^2 x 4 picture, tensors on the device.
        {"name": "adjoint_256", "kind": "adjoint", "geometry": "soup", "tris": 10_000, "extent": 10.0,
         "materials": 64, "width": 256, "height": 256, "spp": 4, "depth": 4, "edges": 0},
        # One step of gradient descent through torch.autograd on the largest scene (the c4 configuration's
        # 1M triangles, 1024 materials and depth 12, fewer pixels and samples): forward and backward.
        {"name": "step_1m_640", "kind": "step", "geometry": "soup", "tris": 1_000_000, "extent": 50.0,
         "materials": 1024, "width": 640, "height": 640, "spp": 16, "depth": 12},
        # The camera's gradient where lights and outlines move it: next-event terms (per-pixel adjoint) and the
        # triangles' outlines (edge sampling).
        {"name": "campos_160", "kind": "adjoint", "geometry": "mixed", "tris": 400, "spheres": 24, "lights": 1,
         "extent": 10.0, "materials": 16, "width": 160, "height": 160, "spp": 4, "depth": 4, "edges": 4},
        # The present pass alone: two 1024^2 pictures into a 1080p window.
        {"name": "present_1080p", "kind": "present", "src_width": 1024, "src_height": 1024, "src": "rgba8",
         "fb_width": 1920, "fb_height": 1080, "fb": "rgba8"},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _image(rng, c, lo, hi, spp_hi, depth_hi):
    """Width and height over the range (odd ones among them), then samples and depth within the cost of the largest."""
    c["width"] = _logint(rng, lo, hi)
    c["height"] = max(1, int(round(c["width"] * rng.choice([1.0, 9 / 16, 3 / 4, rng.uniform(0.4, 1.2)]))))
    c["spp"] = _logint(rng, 1, spp_hi)
    c["depth"] = rng.randint(2, depth_hi)
    while c["width"] * c["height"] * c["spp"] * c["depth"] > MOST_BOUNCES:
        c["spp"] = max(1, c["spp"] // 2)
        if c["spp"] == 1:
            c["depth"] = max(2, c["depth"] // 2)
            c["width"], c["height"] = c["width"] * 3 // 4, c["height"] * 3 // 4


def _geometry(rng, c, kinds, tris_hi):
    c["geometry"] = g = rng.choice(kinds)
    if g in ("soup", "mesh", "mixed"):
        c["tris"] = _logint(rng, 200, min(tris_hi, 20_000) if g == "mixed" else tris_hi)
    if g in ("soup", "mixed"):
        c["extent"] = rng.choice([10.0, 50.0])
    if g in ("spheres", "mixed"):
        c["spheres"] = _logint(rng, 8, 200)
    if g == "mixed":
        c["lights"] = rng.randint(0, 3)


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "draw", "noalloc", "batch", "adjoint", "adjoint", "step", "present"])
    c = {"kind": kind}
    if kind == "frame":
        _geometry(rng, c, ["soup", "soup", "mesh", "mesh", "mixed", "spheres", "ref"], 200_000)
        _image(rng, c, 64, 1920, 32, 12)
        c["aov"] = rng.choice(["rgba8", "rgba8+rgba32f", "rgba8+linear", "rgba8+hit"])
    elif kind == "draw":
        _geometry(rng, c, ["soup", "mesh", "mixed", "ref"], 100_000)
        _image(rng, c, 100, 1280, 4, 6)
        c["mode"] = rng.choice(["pingpong", "accumulate"])
        c["fb_width"], c["fb_height"] = _logint(rng, 100, 1920), _logint(rng, 100, 1080)
        c["fb"] = rng.choice(["rgba8", "rgba32f"])
    elif kind == "noalloc":
        _geometry(rng, c, ["soup", "mesh", "mixed", "spheres"], 50_000)
        _image(rng, c, 16, 128, 8, 8)
        c["height"] = min(c["height"], 128)
    elif kind == "batch":
        c.update(scenes=rng.randint(2, 24), tris_lo=rng.choice([200, 1000]), tris_hi=_logint(rng, 4000, 60_000),
                 res_lo=rng.choice([64, 100, 128]), res_hi=rng.choice([256, 512, 700]), spp=_logint(rng, 1, 8),
                 depth=rng.randint(2, 8))
    elif kind in ("adjoint", "step"):
        _geometry(rng, c, ["soup", "soup", "mesh", "mixed"] if kind == "adjoint" else ["soup", "mesh"], 100_000)
        _image(rng, c, 64, 640, 16, 8)
        c["materials"] = _logint(rng, 8, 1024)
        if kind == "adjoint":
            c["edges"] = rng.choice([0, 0, 4]) if c["tris"] <= 5000 else 0
    else:
        c.update(src_width=_logint(rng, 64, 2048), src_height=_logint(rng, 64, 2048),
                 src=rng.choice(["rgba8", "rgba32f"]), fb_width=_logint(rng, 64, 3840),
                 fb_height=_logint(rng, 64, 2160), fb=rng.choice(["rgba8", "rgba32f"]))
    return c


# ------------------------------------------------------------------ scenes --
def _triangles(v, material):
    t = np.zeros(len(v), S.TRIANGLE)
    t["v0"], t["v1"], t["v2"] = v[:, 0], v[:, 1], v[:, 2]
    t["material"] = material
    return t


def _soup(g, n, extent, n_mat):
    """The configurations' soup: centroids uniform in a cube, vertices normal about them (1 % of its half side)."""
    c = g.uniform(-extent, extent, (n, 1, 3))
    return _triangles((c + 0.01 * extent * g.standard_normal((n, 3, 3))).astype(np.float32), g.integers(0, n_mat, n))


def _mesh(g, n, n_mat):
    """A height field of about n triangles over unit cells, faces up; returns the triangles and its half side."""
    k = max(2, int(round(math.sqrt(n / 2))))
    x = np.arange(k + 1) - k / 2
    xx, zz = np.meshgrid(x, x, indexing="ij")
    y = 0.15 * g.standard_normal((k + 1, k + 1))
    for _ in range(6):
        w = 2 * math.pi * g.uniform(1.0, 6.0, 2) / k
        y += 0.02 * k * np.sin(w[0] * xx + w[1] * zz + g.uniform(0, 2 * math.pi))
    p = np.stack([xx, y, zz], -1).astype(np.float32)
    a, b, c, d = p[:-1, :-1], p[1:, :-1], p[:-1, 1:], p[1:, 1:]
    v = np.concatenate([np.stack([a, c, b], 2).reshape(-1, 3, 3), np.stack([b, c, d], 2).reshape(-1, 3, 3)])
    return _triangles(v, g.integers(0, n_mat, len(v))), k / 2


def _spheres(g, rng, n, lights, extent):
    s = np.zeros(n, S.SPHERE)
    s["P"] = g.uniform(-extent, extent, (n, 3))
    s["r"] = g.uniform(0.02, 0.15, n) * extent
    s["mat"] = S.random_materials(rng, n)
    for i in range(min(lights, n)):
        s[i]["mat"] = S.material((1.0, 1.0, 1.0), (40.0, 36.0, 30.0), 0.6, 0.0)
        s[i]["P"] = (g.uniform(-extent, extent), 1.2 * extent, g.uniform(-extent, extent))
    return s


def _scene(case, seed):
    """The scene, a camera that looks at it, and the parameters that go with its geometry."""
    g, rng = np.random.default_rng(seed), S.SplitMix64(seed)
    kind, n_mat = case["geometry"], case.get("materials", 256)
    if kind == "ref":
        return S.reference_scene(), S.reference_camera(), {"rr_start": 0, "tie_mode": abi.TIES_REFERENCE}
    if kind == "spheres":
        s = _spheres(g, rng, case["spheres"], 0, 10.0)
        return S.Scene(spheres=s, bvh=S.BVH_MEDIAN, leaf_size=2), S.look_at((0.0, 0.0, 25.0), (0.0, 0.0, 0.0), 40.0), \
            {"rr_start": 0, "sky": SKY}
    if kind == "mesh":
        t, half = _mesh(g, case["tris"], n_mat)
        sc = S.Scene(triangles=t, materials=S.random_materials(rng, n_mat), bvh=S.BVH_SAH)
        return sc, S.look_at((0.3 * half, 0.9 * half, -1.1 * half), (0.0, 0.0, 0.0), 60.0), {"rr_start": 3, "sky": SKY}
    extent = case["extent"]
    sc = S.Scene(triangles=_soup(g, case["tris"], extent, n_mat), materials=S.random_materials(rng, n_mat),
                 bvh=S.BVH_SAH, leaf_size=4, sah_bins=16)
    if kind == "mixed":
        sc.spheres = _spheres(g, rng, case["spheres"], case["lights"], extent)
        sc.planes = np.zeros(1, S.PLANE)
        sc.planes[0]["mat"] = S.material((0.8, 0.8, 0.8), roughness=0.4)
        sc.planes[0]["N"], sc.planes[0]["len"] = (0.0, 1.0, 0.0), 1.3 * extent
        return sc, S.look_at((0.0, 0.4 * extent, 2.5 * extent), (0.0, 0.0, 0.0), 40.0), \
            {"rr_start": 3, "sky": (0.2, 0.2, 0.2)}
    return sc, S.look_at((0.0, 0.0, 2.4 * extent), (0.0, 0.0, 0.0), 40.0), {"rr_start": 3, "sky": SKY}


_shared = {}


def _stream():
    if "stream" not in _shared:
        _shared["stream"] = torch.cuda.Stream()
    return _shared["stream"].cuda_stream


def _frame(camera, case, seed):
    g = np.random.default_rng(seed + 1)
    return S.frame(camera, case["width"] / case["height"] if case.get("geometry") != "ref" else S.REF_ASPECT,
                   float(np.float32(g.uniform(0.05, 0.95))))


AOVS = {"rgba8": abi.AOV_RGBA8, "rgba32f": abi.AOV_RGBA32F, "linear": abi.AOV_LINEAR, "hit": abi.AOV_PRIMARY_HIT}
TYPES = {abi.AOV_RGBA8: ("|u1", 4), abi.AOV_RGBA32F: ("<f4", 4), abi.AOV_LINEAR: ("<f4", 4),
         abi.AOV_PRIMARY_HIT: ("<i4", 2)}


def _buffer(width, height, aov):
    return torch.zeros((height, width, 4), dtype=torch.uint8 if aov == "rgba8" else torch.float32, device="cuda")


def _picture(case, seed, k):
    """A picture as the tracer leaves it: a smooth one with noise, in some parts more of it than in others."""
    w, h = case["src_width"], case["src_height"]
    base = torch.Generator(device="cuda").manual_seed(seed)
    low = torch.rand((1, 4, 9, 9), generator=base, device="cuda")
    low = torch.nn.functional.interpolate(low, size=(h, w), mode="bilinear", align_corners=True)[0]
    noise = torch.Generator(device="cuda").manual_seed(seed + 1 + k)
    im = low[:3] + (0.002 + 0.04 * (low[3] > 0.5)) * torch.randn((3, h, w), generator=noise, device="cuda")
    im = torch.cat([im.clamp(0, 1), torch.ones((1, h, w), device="cuda")]).permute(1, 2, 0).contiguous()
    return (im * 255 + 0.5).floor().to(torch.uint8) if case["src"] == "rgba8" else im


# ----------------------------------------------------------------- prepare --
def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "kind": kind, "tr": abi.Tracer(0), "stream": _stream()}
    tr = st["tr"]
    if kind == "present":
        st["images"] = [_picture(case, seed, 0), _picture(case, seed, 1)]
        st["out"] = _buffer(case["fb_width"], case["fb_height"], case["fb"])
        return st
    if kind == "batch":
        g = np.random.default_rng(seed)
        n = case["scenes"]
        tris = np.exp(g.uniform(math.log(case["tris_lo"]), math.log(case["tris_hi"]), n)).round().astype(int)
        tris[0], tris[-1] = case["tris_hi"], case["tris_lo"]
        res = np.exp2(np.linspace(math.log2(case["res_lo"]), math.log2(case["res_hi"]), n)).round().astype(int)
        scenes, st["frames"], st["params"], st["out"] = [], [], [], []
        for i in range(n):
            sub = {"geometry": "soup", "tris": int(tris[i]), "extent": 50.0, "width": int(res[i]),
                   "height": int(res[i])}
            sc, cam, extra = _scene(sub, seed + 1000 * i)
            scenes.append(sc)
            st["frames"].append(_frame(cam, sub, seed + 1000 * i))
            st["params"].append(abi.Tracer.params(sub["width"], sub["height"], spp=case["spp"],
                                                  max_depth=case["depth"], **extra))
            st["out"].append(torch.zeros((sub["height"], sub["width"], 4), dtype=torch.uint8).pin_memory().numpy())
        tr.upload_scenes(scenes)
        return st
    sc, cam, extra = _scene(case, seed)
    w, h = case["width"], case["height"]
    aovs = [AOVS[a] for a in case.get("aov", "rgba8").split("+")]
    st["frame"] = _frame(cam, case, seed)
    st["params"] = abi.Tracer.params(w, h, spp=case["spp"], max_depth=case["depth"], aovs=aovs, **extra)
    st["aovs"] = aovs
    if kind == "step":
        st["renderer"] = autograd.DifferentiableRenderer(tr, sc, st["frame"], st["params"])
        leaf = lambda a: torch.tensor(np.array(a, np.float32), device="cuda", requires_grad=True)  # noqa: E731
        st["leaves"] = [leaf(sc.materials["albedo"]), leaf(sc.materials["emissive"]), leaf(cam["pos"])]
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["target"] = torch.rand((h, w, 3), generator=g, device="cuda")
        return st
    tr.upload_scene(sc)
    if kind == "frame" and case.get("readback"):
        st["out"] = torch.zeros((h, w, 4), dtype=torch.uint8).pin_memory().numpy()
    elif kind == "draw":
        st["out"] = _buffer(case["fb_width"], case["fb_height"], case["fb"])
    elif kind == "noalloc":
        st["out"] = [_buffer(w, h, "rgba8"), _buffer(w, h, "rgba32f")]
    elif kind == "adjoint":
        # the loss gradient and the forward's linear image, as the forward pass of the same frame left them
        tr.set_edge_sampling(case["edges"])
        p = abi.Tracer.params(w, h, spp=case["spp"], max_depth=case["depth"], aovs=(abi.AOV_LINEAR,), **extra)
        tr.trace(st["frame"], p)
        g = np.random.default_rng(seed + 2)
        st["linear"] = torch.from_numpy(tr.readback(abi.AOV_LINEAR)).cuda()
        st["dl"] = torch.from_numpy((g.standard_normal((h, w, 4)) / (h * w)).astype(np.float32)).cuda()
        n_mat = len(sc.materials)
        st["out"] = [torch.zeros((n_mat, 3), device="cuda"), torch.zeros((n_mat, 3), device="cuda"),
                     torch.zeros(3, device="cuda")]
    return st


# --------------------------------------------------------------------- run --
def run(st):
    case, kind, tr, stream = st["case"], st["kind"], st["tr"], st["stream"]
    if kind == "frame":
        tr.trace(st["frame"], st["params"], stream=stream)
        if case.get("readback"):
            return tr.readback(abi.AOV_RGBA8, st["out"])
        if "views" not in st:  # device addresses stay the same while the image size does
            st["views"] = []
            for a in st["aovs"]:
                typestr, ch = TYPES[a]
                view = autograd._DeviceView(tr.device_image(a)[0], (case["height"], case["width"], ch), typestr)
                view.tracer = tr  # the picture's memory is the tracer's
                st["views"].append(torch.as_tensor(view, device="cuda"))
        return st["views"]
    if kind == "draw":
        mode = abi.PRESENT_PINGPONG if case["mode"] == "pingpong" else abi.PRESENT_ACCUMULATE
        tr.draw(st["frame"], st["params"], case["fb_width"], case["fb_height"], mode=mode, out_aov=AOVS[case["fb"]],
                out=st["out"].data_ptr(), stream=stream)
        return st["out"]
    if kind == "noalloc":
        tr.trace_noalloc(st["frame"], st["params"], st["out"][0].data_ptr(), st["out"][1].data_ptr(), stream=stream)
        return st["out"]
    if kind == "batch":
        tr.trace_batched(st["frames"], st["params"], use_graph=True, stream=stream)
        return [tr.readback_scene(i, abi.AOV_RGBA8, st["out"][i]) for i in range(case["scenes"])]
    if kind == "adjoint":
        tr.trace_adjoint(st["frame"], st["params"], st["dl"].data_ptr(), st["linear"].data_ptr(),
                         outputs=[t.data_ptr() for t in st["out"]], stream=stream)
        return st["out"]
    if kind == "step":
        for t in st["leaves"]:
            t.grad = None
        image = st["renderer"].render(*st["leaves"])
        # column 0 of every picture is NaN by definition (the shader divides by uv.x = 0 there)
        ((image[:, 1:] - st["target"][:, 1:]) ** 2).mean().backward()
        return {"image": image.detach(), "albedo": st["leaves"][0].grad, "emission": st["leaves"][1].grad,
                "campos": st["leaves"][2].grad}
    a, b = st["images"]
    tr.present((a.data_ptr(), case["src_width"], case["src_height"], AOVS[case["src"]]), (b.data_ptr(),),
               case["fb_width"], case["fb_height"], out_aov=AOVS[case["fb"]], out=st["out"].data_ptr(), stream=stream)
    return st["out"]


# -------------------------------------------------------------------- work --
def _trace_flops(prims, samples, depth, shadow):
    """Two rays a sample (fewer hit than miss, and roulette ends many of the rest), each down one path of a binary
    tree over the primitives (two boxes of 24 operations a level) and through four primitive tests of 45; a shadow ray
    more for each with lights; 300 operations of shading a ray."""
    rays = samples * min(depth, 2) * (2 if shadow else 1)
    return rays * (48.0 * math.log2(max(2, prims)) + 4 * 45.0 + 300.0)


def work(case):
    kind = case["kind"]
    size = {"rgba8": 4, "rgba32f": 16, "linear": 16, "hit": 8}
    if kind == "present":
        src, fb = case["src_width"] * case["src_height"], case["fb_width"] * case["fb_height"]
        return {"bytes": 2 * src * size[case["src"]] + fb * size[case["fb"]], "flops": fb * 2 * 60.0}
    if kind == "batch":
        n = case["scenes"]
        prims = math.sqrt(case["tris_lo"] * case["tris_hi"])
        px = sum(round(2 ** (math.log2(case["res_lo"]) + i / max(1, n - 1) *
                             math.log2(case["res_hi"] / case["res_lo"]))) ** 2 for i in range(n))
        return {"bytes": n * prims * 48 + px * 4, "flops": _trace_flops(prims, px * case["spp"], case["depth"], False)}
    px = case["width"] * case["height"]
    prims = 10 if case["geometry"] == "ref" else case.get("tris", 0) + case.get("spheres", 0)
    flops = _trace_flops(prims, px * case["spp"], case["depth"], case["geometry"] == "ref" or case.get("lights", 0) > 0)
    scene = 48 * prims + 48 * case.get("materials", 256)
    if kind == "adjoint":  # every sample's path once more, with dL/dI and the linear image read
        return {"bytes": scene + px * 32, "flops": flops}
    if kind == "step":  # forward (two float images) and backward
        return {"bytes": scene + px * 64, "flops": 2 * flops}
    if kind == "noalloc":
        return {"bytes": scene + px * 20, "flops": flops}
    if kind == "draw":
        fb = case["fb_width"] * case["fb_height"] * size[case["fb"]]
        return {"bytes": scene + px * (4 if case["mode"] == "pingpong" else 52) + fb, "flops": flops}
    return {"bytes": scene + px * sum(size[a] for a in case["aov"].split("+")), "flops": flops}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """The present pass in 64 bits.  A traced picture has no 64-bit value: its random numbers are the fraction of
    12345.6789 times the cosine of a number near 1e6 in 32 bits, and other digits there are another path."""
    if case["kind"] != "present" or case["fb"] == "rgba8":
        return None
    im = [_picture(case, seed, k).double() for k in (0, 1)]
    if case["src"] == "rgba8":
        im = [x / 255 for x in im]
    w, h, fw, fh = case["src_width"], case["src_height"], case["fb_width"], case["fb_height"]
    # bilinear, with a border of black
    pad = [torch.nn.functional.pad(x[..., :3].permute(2, 0, 1), (1, 1, 1, 1)).permute(1, 2, 0) for x in im]

    def tap(k, s, t):
        u, v = s * w - 0.5, t * h - 0.5
        i, j = u.floor(), v.floor()
        a, b = (u - i)[None, :, None], (v - j)[:, None, None]
        i, j = i.long() + 1, j.long() + 1
        at = lambda jj, ii: pad[k][jj.clamp(0, h + 1)][:, ii.clamp(0, w + 1)]  # noqa: E731
        return (1 - b) * ((1 - a) * at(j, i) + a * at(j, i + 1)) + b * ((1 - a) * at(j + 1, i) + a * at(j + 1, i + 1))

    s = (torch.arange(fw, device="cuda", dtype=torch.float64) + 0.5) / fw
    t = 1 - (torch.arange(fh, device="cuda", dtype=torch.float64) + 0.5) / fh
    c, o = tap(0, s, t), 1 / 2048
    mean = (tap(0, s, t + o) + tap(0, s, t - o) + tap(0, s + o, t) + tap(0, s - o, t)) / 4
    d = c - tap(1, s, t)
    rgb = torch.where((d * d).sum(-1, keepdim=True) > 0.0005, mean, c)
    return torch.cat([rgb, torch.ones_like(rgb[..., :1])], -1)
