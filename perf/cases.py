"""The work that programs have this renderer do, as timed cases.

Every case goes through the public entry points of ``spr.py`` (the mirror of
the C ABI), on seeded synthetic scenes of the kinds that the tests and the
benchmark use.  A case names what is done (``do``) and its sizes:

  frame     one RGBA8 frame of a device-resident scene, its image taken from
            the device (``rasterize`` + ``image_device_ptr``)
  upload    a document from host arrays to an image in host memory
            (``add_vg`` + ``rasterize`` + ``read_image``)
  animate   moved control points and the next frame (``update_vertices`` +
            ``rasterize``), with graph replay on, as a viewer does
  batch     many scenes of uneven size in one render
  fit       differentiable forward, L2 loss gradient, backward
  fit_batch the same for a batch of scenes, with the vertex update of a
            fitting step before it

Sizes are pixels, paths and curve segments per path (``seg_min`` to
``seg_max``); ``scene`` is the generator's kind.  Gradients and images come
back whole.
"""
import math
import pathlib
import sys

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parents[1]
PKG = ROOT / "gpu-scanline-path-rendering_gb300"
if str(PKG) not in sys.path:
    sys.path.insert(0, str(PKG))

import spr  # noqa: E402

KINDS = {"random": spr.SCENE_RANDOM, "mixed": spr.SCENE_MIXED, "cubics": spr.SCENE_CUBICS, "local": spr.SCENE_LOCAL}


def _frame(name, do, scene, width, height, samples, paths, large=0, seg_min=8, seg_max=32, rational=False,
           affine=False, ms_output=True, srgb=True, gradients=False):
    return {"name": name, "do": do, "scene": scene, "width": width, "height": height, "samples": samples,
            "paths": paths, "large": large, "seg_min": seg_min, "seg_max": seg_max, "rational": rational,
            "affine": affine, "ms_output": ms_output, "srgb": srgb, "gradients": gradients}


def listed():
    return [
        # an icon or a single glyph run: a handful of paths, where launches and latency count
        _frame("icon", "frame", "local", 128, 128, 8, 8),
        # the small plain scene of the benchmark: few overlapping paths over a whole small viewport
        _frame("small scene", "frame", "random", 512, 512, 8, 64),
        # a page of text and drawings from a file with per-path transforms and arcs
        _frame("page", "frame", "mixed", 1024, 1024, 32, 3000, large=300, rational=True, affine=True),
        # the benchmark's large scene: a dense map or drawing at full quality
        _frame("large drawing", "frame", "mixed", 2048, 2048, 32, 15000, large=5000, affine=True),
        # an odd widescreen viewport, 16 samples, coverage as alpha and no sRGB (the reference's non-multisample output)
        _frame("widescreen coverage", "frame", "local", 1917, 1079, 16, 2500, ms_output=False, srgb=False),
        # artwork with linear and radial paints on half of its paths
        _frame("gradient artwork", "frame", "local", 1366, 767, 8, 1200, gradients=True),
        # 256 samples per pixel: a still at reference quality
        _frame("still 256 samples", "frame", "cubics", 1024, 1024, 256, 256, seg_min=16, seg_max=64),
        # a document opened: host arrays in, image out, every pass
        _frame("open document", "upload", "mixed", 1280, 721, 32, 2000, large=100),
        # an animation: all control points move, the next frame follows
        _frame("animation", "animate", "cubics", 800, 600, 32, 256, seg_min=16, seg_max=64),
        # a server's batch of small documents of uneven size and two sample counts
        {"name": "batch of documents", "do": "batch", "scenes": 48, "size_min": 256, "size_max": 2048, "paths_min": 10,
         "paths_max": 5000, "seg_min": 8, "seg_max": 32, "samples": 8, "samples_2": 32},
        # one scene fitted to an image by gradient descent: forward, loss gradient, backward
        _frame("fit a scene", "fit", "cubics", 1024, 1024, 16, 256, seg_min=16, seg_max=64),
        # a batch of scenes fitted together, one descent step's renders
        {"name": "fit a batch", "do": "fit_batch", "scenes": 16, "size_min": 512, "size_max": 1024, "paths_min": 128,
         "paths_max": 512, "seg_min": 16, "seg_max": 64, "samples": 16, "samples_2": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["frame", "frame", "frame", "frame", "upload", "animate", "batch", "fit", "fit_batch"])
    if do == "batch":
        return {"do": do, "scenes": rng.randint(8, 40), "size_min": _log(rng, 64, 256), "size_max": _log(rng, 300, 1800),
                "paths_min": rng.randint(4, 20), "paths_max": _log(rng, 100, 4000), "seg_min": 8, "seg_max": 32,
                "samples": 8, "samples_2": rng.choice([8, 16, 32])}
    if do == "fit_batch":
        s = rng.choice([8, 16, 16, 32])
        return {"do": do, "scenes": rng.randint(2, 10), "size_min": rng.randint(200, 512),
                "size_max": rng.randint(520, 900), "paths_min": rng.randint(16, 128), "paths_max": rng.randint(130, 400),
                "seg_min": 8, "seg_max": rng.randint(16, 64), "samples": s, "samples_2": s}
    w, h = _log(rng, 64, 2048), _log(rng, 64, 2048)
    if do in ("animate", "fit"):
        return _plain(_frame("", do, "cubics", min(w, 1100), min(h, 1100), rng.choice([8, 16, 32]), _log(rng, 4, 300),
                             seg_min=4, seg_max=rng.randint(8, 64), affine=rng.random() < 0.3))
    scene = rng.choice(["local", "local", "mixed", "mixed", "random", "cubics"])
    smp = rng.choice([8, 16, 32, 32])
    kw = dict(rational=rng.random() < 0.5, affine=rng.random() < 0.5)
    if do == "frame":
        kw.update(srgb=rng.random() < 0.75, ms_output=rng.random() < 0.75)
        if scene == "local":
            kw.update(gradients=rng.random() < 0.4)
    if scene == "mixed":
        # (as dense as the large drawing at most: 15000 + 5000 paths on 2048 x 2048)
        most = max(8, int(15000 * w * h / 2048 ** 2))
        n = _log(rng, max(4, most // 64), most)
        return _plain(_frame("", do, scene, w, h, smp, n, large=n // rng.randint(3, 30), **kw))
    if scene == "random":  # every path over the whole viewport
        return _plain(_frame("", do, scene, min(w, 900), min(h, 900), smp, _log(rng, 2, 64), seg_max=rng.randint(8, 32),
                             **kw))
    if scene == "cubics":
        if do == "frame" and rng.random() < 0.3:
            smp, w, h = 256, min(w, 1000), min(h, 1000)
            kw.update(ms_output=True)
        return _plain(_frame("", do, scene, w, h, smp, _log(rng, 4, 250), seg_min=4, seg_max=rng.randint(8, 64), **kw))
    # (as dense as an icon of 64 paths at most)
    return _plain(_frame("", do, scene, w, h, smp, _log(rng, 2, min(2500, max(8, w * h // 256))), seg_min=4,
                         seg_max=rng.randint(8, 32), **kw))


def _plain(c):
    c.pop("name")
    return c


# ---- inputs ------------------------------------------------------------------
def _scene(case, seed):
    return spr.Scene.generate(KINDS[case["scene"]], seed=seed, width=case["width"], height=case["height"],
                              n_paths=case["paths"], n_large=case["large"], seg_min=case["seg_min"],
                              seg_max=case["seg_max"], with_rational=case["rational"], with_affine=case["affine"])


def _move(scene, width, height, rng):
    """Every path moved as a whole: a fit's scenes keep their elements, and so their gradients' shapes, from seed to
    seed."""
    d = rng.uniform(-0.2, 0.2, (scene.n_paths, 2)) * (width, height)
    scene.vertex = scene.vertex + d.astype(np.float32)[scene.vertex_path_id]


def _paint(scene, width, height, rng):
    """Radial paints on every other path: 64 gradients over 16 ramps of 256 texels."""
    n = 64
    table = np.zeros((n, 12), dtype=np.uint32)
    f = table.view(np.float32)
    for i in range(n):
        r = rng.uniform(0.05, 0.6) * min(width, height)
        cx, cy = rng.uniform(0, width), rng.uniform(0, height)
        f[i, 0:6] = (1 / r, 0, -cx / r, 0, 1 / r, -cy / r)
        table[i, 6] = 256 * (i % 16)
        f[i, 7] = 255 / 1024
        fx, fy = rng.uniform(-0.4, 0.4, 2)
        f[i, 8:11] = (fx, fy, max(0.0, 1 - fx * fx - fy * fy))
    stops = rng.uniform(0, 255, (16, 5, 4))
    stops[:, :, 3] = rng.uniform(128, 255, (16, 5))
    at = np.linspace(0, 4, 256)
    ramp = np.stack([np.stack([np.interp(at, np.arange(5), stops[k, :, c]) for c in range(4)], -1) for k in range(16)])
    words = ramp.round().astype(np.uint32).reshape(-1, 4)
    scene.path_fill_rgba[::2] = 1 + (np.arange(len(scene.path_fill_rgba[::2])) % n).astype(np.uint32)
    scene.gradients = (table.reshape(-1), words[:, 0] | words[:, 1] << 8 | words[:, 2] << 16 | words[:, 3] << 24)


def _items(case, seed):
    """The scenes of a batch: squares with sizes and path counts spread over their logarithm."""
    kind = spr.SCENE_LOCAL if case["do"] == "batch" else spr.SCENE_CUBICS
    n = case["scenes"]
    # (sizes, counts and their order are the case's own, the scenes' content the seed's)
    size = np.exp(np.linspace(math.log(case["size_min"]), math.log(case["size_max"]), n)).astype(int)
    paths = np.exp(np.linspace(math.log(case["paths_min"]), math.log(case["paths_max"]), n)).astype(int)
    items = []
    for j, i in enumerate(np.random.default_rng(n).permutation(n)):
        d = int(size[i])
        k = int(paths[(i * 7) % n])
        smp = case["samples"] if i % 2 == 0 else case["samples_2"]
        fit = case["do"] == "fit_batch"
        sc = spr.Scene.generate(kind, seed=(0 if fit else seed * 1000) + j, width=d, height=d, n_paths=k,
                                seg_min=case["seg_min"], seg_max=case["seg_max"])
        if fit:
            _move(sc, d, d, np.random.default_rng(seed * 1000 + j))
        items.append((sc, d, d, smp))
    return items


def _fills(n, rng):
    return np.c_[rng.uniform(0, 1, (n, 3)), rng.uniform(0.5, 1, (n, 1))].astype(np.float32)


def prepare(case, seed):
    rng = np.random.default_rng(seed + 77)
    dev = torch.device("cuda")
    st = {"do": case["do"], "stream": torch.cuda.current_stream().cuda_stream, "images": {}}
    if case["do"] in ("batch", "fit_batch"):
        items = _items(case, seed)
        b = spr.Batch()
        b.set_scenes(items)
        st["renderer"], st["sizes"] = b, [(h, w) for _, w, h, _ in items]
        if case["do"] == "fit_batch":
            vert = np.concatenate([it[0].vertex for it in items])
            pix, paths = sum(w * h for _, w, h, _ in items), sum(it[0].n_paths for it in items)
            st["vertex"] = torch.tensor(vert + rng.normal(0, 0.5, vert.shape).astype(np.float32), device=dev)
            _fit_buffers(st, (pix, 4), paths, len(vert), None, rng, dev)
        return st
    scene = _scene(case, 5 if case["do"] == "fit" else seed)
    if case["do"] == "fit":
        _move(scene, case["width"], case["height"], rng)
    if case["gradients"]:
        _paint(scene, case["width"], case["height"], rng)
    r = spr.VGRasterizer(case["width"], case["height"], samples=case["samples"], ms_output=case["ms_output"],
                         srgb=case["srgb"])
    st["renderer"], st["sizes"] = r, [(case["height"], case["width"])]
    if case["do"] == "upload":
        pinned = [torch.from_numpy(a).pin_memory().numpy() if a is not None else None
                  for a in (getattr(scene, f) for f in spr.Scene.FIELDS)]
        st["scene"] = spr.Scene(*pinned)
        st["host_image"] = torch.empty((case["height"], case["width"], 4), dtype=torch.uint8).pin_memory().numpy()
        return st
    r.add_vg(scene)
    if case["do"] == "animate":
        r.set_graph_replay(True)
        st["vertex"] = torch.tensor(scene.vertex + rng.normal(0, 0.5, scene.vertex.shape).astype(np.float32), device=dev)
    elif case["do"] == "fit":
        affine = scene.n_paths if case["affine"] else None
        _fit_buffers(st, (case["height"], case["width"], 4), scene.n_paths, scene.n_vertices, affine, rng, dev)
    return st


def _fit_buffers(st, image, paths, vertices, affine, rng, dev):
    st["fill"] = torch.tensor(_fills(paths, rng), device=dev)
    g = torch.Generator(device=dev).manual_seed(int(rng.integers(1 << 30)))
    st["target"] = torch.rand(image, device=dev, generator=g)
    st["image"], st["grad_image"] = torch.empty(image, device=dev), torch.empty(image, device=dev)
    st["grad_fill"] = torch.empty((paths, 4), device=dev)
    st["grad_vertex"] = torch.empty((vertices, 2), device=dev)
    st["grad_affine"] = None if affine is None else torch.empty((affine, 6), device=dev)


# ---- one pass ------------------------------------------------------------------
class _DeviceImage:
    """A renderer's RGBA8 image in device memory (keeps the renderer)."""

    def __init__(self, renderer, ptr, shape):
        self.renderer = renderer
        self.__cuda_array_interface__ = {"shape": (*shape, 4), "typestr": "|u1", "data": (ptr, False), "version": 2}


def _image(st, ptr, i):
    key = (i, ptr)
    if key not in st["images"]:
        st["images"][key] = torch.as_tensor(_DeviceImage(st["renderer"], ptr, st["sizes"][i]), device="cuda")
    return st["images"][key]


def run(st):
    r, sp, do = st["renderer"], st["stream"], st["do"]
    if do == "frame":
        r.rasterize(sp)
        return _image(st, r.image_device_ptr(), 0)
    if do == "upload":
        r.add_vg(st["scene"])
        r.rasterize(sp)
        return r.read_image(st["host_image"], sp)
    if do == "animate":
        r.update_vertices(st["vertex"].data_ptr(), sp)
        r.rasterize(sp)
        return _image(st, r.image_device_ptr(), 0)
    if do == "batch":
        r.render(sp)
        return [_image(st, r.image_device_ptr(i), i) for i in range(len(st["sizes"]))]
    if do == "fit_batch":
        r.update_vertices(st["vertex"].data_ptr(), sp)
    r.diff_render(st["fill"].data_ptr(), st["image"].data_ptr(), sp)
    torch.sub(st["image"], st["target"], out=st["grad_image"])
    st["grad_image"].mul_(2.0)
    ga = st["grad_affine"]
    r.diff_backward(st["fill"].data_ptr(), st["grad_image"].data_ptr(), st["grad_fill"].data_ptr(),
                    st["grad_vertex"].data_ptr(), None if ga is None else ga.data_ptr(), sp)
    out = {"image": st["image"], "grad_fill": st["grad_fill"], "grad_vertex": st["grad_vertex"]}
    if ga is not None:
        out["grad_affine"] = ga
    return out


# ---- what a pass cannot do without ---------------------------------------------
def _counts(scene, paths, large, seg_min, seg_max):
    """(curves, vertices) of a generated scene, on average."""
    per = {"random": 2.9, "local": 2.9, "cubics": 4.0}
    if scene == "mixed":  # glyphs: 25 quadratics and cubics; large: 275 segments of every kind
        return paths * 25 + large * 275, paths * 25 * 3.5 + large * 275 * 2.9
    c = paths * 0.5 * (seg_min + seg_max)
    return c, c * per[scene]


def work(case):
    """The scene's arrays read once (a vertex: position and path, 12 bytes; a
    curve: position, type, path and weight, 13; a path: fill, 5, and its
    transform, 24), the image written once, and for a fit its gradients; the
    vertex transform's operations and one blend per pixel."""
    if case["do"] in ("batch", "fit_batch"):
        n = case["scenes"]
        i = np.linspace(0, 1, n)
        size = np.exp(math.log(case["size_min"]) + i * math.log(case["size_max"] / case["size_min"]))
        paths = float(np.exp(math.log(case["paths_min"]) + i * math.log(case["paths_max"] / case["paths_min"])).sum())
        kind = "local" if case["do"] == "batch" else "cubics"
        curves, verts = _counts(kind, paths, 0, case["seg_min"], case["seg_max"])
        pix, per_path = float((size * size).sum()), 5
    else:
        paths = case["paths"] + case["large"]
        curves, verts = _counts(case["scene"], case["paths"], case["large"], case["seg_min"], case["seg_max"])
        pix, per_path = case["width"] * case["height"], 29 if case["affine"] else 5
    nbytes = 12 * verts + 13 * curves + per_path * paths + 4 * pix
    if case["do"] == "animate":
        nbytes += 8 * verts  # the new positions
    flops = 30 * verts + 12 * pix
    if case["do"] in ("fit", "fit_batch"):
        nbytes += 8 * verts + (8 * verts if case["do"] == "fit_batch" else 0) + 32 * paths + (12 + 32 + 16) * pix
        flops *= 2
    return {"bytes": float(nbytes), "flops": float(flops)}


def exact(case, seed):
    """None: images are bytes, and the float images and gradients of a fit
    follow from the renderer's own sample coverage (quantized half-planes of
    chords between cell lines), which plain numpy does not restate in the time
    a check may take."""
    return None
