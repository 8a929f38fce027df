"""The work a user of the framework has it do, as cases that can be timed and compared.

A case is a dict of plain values. ``kind`` selects the public calls that one pass makes:

frame           a renderer's frame: clear, cull, draw, resolve, Hi-Z build, read the image
deferred        a frame drawn by DeferredShader into a three-layer G-buffer
overdraw        a frame drawn by OverdrawShader, shown by resolve_debug
batch           many cameras moved, drawn by one call, and read
environment     a sky map uploaded, its mips built and its IBL maps computed
neural_resolve  a drawn frame shaded from learned textures
neural_train    some training steps of a learned texture set, and its new state
neural_probe    loss, gradients and decoded colours at explicit texels of one learned texture

Scenes are made on the GPU from the seed alone: closed 64-vertex, 124-triangle meshlets on a grid or
scattered in a volume at a constant density, with noise materials of two RGBA8 layers.
"""
import math

import numpy as np
import torch

from glimpsw_gb300 import api, scenes

VOLUME_DENSITY = 100_000 / 200.0 ** 3  # meshlets per cubic unit
# Share of a scene's meshlets that the outer camera's frustum holds, by layout (a camera inside the
# volume sees less); what a frame cannot do without is counted with it.
VISIBLE = {"grid": 0.95, "volume": 0.7, "inside": 0.3}


def listed():
    frame = {"kind": "frame", "layout": "volume", "materials": 32, "texture": 1024, "camera": "outside",
             "occlusion": False, "alpha": False}
    neural = {"materials": 32, "texture": 1024}
    return [
        # A thumbnail or icon view of a small object: every launch and call counts.
        {**frame, "name": "frame_thumbnail", "layout": "grid", "meshlets": 60, "width": 252, "height": 140, "materials": 1,
         "texture": 256},
        # The reference's small workload: 1024 meshlets on a grid at 1280x720, one 512x512 texture.
        {**frame, "name": "frame_720p", "layout": "grid", "meshlets": 1024, "width": 1280, "height": 720, "materials": 1,
         "texture": 512},
        # The benchmark's workload: 100,000 meshlets at 1920x1080, without a previous depth.
        {**frame, "name": "frame_1080p", "meshlets": 100_000, "width": 1920, "height": 1080},
        # The steady state of a renderer: the frame is culled against the previous frame's Hi-Z.
        {**frame, "name": "frame_occlusion_1440p", "meshlets": 150_000, "width": 2560, "height": 1440, "occlusion": True},
        # A camera inside the scene, half of the materials alpha-tested: clipping, near geometry, an odd size.
        {**frame, "name": "frame_alpha_inside", "meshlets": 50_000, "width": 1916, "height": 1036, "camera": "inside",
         "alpha": True},
        # A deferred renderer's G-buffer pass.
        {"name": "deferred_900p", "kind": "deferred", "layout": "volume", "meshlets": 30_000, "width": 1600, "height": 900,
         "materials": 32, "texture": 1024, "camera": "outside", "alpha": True},
        # The overdraw heat map of a scene, as a profiler view shows it.
        {"name": "overdraw_720p", "kind": "overdraw", "layout": "volume", "meshlets": 20_000, "width": 1280, "height": 720,
         "materials": 4, "texture": 256, "camera": "outside"},
        # Many cameras over one scene (shadow faces, sensors, training views), sizes from 256x256 to 2560x1440.
        {"name": "batch_24_views", "kind": "batch", "meshlets": 100_000, "views": 24, "least": 256, "most": 2560},
        # A new sky: upload, mips, irradiance, prefiltered radiance, BRDF table.
        {"name": "environment_1024", "kind": "environment", "texture": 1024, "irradiance": 64, "radiance": 256, "lut": 128},
        # A frame shaded from learned textures.
        {"name": "neural_resolve_1440p", "kind": "neural_resolve", "layout": "volume", "meshlets": 60_000, "width": 2560,
         "height": 1440, "camera": "inside", **neural},
        # Training of a texture set, in the benchmark's step: 8 materials of 8192 texels each.
        {"name": "neural_train_64k", "kind": "neural_train", "steps": 32, "batch": 65536, "step_materials": 8, "materials": 8,
         "texture": 1024},
        # A check or fine-tuning pass at chosen texels: gradients of the samples, colours of the texels.
        {"name": "neural_probe_256k", "kind": "neural_probe", "samples": 32_768, "texels": 262_000, "texture": 512},
    ]


def _log(rng, least, most, multiple=1):
    """A size between least and most, spread over its logarithm, rounded to a multiple."""
    v = math.exp(rng.uniform(math.log(least), math.log(most)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["deferred", "overdraw", "batch", "batch", "environment", "neural_resolve",
                                       "neural_train", "neural_probe"])
    width = _log(rng, 200, 2560, 4)  # landscape to square, as the frame driver's Hi-Z texture needs
    size = {"width": width, "height": min(1440, int(width * rng.uniform(0.45, 1.0)) // 4 * 4)}
    tex = 2 ** rng.randint(7, 10)
    if kind == "frame":
        small = rng.random() < 0.3
        return {"kind": kind, "layout": "grid" if small else "volume",
                "meshlets": _log(rng, 40, 4096) if small else _log(rng, 1000, 100_000), **size,
                "materials": rng.randint(1, 32), "texture": tex, "camera": rng.choice(["outside", "outside", "inside"]),
                "occlusion": rng.random() < 0.4, "alpha": rng.random() < 0.3}
    if kind == "deferred":
        return {"kind": kind, "layout": "volume", "meshlets": _log(rng, 500, 30_000), **size, "materials": rng.randint(1, 32),
                "texture": tex, "camera": rng.choice(["outside", "inside"]), "alpha": rng.random() < 0.5}
    if kind == "overdraw":
        return {"kind": kind, "layout": "volume", "meshlets": _log(rng, 500, 20_000), **size, "materials": rng.randint(1, 4),
                "texture": 256, "camera": "outside"}
    if kind == "batch":
        return {"kind": kind, "meshlets": _log(rng, 1000, 100_000), "views": rng.randint(2, 24), "least": 128,
                "most": _log(rng, 256, 2048)}
    if kind == "environment":
        return {"kind": kind, "texture": 2 ** rng.randint(7, 10), "irradiance": 2 ** rng.randint(3, 6),
                "radiance": 2 ** rng.randint(5, 8), "lut": 2 ** rng.randint(5, 7)}
    if kind == "neural_resolve":
        return {"kind": kind, "layout": "volume", "meshlets": _log(rng, 500, 60_000), **size, "camera": "inside",
                "materials": rng.randint(1, 32), "texture": 2 ** rng.randint(7, 10)}
    if kind == "neural_train":
        group = rng.randint(1, 8)
        return {"kind": kind, "steps": rng.randint(4, 32), "batch": 128 * group * rng.randint(1, 512 // group),
                "step_materials": group, "materials": group + rng.randint(0, 2), "texture": 2 ** rng.randint(7, 9)}
    return {"kind": kind, "samples": 128 * _log(rng, 1, 256), "texels": _log(rng, 100, 262_000), "texture": 2 ** rng.randint(7, 9)}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _octahedral(n):
    """Unit vectors as octahedral coordinates in [0, 1]."""
    w = 1.0 / n.abs().sum(-1)
    t = (-n[..., 2] * w).clamp(min=0.0)
    return torch.stack([n[..., 0] * w + torch.copysign(t, n[..., 0]), n[..., 1] * w + torch.copysign(t, n[..., 1])], -1) * 0.5 + 0.5


def _meshlets(g, centers, scales, materials):
    """Meshlet records (scenes.MESHLET_DTYPE) of displaced, turned, scaled spheres around centers."""
    n = len(centers)
    base, tris = scenes.meshlet_template()
    unit = torch.from_numpy(base).cuda()
    yaw = _uniform(g, 0.0, 2 * math.pi, n)
    local = unit[None] * (1.0 + 0.02 * torch.randn(n, 64, generator=g, device="cuda", dtype=torch.float64))[..., None]
    c, s = yaw.cos()[:, None], yaw.sin()[:, None]
    turned = torch.stack([c * local[..., 0] + s * local[..., 2], local[..., 1], -s * local[..., 0] + c * local[..., 2]], -1)
    world = turned * scales[:, None, None] + centers[:, None]
    rec = torch.zeros(n, scenes.MESHLET_SIZE, dtype=torch.uint8, device="cuda")
    f = rec.view(torch.float32)
    f[:, 16:208] = world.transpose(1, 2).reshape(n, 192).float()
    f[:, 0:3] = centers.float()
    f[:, 3] = ((world - centers[:, None]).norm(dim=2).amax(1) * (1 + 1e-6)).float()
    f[:, 4:7] = centers.float()
    f[:, 8] = 1.0   # a degenerate normal cone: axis +y, cutoff 1
    f[:, 10] = 1.0
    rec[:, 44], rec[:, 45], rec[:, 46] = 64, len(tris), 255
    rec.view(torch.int32)[:, 12] = materials.int()
    uv = ((base[:, :2] * 0.5 + 0.5) * 2.0).astype(np.float16).view(np.uint16).astype(np.int64)
    rec[:, 832:1088] = torch.from_numpy((uv[:, 0] | uv[:, 1] << 16).astype(np.uint32).view(np.uint8)).cuda()
    normal = turned / turned.norm(dim=2, keepdim=True)
    tangent = torch.stack([normal[..., 2], torch.zeros_like(normal[..., 0]), -normal[..., 0]], -1)
    tangent = tangent / tangent.norm(dim=2, keepdim=True).clamp(min=1e-9)
    pair = torch.cat([_octahedral(normal), _octahedral(tangent)], -1)
    rec[:, 1088:1344] = (pair.clamp(0, 1) * 255).round().to(torch.uint8).reshape(n, 256)
    index = np.zeros((3, 128), np.uint8)
    index[:, :len(tris)] = tris.T
    rec[:, 1344:1728] = torch.from_numpy(index.reshape(-1)).cuda()
    return rec.cpu().numpy().view(scenes.MESHLET_DTYPE).reshape(n)


def _noise_words(g, size, low, high):
    """A size x size image of RGBA8 noise (16-texel cells and a finer octave); low and high per channel."""
    def octave(cells):
        lattice = torch.rand(1, 4, cells, cells, generator=g, device="cuda")
        return torch.nn.functional.interpolate(lattice, size=(size, size), mode="bilinear")[0]

    v = 0.75 * octave(max(2, size // 16)) + 0.25 * octave(max(2, size // 4))
    lo, hi = (torch.tensor(x, device="cuda", dtype=torch.float32)[:, None, None] for x in (low, high))
    b = (lo + v * (hi - lo)).round().to(torch.int64)
    return (b[0] | b[1] << 8 | b[2] << 16 | b[3] << 24).to(torch.int32).contiguous()


def _texture(g, size, cutout=False):
    """A material: albedo (noise alpha when cut out), then normal XY, metallic and roughness."""
    t = api.Texture2D(api.FORMAT_RGBA8U, size, size, 16, 2)
    layers = [_noise_words(g, size, [0, 0, 0, 0 if cutout else 255], [255] * 4),
              _noise_words(g, size, [86, 86, 0, 51], [170, 170, 255, 255])]
    for i, words in enumerate(layers):
        t.set_pixels_device(words, i)
    t.generate_mips()
    return t, layers


def _sky_words(g, size):
    """An octahedral HDR sky as R11G11B10 words: a gradient with noise."""
    lattice = torch.rand(1, 3, 16, 16, generator=g, device="cuda")
    c = 0.2 + 3.8 * torch.nn.functional.interpolate(lattice, size=(size, size), mode="bilinear")[0]
    bits = c.contiguous().view(torch.int32).to(torch.int64)
    f11 = ((bits[:2] >> 17) & 0x3FFF) - 0x1C00
    f10 = ((bits[2] >> 18) & 0x1FFF) - 0x0E00
    return (f11[0] << 21 | f11[1] << 10 | f10).to(torch.int32).contiguous()


def _light():
    d = np.array([-0.589494, -0.684509, -0.428906])
    light = api.SwrLight()
    light.type, light.intensity = 0, 1500.0
    light.direction[:] = (d / np.linalg.norm(d)).tolist()
    light.color[:] = [1.0, 1.0, 1.0]
    return light


def _use_stream():
    torch.cuda.synchronize()
    api.load_library()
    api.set_stream(torch.cuda.current_stream())


def _scene(case, g):
    """The device scene of a case with its textures and the camera, and the previous frame's camera."""
    n, m = case["meshlets"], case["materials"]
    if case["layout"] == "grid":
        side = max(2, math.ceil(math.sqrt(n)))
        i = torch.arange(n, device="cuda")
        at = torch.stack([i % side, torch.zeros_like(i), i // side], 1).double() - torch.tensor([1.0, 0.0, 1.0], device="cuda") * (side - 1) / 2
        scale = torch.ones(n, device="cuda", dtype=torch.float64)
        eye, target = np.array([0.0, 0.44 * side, 0.75 * side]), np.array([0.0, 0.0, -0.06 * side])
        if case["camera"] == "inside":
            eye, target = np.array([0.0, 1.5, 0.1 * side]), np.array([0.0, 0.5, -0.5 * side])
    else:
        extent = 0.5 * (n / VOLUME_DENSITY) ** (1 / 3)
        at = _uniform(g, -extent, extent, n, 3)
        scale = _uniform(g, math.log(0.1), math.log(10.0), n).exp()
        eye, target = np.array([0.0, 0.0, -1.3 * extent]), np.zeros(3)
        if case["camera"] == "inside":
            eye, target = np.array([0.0, 0.0, -0.5 * extent]), np.array([0.3 * extent, 0.1 * extent, extent])
    eye = eye + _uniform(g, -0.01, 0.01, 3).cpu().numpy() * np.linalg.norm(target - eye)
    records = _meshlets(g, at, scale, torch.randint(0, m, (n,), generator=g, device="cuda"))
    alpha = case.get("alpha", False)
    textures = [_texture(g, case["texture"], cutout=alpha and i % 2 == 0)[0] for i in range(m)]
    table = np.zeros(m, scenes.MATERIAL_DTYPE)
    table["texture"], table["alpha_cutoff"] = np.arange(m), 255
    if alpha:
        table["alpha_cutoff"][::2], table["is_double_sided"][::2] = 128, 1
    scene = api.Scene()
    scene.upload_meshlets(records)
    scene.set_materials(table, textures)
    step = 0.003 * np.linalg.norm(target - eye)
    w, h = case["width"], case["height"]
    view = scenes.make_view(w, h, eye, target)
    before = scenes.make_view(w, h, eye + step * np.array([0.4, 0.2, 0.6]), target)
    torch.cuda.synchronize()
    return scene, textures, view, before


def _cull_args(s, view, prev, hiz):
    return (s["scene"], 0, s["meshlets"], s["bitmap"], api.mat4(view.proj), api.mat4(view.view), api.mat4(scenes.IDENTITY),
            api.mat4(prev.view), s["width"], s["height"], hiz)


def _image(s, layers=2):
    return [torch.empty(s["height"], s["width"], dtype=torch.int32, device="cuda") for _ in range(layers)]


def _read(s):
    for layer, out in enumerate(s["out"]):
        s["fb"].get_pixels_device(layer, out)
    return list(s["out"])


def _view_state(case, g, layers=2):
    s = {"kind": case["kind"], "meshlets": case["meshlets"], "width": case["width"], "height": case["height"]}
    s["scene"], s["textures"], s["view"], s["before"] = _scene(case, g)
    s["bitmap"] = torch.zeros((case["meshlets"] + 31) // 16, dtype=torch.int16, device="cuda")
    s["fb"] = api.Framebuffer(case["width"], case["height"], layers)
    s["raster"] = api.Rasterizer()
    s["raster"].EnableBinning = False  # the single-threaded reference's semantics: clips what needs it
    view = s["view"]
    s["draw"] = api.ShadingContext(s["scene"], view.world_to_clip, cull_bitmap=s["bitmap"])
    s["sky"] = api.Texture2D(api.FORMAT_R11G11B10F, 256, 256, 16, 1)
    s["sky"].set_pixels_device(_sky_words(g, 256))
    s["sky"].generate_mips()
    s["shade"] = api.ShadingContext(s["scene"], view.world_to_clip, world_to_clip=view.world_to_clip, skybox=s["sky"],
                                    view_pos=view.eye, lights=[_light()])
    s["cull"] = _cull_args(s, view, s["before"], None)
    s["out"] = _image(s, layers)
    return s


def _prepare_frame(case, g):
    s = _view_state(case, g)
    hw, hh = api.hiz_texture_size(case["width"], case["height"])
    s["hiz"] = [api.Texture2D(api.FORMAT_R32F, hw, hh, 16, 1) for _ in range(2)]
    if case["occlusion"]:  # the previous frame, seen from the camera's last place
        before = s["before"]
        s["fb"].clear(0xFF000000, 0.0)
        api.cull_meshlets(*_cull_args(s, before, before, None))
        s["raster"].draw_meshlets(s["fb"], s["meshlets"],
                                  api.ShadingContext(s["scene"], before.world_to_clip, cull_bitmap=s["bitmap"]))
        api.downsample_depth(s["fb"], s["hiz"][0])
        s["cull"] = _cull_args(s, s["view"], before, s["hiz"][0])
    return s


def _prepare_batch(case, g, seed):
    n = case["meshlets"]
    side = math.ceil(math.sqrt(n))
    i = torch.arange(n, device="cuda")
    at = torch.stack([i % side, torch.zeros_like(i), i // side], 1).double() - torch.tensor([1.0, 0.0, 1.0], device="cuda") * (side - 1) / 2
    records = _meshlets(g, at, torch.ones(n, device="cuda", dtype=torch.float64), torch.zeros(n, device="cuda"))
    scene = api.Scene()
    scene.upload_meshlets(records)
    table = np.zeros(1, scenes.MATERIAL_DTYPE)
    table["alpha_cutoff"] = 255
    scene.set_materials(table, [])
    # The sizes and heights are the case's own, so that every seed has the same load; places and
    # directions are the seed's.
    sizes, rng = np.random.default_rng(case["views"] * 100_003 + case["most"]), np.random.default_rng(seed)

    def cameras():
        half = side / 2
        moved = []
        for w, h, height, pitch in shapes:
            eye = np.array([rng.uniform(-0.5, 0.5) * half, height, rng.uniform(-0.5, 0.5) * half])
            yaw = rng.uniform(0, 2 * math.pi)
            moved.append(scenes.make_view(w, h, eye, eye + [math.cos(pitch) * math.cos(yaw), math.sin(pitch),
                                                            math.cos(pitch) * math.sin(yaw)]))
        return moved

    shapes = []
    for k in range(case["views"]):
        w = int(round(math.exp(sizes.uniform(math.log(case["least"]), math.log(case["most"]))) / 4)) * 4
        h = max(64, int(round(w * sizes.uniform(0.5, 1.0) / 4)) * 4)
        shapes.append((w, min(h, 1440), math.exp(sizes.uniform(math.log(1.5), math.log(60.0))),
                       math.radians(sizes.uniform(-70, -8))))
    fbs = [api.Framebuffer(w, h) for w, h, _, _ in shapes]
    # every fourth view keeps its depth alone (a shadow face)
    ways = [[(fb, v.proj, v.view, scenes.IDENTITY, k % 4 == 3) for k, (fb, v) in enumerate(zip(fbs, cameras()))] for _ in range(2)]
    raster = api.Rasterizer()
    raster.EnableBinning = False
    s = {"kind": "batch", "scene": scene, "raster": raster, "fbs": fbs, "ways": ways, "pass": 0}
    s["batch"] = api.Batch(raster, scene, ways[0])
    s["out"] = [torch.empty(h, w, dtype=torch.int32, device="cuda") for w, h, _, _ in shapes]
    return s


def _prepare_environment(case, g):
    def made(fmt, size, levels):
        return api.Texture2D(fmt, size, size, levels, 1)

    hdr = api.FORMAT_R11G11B10F
    return {"kind": "environment", "words": _sky_words(g, case["texture"]), "sky": made(hdr, case["texture"], 16),
            "irradiance": made(hdr, case["irradiance"], 1), "radiance": made(hdr, case["radiance"], 16),
            "lut": made(api.FORMAT_RG16F, case["lut"], 1)}


def _prepare_neural_resolve(case, g, seed):
    s = _view_state(case, g)
    s["model"] = api.NeuralMaterials(s["textures"], latent_levels=4, seed=seed + 1)
    return s


def _prepare_neural_train(case, g, seed):
    textures = [_texture(g, case["texture"])[0] for _ in range(case["materials"])]
    torch.cuda.synchronize()
    return {"kind": "neural_train", "model": api.NeuralMaterials(textures, latent_levels=4, seed=seed + 1),
            "train": {"steps": case["steps"], "batch": case["batch"], "materials_per_step": case["step_materials"],
                      "want_loss": True}}


def _probe_inputs(case, seed):
    """Texture words, network parameters, latents and texels of a neural_probe case."""
    g = _generator(seed)
    size = case["texture"]
    texels = sum((size >> 2 + l) ** 2 for l in range(4))
    spread = [(0, 64, 16, math.sqrt(6 / 75)), (1024, 64, 64, math.sqrt(6 / 128)), (5184, 8, 64, math.sqrt(6 / 72))]
    params = torch.zeros(5704, dtype=torch.float64, device="cuda")
    for start, rows, cols, a in spread:
        w = _uniform(g, -a, a, rows, cols)
        if cols == 16:
            w[:, 11:] = 0.0  # inputs without a meaning
        params[start:start + rows * cols] = w.reshape(-1)
    params[5120:5184] = _uniform(g, -0.1, 0.1, 64)
    params[5696:5704] = 0.5
    latents = _uniform(g, -1.0, 1.0, texels, 8).float()

    def places(count):
        level = torch.randint(0, 6, (count,), generator=g, device="cuda")
        x, y = (torch.rand(count, generator=g, device="cuda", dtype=torch.float64) for _ in range(2))
        edge = (size >> level)
        return level << 28 | (y * edge).long() << 14 | (x * edge).long()

    return g, params.float(), latents, places(case["samples"]), places(case["texels"])


def _prepare_neural_probe(case, seed):
    g, params, latents, samples, texels = _probe_inputs(case, seed)
    texture, _ = _texture(g, case["texture"])
    torch.cuda.synchronize()
    model = api.NeuralMaterials([texture], latent_levels=4, seed=seed + 1)
    model.set_params(0, params.cpu().numpy())
    model.set_latents(0, latents.cpu().numpy())

    def words(v):
        return (v - (v >> 31 << 32)).to(torch.int32)

    return {"kind": "neural_probe", "model": model, "samples": words(samples), "texels": words(texels),
            "colors": torch.empty(case["texels"], 2, dtype=torch.int32, device="cuda")}


def prepare(case, seed):
    _use_stream()
    g = _generator(seed)
    kind = case["kind"]
    if kind == "frame":
        s = _prepare_frame(case, g)
    elif kind in ("deferred", "overdraw"):
        s = _view_state(case, g, 3 if kind == "deferred" else 2)
    elif kind == "batch":
        s = _prepare_batch(case, g, seed)
    elif kind == "environment":
        s = _prepare_environment(case, g)
    elif kind == "neural_resolve":
        s = _prepare_neural_resolve(case, g, seed)
    elif kind == "neural_train":
        s = _prepare_neural_train(case, g, seed)
    else:
        s = _prepare_neural_probe(case, seed)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def _draw(s, shader=api.VisBufferShader):
    s["fb"].clear(0xFF000000 if shader != api.OverdrawShader else 0, 0.0)
    api.cull_meshlets(*s["cull"])
    s["raster"].draw_meshlets(s["fb"], s["meshlets"], s["draw"], shader)


def run(s):
    kind = s["kind"]
    if kind == "frame":
        _draw(s)
        s["shade"].resolve(s["raster"], s["fb"])
        api.downsample_depth(s["fb"], s["hiz"][1])
        return _read(s)
    if kind == "deferred":
        _draw(s, api.DeferredShader)
        return _read(s)
    if kind == "overdraw":
        _draw(s, api.OverdrawShader)
        s["shade"].resolve_debug(s["raster"], s["fb"], api.DEBUG_OVERDRAW_PIXEL)
        return _read(s)
    if kind == "batch":
        views = s["ways"][s["pass"] % 2]
        s["pass"] += 1
        s["batch"].set_views(views)
        s["batch"].render()
        for fb, view, out in zip(s["fbs"], views, s["out"]):
            fb.get_pixels_device(1 if view[4] else 0, out)
        return list(s["out"])
    if kind == "environment":
        s["sky"].set_pixels_device(s["words"])
        s["sky"].generate_mips()
        lib = api.load_library()
        for status in (lib.swr_ibl_irradiance_map(s["sky"].h, s["irradiance"].h),
                       lib.swr_ibl_radiance_map(s["sky"].h, s["radiance"].h), lib.swr_ibl_env_brdf_lut(s["lut"].h)):
            if status != api.SWR_OK:
                raise api.SwrError(status, lib.swr_last_error().decode())
        return [s[k].get_data().view(np.int32) for k in ("irradiance", "radiance", "lut")]
    if kind == "neural_resolve":
        _draw(s)
        s["shade"].resolve_neural(s["raster"], s["fb"], s["model"])
        return _read(s)
    model = s["model"]
    if kind == "neural_train":
        loss = model.train(**s["train"])
        state = range(model.num_materials)
        return {"loss": loss, "params": [model.get_params(i) for i in state], "latents": [model.get_latents(i) for i in state]}
    params, latents, loss = model.gradients(0, s["samples"], len(s["samples"]))
    model.decode(0, s["texels"], len(s["texels"]), s["colors"])
    return {"params": params, "latents": latents, "loss": loss, "colors": s["colors"]}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "environment":
        env = 4 * case["texture"] ** 2
        maps = 4 * (case["irradiance"] ** 2 + case["radiance"] ** 2 * 4 / 3 + case["lut"] ** 2)
        flops = case["irradiance"] ** 2 * 32400 * 110 + case["radiance"] ** 2 * 4 / 3 * 128 * 190 + case["lut"] ** 2 * 1024 * 60
        return {"bytes": env * 7 / 3 + maps, "flops": flops}
    weights = 11 * 64 + 64 * 64 + 64 * 8
    if kind == "neural_train":
        # the latents and the parameters with their two moments, read and written
        latent = sum((case["texture"] >> 2 + l) ** 2 for l in range(4)) * 32
        return {"bytes": case["materials"] * 6.0 * (latent + 4 * 5704),
                "flops": case["steps"] * case["batch"] * 6.0 * weights}
    if kind == "neural_probe":
        latent = sum((case["texture"] >> 2 + l) ** 2 for l in range(4)) * 32
        return {"bytes": 2.0 * latent + 12.0 * case["texels"] + 4.0 * case["samples"],
                "flops": (case["samples"] * 6.0 + case["texels"] * 2.0) * weights}
    if kind == "batch":
        pixels = case["views"] * 0.5 * case["most"] * (case["most"] + case["least"]) / 2 * 0.75
        seen = case["meshlets"] * 0.25 * case["views"]
        return {"bytes": case["meshlets"] * 1184.0 + pixels * 12.0, "flops": seen * (64 * 50 + 124 * 40)}
    seen = case["meshlets"] * VISIBLE["inside" if case["camera"] == "inside" else case["layout"]]
    pixels = case["width"] * case["height"]
    flops = seen * (64 * 50 + 124 * 40) + pixels * 600.0
    if kind == "neural_resolve":
        flops += pixels * 0.8 * 2.0 * weights
    # spheres for the cull, positions and indices of what is seen, four texels a pixel, the layers read back
    return {"bytes": 16.0 * case["meshlets"] + 1168.0 * seen + pixels * (16.0 + 8.0 + 8.0), "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits
def _mip_words(words, levels):
    """The levels of an RGBA8 image: each a 2x2 mean of the one above, rounded to 8 bits (float32
    arithmetic on values in [0, 1], as the format is defined)."""
    size = words.shape[0]
    v = torch.stack([(words.long() >> 8 * c & 255) for c in range(4)])
    out = [v]
    third = torch.tensor(1.0 / 255, dtype=torch.float32, device=words.device)
    for _ in range(1, levels):
        f = v.float() * third
        q = (((f[:, 0::2, 0::2] + f[:, 0::2, 1::2]) + f[:, 1::2, 0::2]) + f[:, 1::2, 1::2]) * 0.25
        v = (q * 255.0).round().clamp(0, 255).long()
        size //= 2
        out.append(v)
    return out


def exact(case, seed):
    """Gradients and loss of a neural_probe case in 64 bits. Images and maps are integers, and the
    samples of a training step are the library's own draw: those have no such value here."""
    if case["kind"] != "neural_probe":
        return None
    g, params, latents, samples, _ = _probe_inputs(case, seed)
    size = case["texture"]
    layers = [_noise_words(g, size, [0, 0, 0, 255], [255] * 4), _noise_words(g, size, [86, 86, 0, 51], [170, 170, 255, 255])]
    mips = [_mip_words(w, 6) for w in layers]
    level, y, x = samples >> 28, samples >> 14 & 0x3FFF, samples & 0x3FFF
    target = torch.ones(len(samples), 8, dtype=torch.float64, device="cuda")
    for l in range(6):
        at = (level == l).nonzero()[:, 0]
        target[at, 0:3] = mips[0][l][:3, y[at], x[at]].double().T / 255
        target[at, 3:7] = mips[1][l][:, y[at], x[at]].double().T / 255
    # bilinear taps on the latent level, wrapping
    lat = (level - 2).clamp(min=0)
    edge = (size // 4) >> lat
    offset = torch.tensor([sum((size >> 2 + k) ** 2 for k in range(l)) for l in range(4)], device="cuda")[lat]
    zoom = torch.where(level == 0, 4.0, torch.where(level == 1, 2.0, 1.0)).double()
    px, py = (x + 0.5) / zoom - 0.5, (y + 0.5) / zoom - 0.5
    fx, fy = px - px.floor(), py - py.floor()
    x0, y0 = px.floor().long() % edge, py.floor().long() % edge
    x1, y1 = (x0 + 1) % edge, (y0 + 1) % edge
    p = params.double().requires_grad_()
    q = latents.double().requires_grad_()

    def tap(tx, ty, w):
        return q[offset + ty * edge + tx] * w[:, None]

    h = tap(x0, y0, (1 - fx) * (1 - fy)) + tap(x1, y0, fx * (1 - fy)) + tap(x0, y1, (1 - fx) * fy) + tap(x1, y1, fx * fy)
    flags = torch.stack([torch.ones_like(fx), (level == 0).double(), (level == 1).double()], 1)
    h = torch.cat([h, flags, torch.zeros(len(h), 5, dtype=torch.float64, device="cuda")], 1)
    h = torch.nn.functional.gelu(h @ p[:1024].view(64, 16).T, approximate="tanh")
    h = torch.nn.functional.gelu(h @ p[1024:5120].view(64, 64).T + p[5120:5184], approximate="tanh")
    error = h @ p[5184:5696].view(8, 64).T + p[5696:] - target
    loss = error.square().sum()
    (loss / 1024).backward()  # the mean over a tile of 128 samples of 8 outputs, summed over tiles
    return {"params": p.grad.detach(), "latents": q.grad.detach(), "loss": float(loss.detach()), "colors": None}
