"""The workloads that this framework's speed is judged by: what a program that renders, serves and
denoises has the library do, through its public calls, from the smallest call to the largest.

  render   agb_render of one view: interactive previews, progressive frames, served requests, with
           the options in earnest use (transparent shadows, distant lights, denoising AOVs, the
           ground plane, layered materials);
  viewer   an interactive viewer's loop: jittered frames of a moving camera, each rendered at one
           sample, resolved against its history and post-processed to 8-bit pixels on the host;
  batch    requests of several scenes, sizes and sample counts in one wavefront (the serving loop);
  load     opening a scene: BVH builds, environment table, uploads and the first image on the host;
  denoise  the learned denoiser's inference;
  train    one step of its training (loss, gradients, Adam);
  conv     one layer of it: the 3x3 convolution, forward;
  wgrad    one layer of it: the weight gradient.

Scenes are the repository's own seeded configurations (aurora_gb300.scenes) at their stated sizes or
smaller ones; sizes of the rest come from the bench's serving mix, training set and inference size.
"""
import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

from aurora_gb300 import _abi, api, scenes
from aurora_gb300.denoiser_training import Denoiser

# ------------------------------------------------------------------------------------- cases


def listed():
    return [
        # The smallest interactive call: a preview of the small scene while the camera is dragged.
        dict(name="preview", kind="render", scene="small", level=0, width=160, height=120, spp=1, depth=5,
             transparent=False, lights=0, aovs=False, ground=False),
        # The small configuration at its stated size.
        dict(name="frame_small", kind="render", scene="small", level=0, width=512, height=512, spp=16, depth=5,
             transparent=False, lights=0, aovs=False, ground=False),
        # The smallest request of the serving mix on a scene of the large type, with the AOVs that
        # a denoised answer needs.
        dict(name="request_large", kind="render", scene="large", level=6, width=640, height=360, spp=1, depth=8,
             transparent=False, lights=0, aovs=True, ground=False),
        # A progressive call of a full frame of the large type (several waves of the default size).
        dict(name="frame_large", kind="render", scene="large", level=7, width=1920, height=1080, spp=16, depth=8,
             transparent=False, lights=0, aovs=False, ground=False),
        # Layered materials under distant lights with transparent shadows, at an odd size.
        dict(name="frame_layered", kind="render", scene="layered", level=0, width=961, height=541, spp=4, depth=5,
             transparent=True, lights=2, aovs=False, ground=False),
        # Three frames of a viewer with temporal anti-aliasing.
        dict(name="viewer", kind="viewer", scene="small", level=0, width=1280, height=720, frames=3, depth=4,
             ground=True),
        # A batch as the serving loop forms it.
        dict(name="batch", kind="batch", requests=6, width=1280, height=720, level=6),
        # Opening a scene of the large type (the size the denoiser's training opens by the dozen).
        dict(name="load", kind="load", scene="large", level=6, env_width=512, env_height=256, width=256,
             height=256, depth=8),
        # Denoising a full frame, a training step on four crops, and two single layers at the
        # sizes that these two run them at.
        dict(name="denoise", kind="denoise", batch=1, height=1080, width=1920),
        dict(name="train", kind="train", batch=4, height=256, width=256),
        dict(name="conv_layer", kind="conv", batch=1, height=540, width=960, c0=128, c1=64, cout=64, up=True,
             relu=True),
        dict(name="wgrad_layer", kind="wgrad", batch=4, height=128, width=128, c0=64, c1=0, cout=64, up=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "viewer", "batch", "load", "denoise", "train", "conv", "wgrad"])
    if kind == "render":
        scene = rng.choice(["tiny", "small", "large", "layered"])
        w = _log(rng, 120, 1920)
        h = max(90, int(w * rng.uniform(0.5, 0.8)))
        spp = max(1, min(16, _log(rng, 1, 16), 8_000_000 // (w * h)))
        return dict(kind=kind, scene=scene, level=rng.randint(4, 6) if scene == "large" else 0, width=w, height=h,
                    spp=spp, depth=rng.randint(2, 8), transparent=rng.random() < 0.3, lights=rng.randint(0, 3),
                    aovs=rng.random() < 0.4, ground=scene in ("tiny", "small") and rng.random() < 0.3)
    if kind == "viewer":
        w = _log(rng, 240, 1920)
        return dict(kind=kind, scene=rng.choice(["tiny", "small"]), level=0, width=w,
                    height=int(w * rng.uniform(0.5, 0.8)), frames=rng.randint(2, 4), depth=rng.randint(2, 5),
                    ground=rng.random() < 0.5)
    if kind == "batch":
        w = _log(rng, 320, 1600)
        return dict(kind=kind, requests=rng.randint(2, 10), width=w, height=int(w * 9 / 16), level=rng.randint(4, 6))
    if kind == "load":
        n = _log(rng, 64, 1024)
        return dict(kind=kind, scene=rng.choice(["small", "large", "large", "layered"]), level=rng.randint(4, 6),
                    env_width=n, env_height=max(16, n // 2), width=_log(rng, 128, 640), height=_log(rng, 96, 360),
                    depth=rng.randint(3, 8))
    if kind == "denoise":
        b = rng.choice([1, 1, 1, 2])
        return dict(kind=kind, batch=b, height=16 * _log(rng, 8, 67 // b), width=16 * _log(rng, 10, 120 // b))
    if kind == "train":
        return dict(kind=kind, batch=rng.randint(1, 8), height=16 * rng.randint(4, 16),
                    width=16 * rng.randint(4, 16))
    c0 = 16 * _log(rng, 1, 16)
    up = rng.random() < 0.4
    c1 = 16 * _log(rng, 1, 8) if up else 0
    cout = rng.choice([16, 32, 64, 128, 256])
    h, w = 2 * _log(rng, 8, 270), 2 * _log(rng, 8, 480)
    batch = max(1, min(4, int(6e10 / (18.0 * (c0 + c1) * cout * h * w))))
    if kind == "conv":
        return dict(kind=kind, batch=batch, height=h, width=w, c0=c0, c1=c1, cout=cout, up=up,
                    relu=rng.random() < 0.7)
    return dict(kind=kind, batch=batch, height=h, width=w, c0=c0, c1=c1, cout=cout, up=up)


# ----------------------------------------------------------------------------- scenes and state


def _scene(name, seed, width, height, spp, depth, level=0, env=None):
    if name == "small":
        return scenes.config_small(seed=seed, width=width, height=height, spp=spp, trace_depth=depth)
    if name == "tiny":
        return scenes.config_tiny(seed=seed, width=width, height=height, spp=spp, trace_depth=depth)
    if name == "layered":
        return scenes.config_layered(seed=seed, width=width, height=height, spp=spp, trace_depth=depth)
    return scenes.config_large(seed=seed, width=width, height=height, spp=spp, trace_depth=depth, level=level,
                               env_size=env or (2048 >> (8 - level), 1024 >> (8 - level)))


def _lights(f, count, seed):
    """`count` distant lights of seeded directions, half a degree wide."""
    rng = np.random.default_rng(seed + 77)
    f["distant_light_count"] = count
    for k in range(count):
        d = np.array([rng.uniform(-1, 1), rng.uniform(0.4, 1), rng.uniform(-1, 1)])
        f["distant_lights"][k]["color_and_intensity"] = (1.0, 0.95, 0.9, rng.uniform(0.5, 2.0))
        f["distant_lights"][k]["direction"] = d / np.linalg.norm(d)
        f["distant_lights"][k]["cos_radius"] = math.cos(math.radians(0.25))


def _ground(s):
    lo, _ = s.bounds()
    s.ground_plane = _abi.ground_plane(position=(0.0, float(lo[1]) - 0.01, 0.0))


class State:
    """What a program keeps between passes; gives the library's objects back in their order."""

    def __init__(self, case):
        self.case = case
        self.views, self.renderers, self.batch, self.denoiser = [], [], None, None

    def __del__(self):
        for o in [self.batch, *self.views, *self.renderers, self.denoiser]:
            if o is not None:
                o.close()


class _Image:
    """An accumulation buffer of the library as a tensor (no copy); keeps the state alive."""

    def __init__(self, state, renderer, mode, width, height):
        self.state = state
        self.__cuda_array_interface__ = dict(shape=(height, width, 4), typestr="<f4", version=3, strides=None,
                                             data=(renderer.accum_device_ptr(mode), False))


def _image(state, renderer, mode, width, height):
    return torch.as_tensor(_Image(state, renderer, mode, width, height), device="cuda")


def _orbit(s, k):
    m = np.asarray(s.frame["camera_inv_view"], np.float64).reshape(-1)
    x, y, z = m[3], m[7], m[11]
    a = 0.06 * k
    return scenes.look_at((x * np.cos(a) + z * np.sin(a), y, -x * np.sin(a) + z * np.cos(a)), (0.0, 0.0, 0.0))


def _viewer_frames(s, count, depth):
    proj = scenes.perspective(45.0, s.width / s.height)
    out = []
    for k in range(count):
        prev = (_orbit(s, k - 1), proj, api.temporal_jitter(k - 1)) if k else None
        out.append(scenes.frame_data(_orbit(s, k), proj, trace_depth=depth, scene_bounds=s.bounds(), aovs=True,
                                     jitter=api.temporal_jitter(k), prev=prev))
    return out


def _requests(case):
    """The batch's requests: scene, size, samples (the serving mix's thirds, halves and sample
    counts, on two scenes)."""
    out = []
    for k in range(case["requests"]):
        div = (2, 3, 1)[k % 3]
        out.append((k % 2, case["width"] // div, case["height"] // div, (1, 4, 1, 1)[k % 4]))
    return out


# The denoiser's layers, as include/agb.h documents them: (inputs, output channels, level), in
# parameter order; a pair of inputs is (upsampled, skip).
_LAYERS = [("x", "e0a", 32, 0), ("e0a", "s0", 32, 0), ("p0", "e1a", 64, 1), ("e1a", "s1", 64, 1),
           ("p1", "e2a", 128, 2), ("e2a", "s2", 128, 2), ("p2", "ba", 256, 3), ("ba", "bb", 256, 3),
           (("bb", "s2"), "d2a", 128, 2), ("d2a", "d2", 128, 2), (("d2", "s1"), "d1a", 64, 1),
           ("d1a", "d1", 64, 1), (("d1", "s0"), "d0a", 32, 0), ("d0a", "d0", 32, 0), ("d0", "out", 16, 0)]


def _layer_shapes():
    ch = {"x": 16}
    out = []
    for src, dst, cout, level in _LAYERS:
        names = src if isinstance(src, tuple) else (src,)
        cin = sum(ch[n.replace("p", "s") if n[0] == "p" else n] for n in names)
        ch[dst] = cout
        out.append((cin, cout, level))
    return out


def _params(seed):
    """Weights of a network in use: He-normal, a small output layer, small biases."""
    g = torch.Generator().manual_seed(seed * 13 + 1)
    parts = []
    shapes = _layer_shapes()
    for i, (cin, cout, _) in enumerate(shapes):
        sd = math.sqrt(2.0 / (9 * cin)) * (0.1 if i == len(shapes) - 1 else 1.0)
        parts.append(torch.randn(9 * cin * cout, generator=g) * sd)
        parts.append(torch.randn(cout, generator=g) * 0.02)
    return torch.cat(parts)


def _features(batch, height, width, seed):
    """Feature images as a rendered frame gives them: log radiance, albedo, normal, depth, variance
    over smooth regions with noise, six channels of zeros (BF16)."""
    g = torch.Generator(device="cuda").manual_seed(seed * 7 + 3)
    def rand(*shape):
        return torch.rand(shape, generator=g, device="cuda")
    coarse = rand(batch, 10, max(2, height // 32), max(2, width // 32))
    smooth = F.interpolate(coarse, size=(height, width), mode="bilinear")
    x = torch.zeros(batch, height, width, 16, device="cuda")
    noise = torch.randn(batch, height, width, 10, generator=g, device="cuda")
    x[..., :10] = smooth.permute(0, 2, 3, 1) + 0.1 * noise
    x[..., :3] = torch.log1p(2.0 * x[..., :3].clamp(min=0.0))
    x[..., 6:8] = 2.0 * x[..., 6:8] - 1.0
    x[..., 8:10] = x[..., 8:10].clamp(min=0.0)
    return x.to(torch.bfloat16).contiguous()


def _target(x, seed):
    """A reference radiance for the features: the noisy one smoothed, scaled and offset."""
    r = torch.expm1(x[..., :3].float()).permute(0, 3, 1, 2)
    r = F.avg_pool2d(r, 5, stride=1, padding=2, count_include_pad=False).permute(0, 2, 3, 1)
    out = torch.ones(*x.shape[:3], 4, device="cuda")
    out[..., :3] = 1.5 * r + 0.3
    return out.contiguous()


def _layer_tensors(case, seed):
    """A layer's inputs: activations after a ReLU (BF16), the output's gradient, weights, bias."""
    g = torch.Generator(device="cuda").manual_seed(seed * 11 + 2)
    b, h, w, up = case["batch"], case["height"], case["width"], case["up"]
    h0, w0 = (h // 2, w // 2) if up else (h, w)
    cin = case["c0"] + case["c1"]
    def act(*shape):
        return torch.randn(shape, generator=g, device="cuda").clamp(min=0.0).to(torch.bfloat16)
    x0 = act(b, h0, w0, case["c0"])
    x1 = act(b, h, w, case["c1"]) if case["c1"] else None
    dy = (torch.randn(b, h, w, case["cout"], generator=g, device="cuda") * 1e-2).to(torch.bfloat16)
    wt = torch.randn(9, cin, case["cout"], generator=g, device="cuda") * math.sqrt(2.0 / (9 * cin))
    bias = torch.randn(case["cout"], generator=g, device="cuda") * 0.02
    return x0, x1, dy, wt, bias


def prepare(case, seed):
    kind = case["kind"]
    st = State(case)
    if kind in ("render", "viewer"):
        s = _scene(case["scene"], seed, case["width"], case["height"], case.get("spp", 1), case["depth"],
                   case["level"])
        if case["ground"]:
            _ground(s)
        r = api.Renderer()
        st.renderers.append(r)
        r.upload(s)
        if kind == "viewer":
            st.frames = _viewer_frames(s, case["frames"], case["depth"])
        else:
            f = np.asarray(s.frame).copy()
            f["is_force_opaque_shadows_enabled"] = 0 if case["transparent"] else 1
            f["is_denoising_aovs_enabled"] = 1 if case["aovs"] else 0
            if case["lights"]:
                _lights(f, case["lights"], seed)
            st.frame = f
    elif kind == "batch":
        for k in range(2):
            s = _scene(("small", "large")[k], seed + k, case["width"], case["height"], 1, (5, 8)[k], case["level"])
            r = api.Renderer()
            st.renderers.append(r)
            r.upload(s)
        st.batch = api.Batch(max_paths=1 << 23)
        st.items = []
        for k, (scene, w, h, spp) in enumerate(_requests(case)):
            v = api.View(st.renderers[scene])
            st.views.append(v)
            f = np.asarray(st.renderers[scene].scene.frame).copy()
            v.set_frame(f)
            st.items.append(dict(view=v, width=w, height=h, spp=spp, seed_offset=1000 * seed + 64 * k,
                                 accumulation=_abi.ACCUM_RUNNING_MEAN))
    elif kind == "load":
        st.scene = _scene(case["scene"], seed, case["width"], case["height"], 1, case["depth"], case["level"],
                          (case["env_width"], case["env_height"]))
    elif kind in ("denoise", "train"):
        b, h, w = case["batch"], case["height"], case["width"]
        st.denoiser = Denoiser(seed=11)
        p = _params(seed)
        st.denoiser.set_params(p.numpy())
        st.x = _features(b, h, w, seed)
        if kind == "denoise":
            st.out = torch.zeros(b, h, w, 4, device="cuda")
        else:
            st.target = _target(st.x, seed)
            st.grads = np.zeros(p.numel(), np.float32)
    else:
        lib = _abi.library()
        st.x0, st.x1, st.dy, wt, st.bias = _layer_tensors(case, seed)
        cin = case["c0"] + case["c1"]
        if kind == "conv":
            st.wpack = torch.zeros(9 * cin * case["cout"], dtype=torch.int16, device="cuda")
            _abi.check(lib.agb_pack_conv_weights(wt.data_ptr(), cin, case["cout"], 0, st.wpack.data_ptr(), None))
            st.out = torch.zeros(case["batch"], case["height"], case["width"], case["cout"], dtype=torch.bfloat16,
                                 device="cuda")
        else:
            st.dw = torch.zeros(9, cin, case["cout"], device="cuda")
        torch.cuda.synchronize()  # the layer calls below run on the default stream, torch's inputs too
    return st


# ------------------------------------------------------------------------------------ one pass


def run(st):
    case = st.case
    kind = case["kind"]
    if kind == "render":
        r, w, h = st.renderers[0], case["width"], case["height"]
        r.set_frame(st.frame)
        r.render(0, case["spp"])
        return [_image(st, r, _abi.ACCUM_RUNNING_MEAN, w, h), _image(st, r, _abi.ACCUM_KAHAN, w, h)]
    if kind == "viewer":
        r = st.renderers[0]
        shown = []
        for k, f in enumerate(st.frames):
            r.set_frame(f)
            r.render(0, 1, accumulation=_abi.ACCUM_RUNNING_MEAN, seed_offset=k + 1)
            r.temporal_resolve(reset=(k == 0))
            _, o8 = r.post_process(mode=_abi.POST_SOURCE_TEMPORAL, tone_map=True)
            shown.append(o8)
        return [shown, r.temporal_read()]
    if kind == "batch":
        st.batch.render(st.items)
        return [_image(st, it["view"], _abi.ACCUM_RUNNING_MEAN, it["width"], it["height"]) for it in st.items]
    if kind == "load":
        with api.Renderer() as r:
            r.upload(st.scene)
            r.render(0, 1)
            return r.read()
    lib = _abi.library()
    b, h, w = case["batch"], case["height"], case["width"]
    if kind == "denoise":
        _abi.check(lib.agb_denoiser_forward(st.denoiser.handle, st.x.data_ptr(), b, h, w, st.out.data_ptr()))
        return st.out
    if kind == "train":
        loss = ctypes.c_float()
        _abi.check(lib.agb_denoiser_train_step(st.denoiser.handle, st.x.data_ptr(), st.target.data_ptr(), b, h, w,
                                               1e-4, 1, ctypes.byref(loss)))
        _abi.check(lib.agb_denoiser_grads(st.denoiser.handle, st.grads.ctypes.data, st.grads.size))
        return [loss.value, st.grads]
    x1 = st.x1.data_ptr() if st.x1 is not None else None
    if kind == "conv":
        _abi.check(lib.agb_conv3x3_bf16(st.x0.data_ptr(), x1, st.wpack.data_ptr(), st.bias.data_ptr(),
                                        st.out.data_ptr(), None, b, h, w, case["c0"], case["c1"], case["cout"],
                                        1 if case["up"] else 0, 1 if case["relu"] else 0, None))
        return st.out
    st.dw.zero_()
    _abi.check(lib.agb_conv3x3_wgrad_bf16(st.x0.data_ptr(), x1, st.dy.data_ptr(), st.dw.data_ptr(), b, h, w,
                                          case["c0"], case["c1"], case["cout"], 1 if case["up"] else 0, None))
    return st.dw


# ------------------------------------------------------------------- what a pass cannot do without


def _trace_work(case, paths):
    """Paths through a binary BVH: per path about 1.7 segments (most rays leave the scene within
    one or two hits), each a closest-hit and, on a hit, two shadow rays; a ray visits about twice
    the tree's depth in nodes (two boxes, about 40 operations each) and a few triangles (60); a hit
    is shaded by three BSDF evaluations of about 500 operations."""
    tris = 20 * 4 ** case["level"] if case.get("scene") == "large" else 1000
    visits = 2.0 * math.log2(tris)
    ray = visits * 40.0 + 4 * 60.0
    return paths * (1.7 * ray + 0.7 * (2 * ray + 1500.0) + 200.0)


def _scene_bytes(case):
    tris = {"large": 20 * 4 ** max(1, case["level"]), "layered": 40_000}.get(case["scene"], 1_000)
    env = 32.0 * (case.get("env_width") or (2048 >> (8 - case["level"]))) * \
        (case.get("env_height") or (1024 >> (8 - case["level"]))) if case["scene"] == "large" else 0.0
    return tris * (48.0 + 32.0 + 16.0 + 12.0) + env


def work(case):
    kind = case["kind"]
    if kind == "render":
        px = case["width"] * case["height"]
        return dict(bytes=_scene_bytes(case) + px * 48.0, flops=_trace_work(case, px * case["spp"]))
    if kind == "viewer":
        px = case["width"] * case["height"]
        # Per frame: the sample, AOVs and history in, the resolved and 8-bit images out.
        return dict(bytes=case["frames"] * px * (16.0 + 36.0 + 16.0 + 16.0 + 4.0),
                    flops=case["frames"] * (_trace_work(case, px) + px * 400.0))
    if kind == "batch":
        px = sum(w * h for _, w, h, _ in _requests(case))
        paths = sum(w * h * n for _, w, h, n in _requests(case))
        return dict(bytes=_scene_bytes(dict(case, scene="large")) + px * 16.0,
                    flops=_trace_work(dict(case, scene="large"), paths))
    if kind == "load":
        px = case["width"] * case["height"]
        tris = _scene_bytes(case)
        # The scene in from the host and out as device records, the table, the image back.
        return dict(bytes=2.0 * tris + px * 16.0, flops=_trace_work(case, px) + tris * 10.0)
    if kind in ("denoise", "train"):
        px = case["batch"] * case["height"] * case["width"]
        fl = sum(2.0 * 9 * cin * cout / 4 ** level for cin, cout, level in _layer_shapes())
        act = sum(cout / 4 ** level for _, cout, level in _layer_shapes()) * 2.0
        if kind == "denoise":
            return dict(bytes=px * (32.0 + 16.0), flops=px * fl)
        # Activations written forward and read backward, gradients of all parameters out.
        n = sum(9 * cin * cout + cout for cin, cout, _ in _layer_shapes())
        return dict(bytes=px * (32.0 + 16.0 + 2.0 * act) + n * 4.0 * 7, flops=3.0 * px * fl)
    px = case["batch"] * case["height"] * case["width"]
    cin = case["c0"] + case["c1"]
    read = px * 2.0 * (case["c0"] / (4.0 if case["up"] else 1.0) + case["c1"])
    weights = 9.0 * cin * case["cout"]
    flops = 18.0 * cin * case["cout"] * px
    return dict(bytes=read + px * 2.0 * case["cout"] + weights * (2.0 if kind == "conv" else 4.0), flops=flops)


# ------------------------------------------------------------------------------- in 64 bits


def _taps(wt):
    """w[tap][ci][co] -> conv2d weights [co][ci][3][3] in 64 bits."""
    return wt.double().reshape(3, 3, wt.shape[1], wt.shape[2]).permute(3, 2, 0, 1).contiguous()


def _layer_input64(x0, x1, up):
    x = x0.double().permute(0, 3, 1, 2)
    if up:
        x = x.repeat_interleave(2, 2).repeat_interleave(2, 3)
    if x1 is not None:
        x = torch.cat([x, x1.double().permute(0, 3, 1, 2)], 1)
    return x


def _network64(p, x):
    """The network on features x (B, H, W, 16) with parameters p, in 64 bits; (B, H, W, 3) added to
    the features' log radiance."""
    acts = {"x": x.double().permute(0, 3, 1, 2)}
    off = 0
    for (src, dst, _, _), (cin, cout, _) in zip(_LAYERS, _layer_shapes()):
        wt = p[off:off + 9 * cin * cout].reshape(9, cin, cout)
        off += 9 * cin * cout
        bias = p[off:off + cout]
        off += cout
        if isinstance(src, tuple):
            a = acts[src[0]].repeat_interleave(2, 2).repeat_interleave(2, 3)
            a = torch.cat([a, acts[src[1]]], 1)
        elif src[0] == "p":
            a = F.avg_pool2d(acts["s" + src[1:]], 2)
        else:
            a = acts[src]
        y = F.conv2d(a, _taps(wt), bias.double(), padding=1)
        acts[dst] = y if dst == "out" else torch.relu(y)
    return (acts["out"] + acts["x"])[:, :3].permute(0, 2, 3, 1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("render", "viewer", "batch", "load"):
        return None  # a path's branches follow 32-bit comparisons: no plain 64-bit restatement is quick
    if kind == "denoise":
        x = _features(case["batch"], case["height"], case["width"], seed)
        with torch.no_grad():
            y = _network64(_params(seed).cuda(), x)
            return torch.cat([torch.expm1(y).clamp(min=0.0), torch.ones_like(y[..., :1])], -1)
    if kind == "train":
        x = _features(case["batch"], case["height"], case["width"], seed)
        t = torch.log1p(_target(x, seed)[..., :3].double().clamp(min=0.0))
        p = _params(seed).cuda().double().requires_grad_(True)
        loss = (_network64(p, x) - t).abs().mean()
        (g,) = torch.autograd.grad(loss, p)
        return [float(loss), g]
    x0, x1, dy, wt, bias = _layer_tensors(case, seed)
    x = _layer_input64(x0, x1, case["up"])
    if kind == "conv":
        y = F.conv2d(x, _taps(wt.to(torch.bfloat16)), bias.double(), padding=1)
        return (torch.relu(y) if case["relu"] else y).permute(0, 2, 3, 1).contiguous()
    xp = F.pad(x, (1, 1, 1, 1))
    d = dy.double().permute(0, 3, 1, 2).reshape(case["batch"], case["cout"], -1)
    h, w = case["height"], case["width"]
    out = []
    for ky in range(3):
        for kx in range(3):
            a = xp[:, :, ky:ky + h, kx:kx + w].reshape(case["batch"], x.shape[1], -1)
            out.append(torch.einsum("bip,bop->io", a, d))
    return torch.stack(out)
