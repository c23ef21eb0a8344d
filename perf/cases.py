"""Performance cases of the reconstruction path: the calls a camera program makes, over the range
of frame sizes, window lengths, formats and options it makes them with.

A case names its `kind`:
  windows  Pipeline.run on a device ring: frames to M0/M1/M2 images (both numeric forms, Fresnel or
           angular spectrum, with or without the clutter filter and the autofocus)
  live     CameraStream.push + process, one window for every `hop` new frames
  multi    Multi.exec: several uneven acquisitions in one graph launch
  graph    the reference's operators node by node: RFFT -> Slice -> Copy -> Fresnel -> Mean
  display  a moment image to an 8-bit picture: fftshift -> flat field -> percentile clip -> U8
"""
from __future__ import annotations

import math

import numpy as np
import torch

import holoflow_b200 as hf
from holoflow_b200 import nodes
from holoflow_b200 import pipeline as pl
from holoflow_b200 import synth
from holoflow_b200.multi import Multi

LAM, PITCH = 852e-9, 12e-6
DTYPES = {"u8": hf.HF_U8, "u16": hf.HF_U16, "mono12p": hf.HF_MONO12P, "f32": hf.HF_F32}
SAMPLE_BYTES = {"u8": 1.0, "u16": 2.0, "mono12p": 1.5, "f32": 4.0}
PROPAGATION = {"fresnel": hf.HF_PROP_FRESNEL, "angular": hf.HF_PROP_ANGULAR_SPECTRUM}
AF_ORDERS = (4, 5, 6)


def _windows(name, height, width, frames, hop, windows, z_begin, z_end, dtype="mono12p", form=0, rank=4, fs=67e3,
             z=0.25, propagation="fresnel", two_sided=False, pad_h=0, pad_w=0, r_outer=0, subaps=0, kind="windows"):
    c = dict(kind=kind, height=height, width=width, frames=frames, hop=hop, windows=windows, z_begin=z_begin,
             z_end=z_end, dtype=dtype, form=form, rank=rank, fs=fs, z=z, propagation=propagation,
             two_sided=two_sided, pad_h=pad_h, pad_w=pad_w, r_outer=r_outer, subaps=subaps)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # the smallest call: one preview window of a small 8-bit camera, default (plain) form
        _windows("preview_256_u8", 256, 256, 32, 32, 1, 6, 16, dtype="u8", rank=0, fs=37e3, z=0.3),
        # 16-bit camera, angular spectrum, one non-overlapping window per call
        _windows("angular_512_u16", 512, 512, 32, 32, 1, 6, 16, dtype="u16", rank=0, fs=37e3, z=0.3,
                 propagation="angular"),
        # full-size frames, clutter filter, overlapping windows: the all-FP32 form
        _windows("fresnel_1024_plain", 1024, 1024, 64, 16, 8, 4, 32),
        # the same windows in the tensor-core form: offline reconstruction of a recording
        _windows("fresnel_1024_chosen", 1024, 1024, 64, 16, 8, 4, 32, form=1),
        # live view: every 16 new frames one window, images wanted at once
        _windows("live_1024_chosen", 1024, 1024, 64, 16, 4, 4, 32, form=1, kind="live"),
        # the largest frames and the longest window in use
        _windows("wide_1536_t128_chosen", 1024, 1536, 128, 32, 4, 8, 64, form=1),
        # angular spectrum into a padded plane with the annular band-pass filter
        _windows("angular_768_padded", 768, 768, 64, 16, 4, 4, 32, form=1, propagation="angular", pad_h=1024,
                 pad_w=1024, r_outer=300),
        # an eye moves: Shack-Hartmann autofocus on every window
        _windows("autofocus_1024", 1024, 1024, 64, 16, 4, 4, 32, form=1, subaps=5),
        # a camera whose sides are no power of two (SVGA), 16-bit samples
        _windows("camera_600x800_u16", 600, 800, 32, 16, 2, 6, 16, dtype="u16", rank=2, fs=37e3, z=0.3),
        # a recording session: uneven acquisitions reconstructed together
        dict(name="multi_uneven_6", kind="multi", count=6, pick=3, form=1, rank=4),
        # the operator API, one node after the other, on float frames
        dict(name="graph_512", kind="graph", height=512, width=512, frames=32, batch=2, z_begin=6, z_end=16, z=0.3),
        # what the viewer does with every image
        dict(name="display_1024", kind="display", depth=1, height=1024, width=1024, sigma=4.0, min_pct=0.5,
             max_pct=99.5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _band(rng, frames, most):
    """A band of the one-sided spectrum, odd widths among them."""
    width = rng.randint(max(2, frames // 8), min(most, (7 * frames) // 16))
    z0 = rng.randint(1, frames // 2 - width)
    return z0, z0 + width


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["plain", "chosen", "chosen", "live", "angular", "autofocus", "ragged", "multi", "graph",
                       "display"])
    sides = [256, 512, 768, 1024]
    fs, z = rng.choice([37e3, 67e3]), round(rng.uniform(0.15, 0.40), 4)
    if kind in ("plain", "chosen", "live"):
        h, w = rng.choice(sides), rng.choice(sides + [1536])
        frames = rng.choice([32, 64, 64, 128])
        z0, z1 = _band(rng, frames, 56)
        two = kind == "chosen" and rng.random() < 0.25 and z1 - z0 <= 32
        hop = rng.choice([frames // 4, frames // 2, frames])
        n = frames // hop if kind == "live" else rng.randint(1, 4 if frames == 128 or kind == "plain" else 8)
        dtype = rng.choice(["mono12p", "mono12p", "u16", "u8"])
        return _windows(None, h, w, frames, hop, n, z0, z1, dtype=dtype, form=0 if kind == "plain" else 1,
                        rank=rng.choice([0, 2, 4]), fs=fs, z=z, two_sided=two,
                        kind="live" if kind == "live" else "windows")
    if kind == "angular":
        h, w = rng.choice(sides), rng.choice(sides)
        pad = rng.random() < 0.5
        frames = rng.choice([32, 64])
        z0, z1 = _band(rng, frames, 28)
        return _windows(None, h, w, frames, rng.choice([frames // 2, frames]), rng.randint(1, 4), z0, z1,
                        dtype=rng.choice(["mono12p", "u16"]), form=rng.choice([0, 1]), rank=rng.choice([0, 4]), fs=fs,
                        z=z, propagation="angular", pad_h=1024 if pad else 0, pad_w=1024 if pad else 0,
                        r_outer=rng.choice([0, 120]))
    if kind == "autofocus":
        h = rng.choice([512, 768, 1024])
        z0, z1 = _band(rng, 64, 28)
        return _windows(None, h, h, 64, rng.choice([16, 32]), rng.randint(1, 4), z0, z1, form=1, fs=fs, z=z,
                        subaps=rng.choice([3, 5, 7]))
    if kind == "ragged":
        h, w = _log_int(rng, 90, 640), _log_int(rng, 90, 800)
        frames = rng.choice([16, 32, 32, 50, 64])
        z0, z1 = _band(rng, frames, 12)
        dtype = rng.choice(["u8", "u16"])
        return _windows(None, h, w, frames, max(1, frames // 2), rng.randint(1, 2), z0, z1, dtype=dtype, form=0,
                        rank=rng.choice([0, 2]), fs=fs, z=z)
    if kind == "multi":
        return dict(kind="multi", count=rng.randint(3, 6), pick=rng.randint(4, 1 << 20), form=1,
                    rank=rng.choice([2, 4]))
    if kind == "graph":
        h, w = rng.choice([256, 512, 768]), rng.choice([256, 512, 768])
        frames = rng.choice([16, 32, 64])
        z0, z1 = _band(rng, frames, 16)
        return dict(kind="graph", height=h, width=w, frames=frames, batch=rng.randint(1, 3), z_begin=z0, z_end=z1, z=z)
    return dict(kind="display", depth=rng.randint(1, 3), height=_log_int(rng, 150, 1536),
                width=_log_int(rng, 150, 1536), sigma=round(rng.uniform(1.5, 9.0), 2), min_pct=0.5, max_pct=99.5)


# ---- inputs ------------------------------------------------------------------------------------

def _seed(case, seed):
    return 1000 + seed % 1000003


def _frames(case, seed, n, sub=0):
    """n seeded off-axis interferograms [n, H, W] of 12-bit values (int16)."""
    h, w = case["height"], case["width"]
    scene = synth.Scene(h, w, case.get("fs", 37e3), int(round(0.85 * min(h, w))), case["z"],
                        seed=_seed(case, seed) + 17 * sub)
    return synth.DeviceInterferograms(scene).frames(0, n)


def _samples(f, dtype):
    """The camera's bytes of 12-bit frames."""
    if dtype == "u8":
        return (f >> 4).to(torch.uint8)
    if dtype == "mono12p":
        return pl.pack12(f.reshape(-1))
    return f.to(torch.float32) if dtype == "f32" else f


def _config(c, max_batch):
    extra = {}
    if c["propagation"] == "angular":
        extra = dict(pad_w=c["pad_w"], pad_h=c["pad_h"])
        if c["r_outer"]:
            extra |= dict(as_filter=1, r_inner=4, r_outer=c["r_outer"], s_inner=3, s_outer=20)
    if c["subaps"]:
        extra |= dict(autofocus_nb_subaps=c["subaps"], autofocus_orders=AF_ORDERS)
    return pl.PipelineConfig(height=c["height"], width=c["width"], frames=c["frames"], hop=c["hop"],
                             z_begin=c["z_begin"], z_end=c["z_end"], input_dtype=DTYPES[c["dtype"]],
                             propagation=PROPAGATION[c["propagation"]], clutter_rank=c["rank"], form=c["form"],
                             max_batch=max_batch, lam=LAM, pitch=PITCH, z=c["z"], fs=c["fs"],
                             time_method=hf.HF_TIME_FFT if c["two_sided"] else hf.HF_TIME_RFFT, **extra)


def _acquisitions(case):
    """The window cases of a multi-acquisition launch."""
    out = []
    for a in synth.config3_acquisitions(case["count"], seed=1000 + case["pick"]):
        out.append(_windows(None, a.scene.height, a.scene.width, a.frames, a.hop, 1, a.z_begin, a.z_end,
                            form=case["form"], rank=case["rank"], fs=a.scene.fs, z=round(a.z, 4)))
    return out


def _n_frames(c):
    return c["frames"] if c["kind"] == "live" else c["frames"] + (c["windows"] - 1) * c["hop"]


# ---- the calls ---------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "windows":
        n = _n_frames(case)
        ring = _samples(_frames(case, seed, n), case["dtype"])
        return dict(kind=kind, pipe=pl.Pipeline(_config(case, case["windows"])), ring=ring, frames=n,
                    windows=case["windows"], subaps=case["subaps"])
    if kind == "live":
        # a cycle of `frames` frames: every pass pushes one cycle and so sees the same windows
        T, hop = case["frames"], case["hop"]
        pool = _samples(_frames(case, seed, T), case["dtype"])
        pool = pool.view(torch.uint8).reshape(T, -1)
        pipe = pl.Pipeline(_config(case, 1))
        cam = pl.CameraStream(pipe, 2 * T)
        if hop < T:
            cam.push(pool[hop:], T - hop)
        out = torch.empty((case["windows"], *pipe.out_shape), dtype=torch.float32, device="cuda")
        return dict(kind=kind, pipe=pipe, cam=cam, pool=pool, hop=hop, out=out)
    if kind == "multi":
        acqs = _acquisitions(case)
        rings, frames, outs = [], [], []
        for i, c in enumerate(acqs):
            frames.append(_n_frames(c))
            rings.append(_samples(_frames(c, seed, frames[-1], i), c["dtype"]))
            outs.append(torch.empty((1, 3, c["height"], c["width"]), dtype=torch.float32, device="cuda"))
        m = Multi([_config(c, 1) for c in acqs])
        m.set_schedule(branches=4, largest_first=1, fused=1)
        return dict(kind=kind, multi=m, rings=rings, frames=frames, outs=outs)
    if kind == "graph":
        b, T, h, w = case["batch"], case["frames"], case["height"], case["width"]
        x = _frames(case, seed, b * T).to(torch.float32).reshape(b, T, h, w)
        steps = [("RFFT", {"axis": 1}),
                 ("Slice", {"slices": [{}, {"start": case["z_begin"], "stop": case["z_end"]}, {}, {}]}),
                 ("Copy", {}),
                 ("FresnelDiffraction", {"lambda": LAM, "dx": PITCH, "dy": PITCH, "z": case["z"],
                                         "output_magnitude": True, "skip_phase_shift": True}),
                 ("Mean", {"axis": [-3], "keepdims": True})]
        return dict(kind=kind, **_node_chain(steps, x))
    shape = (case["depth"], case["height"], case["width"])
    c = dict(height=case["height"], width=case["width"], z=0.25)
    x = torch.stack([torch.fft.fft2(_frames(c, seed, 1, i)[0].to(torch.float32) - 2048.0).abs().sqrt()
                     for i in range(case["depth"])]).contiguous()
    assert tuple(x.shape) == shape
    roi = {"cx": 0.5, "cy": 0.5, "rx": 0.5, "ry": 0.5, "angle": 0.0}
    steps = [("FFTShiftNp", {"axes": [-2, -1]}),
             ("Flatfield", {"sigma_y": case["sigma"], "sigma_x": case["sigma"]}),
             ("PctClip", {"min_pct": case["min_pct"], "max_pct": case["max_pct"], "roi": roi}),
             ("Conversion", {"target": "U8", "strategy": "Scaled"})]
    return dict(kind=kind, **_node_chain(steps, x))


_TORCH = {hf.HF_U8: torch.uint8, hf.HF_U16: torch.int16, hf.HF_F32: torch.float32, hf.HF_CF32: torch.complex64}


def _node_chain(steps, x):
    """The nodes of a chain and their output tensors; a view node (Slice) owns none."""
    chain, outs, d = [], [], nodes.desc_of(x)
    for kind, settings in steps:
        (o,) = nodes.infer(kind, settings, [d])
        node = nodes.Node(kind, settings, [d])
        view = node.alias(0) >= 0
        out = None if view else torch.empty(nodes.shape_of(o), dtype=_TORCH[o.dtype], device="cuda")
        chain.append(node)
        outs.append(out)
        d = o if view else nodes.desc_of(out)
    return dict(chain=chain, outs=outs, x=x)


def run(state):
    kind = state["kind"]
    if kind == "windows":
        images = state["pipe"].run(state["ring"], state["frames"], 0, state["windows"])
        if not state["subaps"]:
            return {"images": images}
        return {"images": images,
                "zernike": [state["pipe"].autofocus_coefficients(w) for w in range(state["windows"])]}
    if kind == "live":
        cam, pool, hop, out = state["cam"], state["pool"], state["hop"], state["out"]
        for w in range(out.shape[0]):
            cam.push(pool[w * hop:(w + 1) * hop], hop)
            cam.process(1, out[w:w + 1])
        return {"images": out}
    if kind == "multi":
        state["multi"].exec(state["rings"], state["frames"], [0] * len(state["rings"]), state["outs"])
        return {"images": state["outs"]}
    at = state["x"]
    for node, out in zip(state["chain"], state["outs"]):
        node.execute([at], [out])
        at = node.output_ptr(0)[0] if out is None else out
    if kind == "graph":
        return {"magnitude": state["outs"][3], "m0": state["outs"][4]}
    return {"flat": state["outs"][1], "clipped": state["outs"][2], "picture": state["outs"][3]}


# ---- what a pass cannot do without -------------------------------------------------------------

def _window_work(c):
    P, T, n = c["height"] * c["width"], c["frames"], c["windows"]
    nz = (c["z_end"] - c["z_begin"]) * (2 if c["two_sided"] else 1)
    oh, ow = c["pad_h"] or c["height"], c["pad_w"] or c["width"]
    frames_in = n * c["hop"] if c["kind"] == "live" else _n_frames(c)
    nbytes = frames_in * P * SAMPLE_BYTES[c["dtype"]] + n * 12 * oh * ow
    fft = nz * 5 * oh * ow * math.log2(oh * ow) * (2 if c["propagation"] == "angular" else 1)
    if c["subaps"]:
        fft += nz * 5 * P * math.log2(P / c["subaps"] ** 2)
    return {"bytes": nbytes, "flops": n * ((P * T * (T + 1) if c["rank"] else 0) + 4 * P * T * nz + fft + 8 * nz * P)}


def work(case):
    kind = case["kind"]
    if kind in ("windows", "live"):
        return _window_work(case)
    if kind == "multi":
        parts = [_window_work(c) for c in _acquisitions(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "graph":
        P, b, T, nz = case["height"] * case["width"], case["batch"], case["frames"], case["z_end"] - case["z_begin"]
        return {"bytes": 4 * P * b * (T + nz + 1),
                "flops": b * (4 * P * T * nz + nz * P * (6 + 5 * math.log2(P)) + 2 * nz * P)}
    n = case["depth"] * case["height"] * case["width"]
    return {"bytes": n * (4 + 4 + 4 + 1), "flops": n * 4 * (2 * math.ceil(3 * case["sigma"]) + 1)}


# ---- the same in 64 bits -----------------------------------------------------------------------

F32 = np.float32
PI32 = F32(np.pi)


def _cis(phase):
    p = torch.from_numpy(np.ascontiguousarray(phase.astype(np.float64))).cuda()
    return torch.polar(torch.ones_like(p), p)


def _lens(h, w, z):
    """The quadratic lens exp(i phase); the phase itself is defined in float32."""
    size = max(h, w)
    x = ((np.arange(w) + (size - w) // 2).astype(F32) - F32(size / 2.0)) * F32(PITCH)
    y = ((np.arange(h) + (size - h) // 2).astype(F32) - F32(size / 2.0)) * F32(PITCH)
    k = PI32 / (F32(LAM) * F32(z))
    return _cis((k * ((x * x)[None, :] + (y * y)[:, None])).astype(F32))


def _transfer(h, w, z, r_outer):
    """The angular spectrum's transfer function in natural frequency order, phase in float32."""
    u = (np.arange(w) - w // 2).astype(F32) * (F32(1.0) / F32(F32(w) * F32(PITCH)))
    v = (np.arange(h) - h // 2).astype(F32) * (F32(1.0) / F32(F32(h) * F32(PITCH)))
    tmp = F32(1.0) - F32(F32(LAM) * F32(LAM)) * ((u * u)[None, :] + (v * v)[:, None])
    k = F32(F32(F32(2.0) * PI32) * F32(z)) / F32(LAM)
    tf = _cis((k * np.sqrt(np.maximum(tmp, F32(0.0)))).astype(F32))
    if r_outer:
        dist = np.hypot(np.arange(w)[None, :] - w / 2.0, np.arange(h)[:, None] - h / 2.0)
        ri, ro, si, so = 4.0, float(r_outer), 3.0, 20.0
        rise = 0.5 * (1 + np.sin(np.pi / (2 * si) * (dist - (ri - si))))
        fall = 0.5 * (1 + np.sin(np.pi / (2 * so) * (ro + so - dist)))
        val = np.where(dist < ri - si, 0.0, np.where(dist < ri + si, rise, np.where(
            dist < ro - so, 1.0, np.where(dist < ro + so, fall, 0.0))))
        tf = tf * torch.from_numpy(val * val).cuda()
    return torch.fft.ifftshift(tf)


def _exact_window(c, x):
    """M0/M1/M2 of one window x [T, H, W] float64."""
    T, h, w = x.shape
    bins = list(range(c["z_begin"], c["z_end"]))
    df = c["fs"] / T
    freqs = [k * df for k in bins]
    if c["two_sided"]:
        freqs += [k * df - c["fs"] for k in bins]
        bins += list(range(T - c["z_end"], T - c["z_begin"]))
    t = torch.arange(T, dtype=torch.float64, device="cuda")
    arg = -2 * math.pi * torch.remainder(t[:, None] * torch.tensor(bins, dtype=torch.float64, device="cuda"), T) / T
    D = torch.polar(torch.ones_like(arg), arg)
    X = x.reshape(T, -1)
    if c["rank"]:
        V = torch.linalg.eigh(X @ X.T)[1][:, T - c["rank"]:]
        D = D - (V @ (V.T @ D.real)) - 1j * (V @ (V.T @ D.imag))
    S = torch.complex(D.real.T.contiguous() @ X, D.imag.T.contiguous() @ X).reshape(-1, h, w)
    oh, ow = c["pad_h"] or h, c["pad_w"] or w
    if c["propagation"] == "fresnel":
        lens = _lens(h, w, c["z"])
        mags = (torch.fft.fft2(s * lens).abs() for s in S)
    else:
        tf = _transfer(oh, ow, c["z"], c["r_outer"])
        pad = ((ow - w) // 2, (ow - w) // 2, (oh - h) // 2, (oh - h) // 2)
        mags = (torch.fft.ifft2(torch.fft.fft2(torch.nn.functional.pad(s, pad)) * tf, norm="forward").abs() for s in S)
    m = torch.zeros((3, oh, ow), dtype=torch.float64, device="cuda")
    for f, a in zip(freqs, mags):
        f1 = F32(f)
        m += torch.stack([a, float(f1) * a, float(F32(f1 * f1)) * a])
    return m / len(freqs)


def _values(c, f):
    return (f >> 4 if c["dtype"] == "u8" else f).to(torch.float64)


def exact(case, seed):
    kind = case["kind"]
    if kind == "windows":
        if case["subaps"]:
            return None
        f = _frames(case, seed, _n_frames(case))
        hop, T = case["hop"], case["frames"]
        return {"images": torch.stack([_exact_window(case, _values(case, f[w * hop:w * hop + T]))
                                       for w in range(case["windows"])])}
    if kind == "live":
        f = _frames(case, seed, case["frames"])
        return {"images": torch.stack([_exact_window(case, _values(case, torch.roll(f, -(w + 1) * case["hop"], 0)))
                                       for w in range(case["windows"])])}
    if kind == "multi":
        return {"images": [_exact_window(c, _values(c, _frames(c, seed, _n_frames(c), i)))[None]
                           for i, c in enumerate(_acquisitions(case))]}
    if kind == "graph":
        b, T, h, w = case["batch"], case["frames"], case["height"], case["width"]
        x = _frames(case, seed, b * T).to(torch.float64).reshape(b, T, h, w)
        S = torch.fft.rfft(x, dim=1)[:, case["z_begin"]:case["z_end"]]
        mag = torch.fft.fft2(S * _lens(h, w, case["z"])).abs()
        return {"magnitude": mag, "m0": mag.mean(dim=1, keepdim=True)}
    # display: the flat field x - G x (clamped borders); the clip bounds and the 8-bit picture follow
    # from its float32 values
    c = dict(height=case["height"], width=case["width"], z=0.25)
    x = torch.stack([torch.fft.fft2(_frames(c, seed, 1, i)[0].to(torch.float32) - 2048.0).abs().sqrt()
                     for i in range(case["depth"])]).double()
    x = torch.roll(x, (-(case["height"] // 2), -(case["width"] // 2)), (1, 2))
    r = int(math.ceil(float(F32(3.0) * F32(case["sigma"]))))
    i = torch.arange(-r, r + 1, dtype=torch.float64, device="cuda")
    g = torch.exp(-(i * i) / (2.0 * case["sigma"] ** 2))
    g = g / g.sum()
    b = x
    for dim in (2, 1):
        n = b.shape[dim]
        at = torch.clamp(torch.arange(n, device="cuda")[:, None] + i.long()[None, :], 0, n - 1)
        b = torch.stack([b.index_select(dim, at[:, k]) * g[k] for k in range(2 * r + 1)]).sum(0)
    return {"flat": x - b, "clipped": None, "picture": None}
