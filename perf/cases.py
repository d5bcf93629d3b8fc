"""The work that programs have this framework do, as cases that can be timed.

A case is one call, or one short sequence of calls, of a public entry point
with the inputs such a program holds: `Synthesizer` (a style exemplar and
frames resident on the device, one still or a clip synthesised), `TexSynth`
(the step-wise interface a host application drives itself), `Server` (many
requests at once) and the separable Gaussian.  Sizes and settings are those
of the configurations in painttween_gb300/synthetic.py, of the tests and of
bench.py, and odd ones between them.  Inputs follow the generators of
painttween_gb300/synthetic.py (oriented strokes; flat-shaded discs in rigid
motion with analytic velocities), made on the GPU from the seed.
"""
import ctypes
import math
import random

import numpy as np
import torch

from painttween_gb300 import Synthesizer, TexSynth, _abi, host_array, serving
from painttween_gb300._lib import lib

SCHEMES = {"FMBM": _abi.S_FMBM, "FMBM_RM": _abi.S_FMBM_RM, "FBMO": _abi.S_FBMO, "TCTF": _abi.S_TCTF,
           "IND": _abi.S_IND}
STILL = dict(kind="clip", frames=1, discs=3, radius=2, levels=3, iterations=4)


def listed():
    return [
        # the smallest still of a batch: a preview or a thumbnail, where launches and latency count
        dict(STILL, name="still 128", w=128, h=128, ew=256, eh=256),
        # an odd-sized still with an exemplar that is not square and every static energy term in use
        dict(STILL, name="still ragged terms", w=333, h=517, ew=411, eh=290, radius=3, levels=4, terms=True),
        # the largest still of a batch
        dict(STILL, name="still 1024", w=1024, h=1024, ew=1024, eh=1024),
        # two brush styles whose strokes leave parts of the exemplar unpainted, at the default settings
        # (patch radius 4, 4 levels, 3 iterations)
        dict(STILL, name="still two styles holes", w=192, h=160, ew=256, eh=256, styles=2, holes=True, radius=4,
             levels=4, iterations=3),
        # an animation in its usual form: forward and backward passes with temporal coherence
        dict(kind="clip", name="clip 512", w=512, h=512, ew=512, eh=512, frames=4, discs=3, radius=2, levels=4,
             iterations=4, coherence=0.5),
        # the headline workload, cut to two frames: a full-HD clip with the histogram term
        dict(kind="clip", name="clip 1080p", w=1920, h=1080, ew=1024, eh=1024, frames=2, discs=6, radius=3, levels=5,
             iterations=6, histogram=True),
        # a clip at the default settings with exact FP32 filtering in place of the texture unit's
        dict(kind="clip", name="clip 640x360 exact", w=640, h=360, ew=512, eh=512, frames=2, discs=4, radius=4,
             levels=4, iterations=3, exact_filter=True),
        # the scheme that ends with passes between both advected neighbours (forward and backward terms at once)
        dict(kind="clip", name="clip both neighbours", w=240, h=180, ew=256, eh=256, frames=3, discs=3, radius=3,
             levels=3, iterations=3, scheme="FBMO", coherence=0.5),
        # keyframe interpolation: two painted keys of the image's size, the frames between them filled in
        dict(kind="clip", name="keys 160x120", w=160, h=120, ew=160, eh=120, frames=4, discs=3, radius=2, levels=3,
             iterations=2, styles=2, keys=True),
        # a host application driving one level itself through the step-wise interface
        dict(kind="steps", name="steps 480x270", w=480, h=270, ew=512, eh=512, discs=4, radius=3, iterations=2),
        # requests of uneven sizes, all at once, from host memory to host memory
        dict(kind="serve", name="serve 8 stills", requests=8, low=128, high=768, in_flight=8),
        # the separable Gaussian on a full-HD plane
        dict(kind="blur", name="blur 1080p", w=1920, h=1080, pitch=1920, radius=7),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["still", "still", "still", "clip", "clip", "scheme", "keys", "steps", "serve", "blur"])
    if what == "still":
        c = dict(STILL, w=_log(rng, 128, 1024), h=_log(rng, 128, 1024), ew=_log(rng, 256, 1024),
                 eh=_log(rng, 256, 1024), radius=rng.choice([2, 2, 3, 4]), levels=rng.choice([3, 4]),
                 iterations=rng.choice([3, 4]))
        if rng.random() < 0.3:
            c["terms"] = True
        if rng.random() < 0.2:
            c["exact_filter"] = True
        return c
    if what == "clip":
        return dict(kind="clip", w=_log(rng, 192, 1280), h=_log(rng, 192, 720), ew=_log(rng, 256, 1024),
                    eh=_log(rng, 256, 1024), frames=rng.randint(2, 3), discs=rng.randint(2, 6),
                    radius=rng.choice([2, 3]), levels=4, iterations=rng.choice([3, 4]),
                    coherence=rng.choice([0.2, 0.5]), scheme=rng.choice(["FMBM", "FMBM_RM", "FMBM_RM"]),
                    exact_filter=rng.random() < 0.2)
    if what == "scheme":
        return dict(kind="clip", w=_log(rng, 96, 190), h=_log(rng, 96, 170), ew=_log(rng, 128, 384),
                    eh=_log(rng, 128, 384), frames=rng.randint(2, 3), discs=3, radius=rng.choice([2, 3]), levels=3,
                    iterations=rng.randint(2, 3), coherence=0.5, scheme=rng.choice(["FBMO", "TCTF", "IND"]))
    if what == "keys":
        w, h = _log(rng, 64, 160), _log(rng, 64, 110)
        return dict(kind="clip", w=w, h=h, ew=w, eh=h, frames=rng.randint(3, 4), discs=3, radius=2, levels=2,
                    iterations=2, styles=2, keys=True)
    if what == "steps":
        return dict(kind="steps", w=_log(rng, 96, 640), h=_log(rng, 96, 640), ew=_log(rng, 256, 768),
                    eh=_log(rng, 256, 768), discs=4, radius=rng.choice([2, 3, 4]), iterations=rng.randint(1, 2))
    if what == "serve":
        return dict(kind="serve", requests=rng.randint(3, 8), low=128, high=_log(rng, 256, 768),
                    in_flight=rng.choice([2, 4, 8]))
    w = _log(rng, 64, 2048)
    return dict(kind="blur", w=w, h=_log(rng, 64, 1100), pitch=w + rng.choice([0, 0, 3, 64]),
                radius=rng.randint(1, 15))


# --- inputs -------------------------------------------------------------------

def _dev(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _grid(w, h):
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                            torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    return xx, yy


def _lum(rgb):
    return 0.2126 * rgb[..., 0] + 0.7152 * rgb[..., 1] + 0.0722 * rgb[..., 2]


def _exemplar(w, h, seed, holes=False, terms=False):
    """Oriented sinusoidal strokes and noise (synthetic.make_exemplar's
    distribution); holes: unpainted bands (alpha 0.2); terms: a distance
    transform other than zero."""
    rng, gen = random.Random(seed), _dev(seed)
    xx, yy = _grid(w, h)
    acc = torch.zeros((h, w, 3), device="cuda")
    best = torch.full((h, w), -1.0, device="cuda")
    dom = torch.zeros((h, w), device="cuda", dtype=torch.int32)
    phi_of = torch.zeros((h, w), device="cuda")
    for k in range(8):
        phi, period = rng.uniform(0.0, math.pi), rng.uniform(6.0, 20.0)
        amp, psi = rng.uniform(0.1, 0.3), rng.uniform(0.0, 2 * math.pi)
        tint = torch.tensor([rng.uniform(0.4, 1.0) for _ in range(3)], device="cuda")
        s = amp * torch.sin(2 * math.pi * (xx * math.cos(phi) + yy * math.sin(phi)) / period + psi)
        acc += s[..., None] * tint / 2.0
        sel = s.abs() > best
        best = torch.where(sel, s.abs(), best)
        dom = torch.where(sel, torch.full_like(dom, k), dom)
        phi_of = torch.where(sel, torch.full_like(phi_of, phi), phi_of)
    acc += 0.05 * torch.randn(acc.shape, generator=gen, device="cuda")
    out = torch.ones((h, w, 4), device="cuda")
    out[..., :3] = (acc + 0.5).clamp(0.0, 1.0)
    base = torch.ones_like(out)
    base[..., :3] = _lum(out)[..., None]
    if holes:
        bare = (torch.sin(0.11 * xx + rng.uniform(0, 6)) > 0.8)
        out[..., 3] = torch.where(bare, 0.2, 1.0)
        base[..., 3] = out[..., 3]
    c, s = torch.cos(phi_of), torch.sin(phi_of)
    dt = torch.rand((h, w), generator=gen, device="cuda") * 30.0 if terms else torch.zeros((h, w), device="cuda")
    return dict(base=_np(base), output=_np(out), orient_tensor=_np(torch.stack([c * c, c * s, s * s], -1)),
                dist_trans=_np(dt), object_ids=_np(dom % 4))


def _np(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _frames(w, h, discs, n, seed):
    """Flat-shaded discs on grey in rigid motion, with analytic velocities and
    the distance to the nearest disc edge (synthetic.make_clip's distribution)."""
    rng = random.Random(seed)
    m = min(w, h)
    ds = [dict(cx=rng.uniform(0.1 * w, 0.9 * w), cy=rng.uniform(0.1 * h, 0.9 * h), r=rng.uniform(0.08, 0.25) * m,
               color=[rng.random() for _ in range(3)], rot=math.radians(rng.uniform(-2, 2)), tx=rng.uniform(-4, 4),
               ty=rng.uniform(-4, 4), ident=1 + k % 3) for k in range(discs)]
    xx, yy = _grid(w, h)
    out = []
    for f in range(n):
        rgba = torch.full((h, w, 4), 0.5, device="cuda")
        rgba[..., 3] = 1.0
        ids = torch.zeros((h, w), device="cuda", dtype=torch.int32)
        vf = torch.zeros((h, w, 2), device="cuda")
        vb = torch.zeros((h, w, 2), device="cuda")
        dt = torch.full((h, w), 1e4, device="cuda")
        for d in ds:
            cx, cy = d["cx"] + f * d["tx"], d["cy"] + f * d["ty"]
            px, py = xx - cx, yy - cy
            dist = torch.sqrt(px * px + py * py)
            sel = (dist <= d["r"])[..., None]
            rgba[..., :3] = torch.where(sel, torch.tensor(d["color"], device="cuda"), rgba[..., :3])
            ids = torch.where(sel[..., 0], torch.full_like(ids, d["ident"]), ids)
            ca, sa = math.cos(d["rot"]), math.sin(d["rot"])
            fwd = torch.stack([ca * px - sa * py + d["tx"] - px, sa * px + ca * py + d["ty"] - py], -1)
            bwd = torch.stack([ca * px + sa * py - d["tx"] - px, -sa * px + ca * py - d["ty"] - py], -1)
            vf, vb = torch.where(sel, fwd, vf), torch.where(sel, bwd, vb)
            dt = torch.minimum(dt, (dist - d["r"]).abs())
        lum = _lum(rgba)
        gx, gy = torch.zeros_like(lum), torch.zeros_like(lum)
        gx[:, 1:-1] = 0.5 * (lum[:, 2:] - lum[:, :-2])
        gy[1:-1, :] = 0.5 * (lum[2:, :] - lum[:-2, :])
        out.append(dict(rgba=_np(rgba), orient_tensor=_np(torch.stack([gx * gx, gx * gy, gy * gy], -1)),
                        dist_trans=_np(dt), object_ids=_np(ids), vel_fwd=_np(vf), vel_bwd=_np(vb),
                        scale=np.ones((h, w, 2), np.float32)))
    return out


def _params(case):
    p = _abi.default_params()
    p.residualWindowSize, p.iterations = case.get("radius", 2), case.get("iterations", 4)
    p.levels = case.get("levels", 1)
    p.numStyles = case.get("styles", 1)
    p.scheme = SCHEMES[case.get("scheme", "FMBM_RM")]
    if case.get("coherence"):
        p.temporalCoherenceWeight = case["coherence"]
    if case.get("histogram"):
        p.offsetsHistogramSlope[0] = 1.0
    if case.get("terms"):
        p.distTransWeight, p.styleObjIdWeight, p.alphaWeight = 0.01, 0.05, 0.5
    if case.get("exact_filter"):
        p.filterMode = _abi.FILTER_EXACT
    if case.get("keys"):
        p.interpolateKeyFrame = 1
    return p


def _pinned(d):
    out = {}
    for k, v in d.items():
        out[k] = host_array(v.shape, v.dtype)
        out[k][...] = v
    return out


def _prepare_clip(case, seed):
    """The style and the frames resident on the device, and page-locked host
    arrays for the results."""
    w, h, n, ns = case["w"], case["h"], case["frames"], case.get("styles", 1)
    p = _params(case)
    s = Synthesizer(device=0)
    s.setup(p, w, h, case["ew"], case["eh"], ns)
    for i in range(ns):
        ex = _exemplar(case["ew"], case["eh"], 7919 * seed + 31 * i, case.get("holes", False),
                       case.get("terms", False))
        s.set_style(i, ex["base"], ex["output"], ex["orient_tensor"], ex["dist_trans"], ex["object_ids"])
    for i, fr in enumerate(_frames(w, h, case["discs"], n, 104729 * seed + 17)):
        s.set_frame_dict(i, fr)
    if case.get("keys"):
        s.set_keyframes([0, n - 1])
    fl = _abi.output_level(p)
    res = [(host_array((h >> fl, w >> fl, 4), np.float32), host_array((h >> fl, w >> fl), _abi.PATCH_DTYPE))
           for _ in range(n)]
    s.synchronize()
    return dict(case=case, s=s, res=res)


def _angle(tensor):
    a = 0.5 * np.arctan2(2.0 * tensor[..., 1], tensor[..., 0] - tensor[..., 2]) + 0.5 * math.pi
    return np.where(a >= 0.5 * math.pi, a - math.pi, a).astype(np.float32)


def _prepare_steps(case, seed):
    """The level's images and the exemplar uploaded through the step-wise calls."""
    w, h, ew, eh = case["w"], case["h"], case["ew"], case["eh"]
    ex = _exemplar(ew, eh, 7919 * seed + 3)
    fr = _frames(w, h, case["discs"], 1, 104729 * seed + 5)[0]
    t = TexSynth(device=0)
    t.initialize(w, h, ew, eh, 1)
    t.set_params(_params(case))
    t.initialize_exemplars(ew, eh, 1)
    t.upload_image_color4(0, _abi.LAYER_EXEMPLAR_BASE, ex["base"])
    t.upload_image_color4(0, _abi.LAYER_EXEMPLAR_OUTPUT, ex["output"])
    t.upload_image_float(0, _abi.LAYER_EXEMPLAR_ORIENTATION, _angle(ex["orient_tensor"]))
    t.upload_image_float(0, _abi.LAYER_EXEMPLAR_DIST_TRANS, ex["dist_trans"])
    t.upload_image_int(0, _abi.LAYER_EXEMPLAR_OBJECT_IDS, ex["object_ids"])
    t.upload_image_color4(0, _abi.LAYER_INPUT_COLOR, fr["rgba"])
    t.upload_image_float(0, _abi.LAYER_INPUT_ORIENTATION, _angle(fr["orient_tensor"]))
    t.upload_image_int(0, _abi.LAYER_INPUT_ID, fr["object_ids"])
    t.upload_image_float2(0, _abi.LAYER_INPUT_VEL_B, fr["vel_bwd"])
    t.upload_image_float2(0, _abi.LAYER_INPUT_VEL_F, fr["vel_fwd"])
    t.upload_image_float(0, _abi.LAYER_INPUT_DIST_TRANS, fr["dist_trans"])
    t.upload_image_float2(0, _abi.LAYER_INPUT_SCALE, fr["scale"])
    return dict(case=case, t=t)


def _request_sizes(case):
    """(w, h, exemplar) of each request, spread over [low, high] (the same for every seed)."""
    n, lo, hi = case["requests"], case["low"], case["high"]
    rng = random.Random(n * 1000003 + lo * 1009 + hi)
    at = [lo * (hi / lo) ** (i / max(n - 1, 1)) for i in range(n)]
    return [(int(a), max(lo, int(a * rng.uniform(0.6, 1.0))), int(rng.uniform(256, 768))) for a in at]


def _prepare_serve(case, seed):
    """The requests' inputs and result arrays in page-locked host memory, as
    the C ABI's request records, and a server."""
    reqs = []
    for i, (w, h, e) in enumerate(_request_sizes(case)):
        reqs.append(dict(params=_params(dict(STILL)), style=_pinned(_exemplar(e, e, 7919 * seed + 11 * i)),
                         frames=[_pinned(_frames(w, h, 3, 1, 104729 * seed + 13 * i)[0])]))
        reqs[-1]["params"].levels = 3
    arr, keep, outs = serving._build(reqs, True, pinned=True)
    return dict(case=case, server=serving.Server(max_in_flight=case["in_flight"]), reqs=arr, keep=keep, outs=outs)


def _prepare_blur(case, seed):
    n = case["pitch"] * case["h"]
    src = 5.0 * torch.rand((n,), generator=_dev(seed), device="cuda")
    return dict(case=case, t=TexSynth(device=0), src=src.view(case["h"], case["pitch"]),
                dst=torch.zeros((case["h"], case["pitch"]), device="cuda"))


def prepare(case, seed):
    return dict(clip=_prepare_clip, steps=_prepare_steps, serve=_prepare_serve, blur=_prepare_blur)[case["kind"]](
        case, seed)


# --- one pass -----------------------------------------------------------------

def _result(rgba, offs):
    """Colours, the records' nine 32-bit fields and the style layers."""
    return dict(rgba=rgba, records=offs.view(np.float32).reshape(offs.shape + (9,)), layer=offs["layer"])


def _run_clip(st):
    """Synthesises the resident frames and fetches every frame's result into
    page-locked memory (the calls a native host application makes)."""
    s, n = st["s"], len(st["res"])
    if n == 1:
        s._check(lib().pt_synthesize_frame(s.h, 0, None, None), "pt_synthesize_frame")
    else:
        s._check(lib().pt_synthesize_animation(s.h, 0, n - 1, None, None), "pt_synthesize_animation")
    return [_result(*s.get_frame_result(f, *st["res"][f])) for f in range(n)]


def _run_steps(st):
    """One level from random offsets, as SynthesisFrame::propagateAndScatter
    sequences the steps, and its offsets, residual and output."""
    t, its = st["t"], st["case"]["iterations"]
    t.create_random_level(0, 1)
    t.randomize_offsets(0)
    for i in range(its):
        jump = 128
        while jump > 1:
            t.propagate(0, jump)
            jump //= 2
        t.propagate(0, 1)
        t.propagate(0, 1)
        if i < its - 1:
            t.scatter(0)
    out = _result(t.get_output(0), t.get_offsets(0))
    out["residual"] = t.get_residual(0)
    return out


def run(state):
    kind = state["case"]["kind"]
    if kind == "clip":
        return _run_clip(state)
    if kind == "steps":
        return _run_steps(state)
    if kind == "serve":
        st = lib().pt_server_run(state["server"].h, ctypes.cast(state["reqs"], ctypes.c_void_p), len(state["outs"]))
        if st != _abi.PT_OK:
            raise RuntimeError("pt_server_run: %s" % _abi.status_name(st))
        return [_result(rgba[0], offs[0]) for rgba, offs in state["outs"]]
    c, src, dst = state["case"], state["src"], state["dst"]
    state["t"].convolve_separable(src.data_ptr(), dst.data_ptr(), c["w"], c["h"], c["pitch"], c["radius"])
    return dst


# --- what a pass cannot do without ----------------------------------------------

def _still_work(w, h, ew, eh, frames, ns, radius, levels, iterations, passes):
    """Bytes: the frames' seven planes and the exemplars' five read once, the
    colours and records written once.  Operations: the culling leaves about a
    third of the pixels; on each level and pass, each of those has its patch
    distance evaluated once in full (84 operations a tap) and each candidate
    of the first iteration (40 propagated, 25 searched) for at least one tap."""
    px, taps = w * h * frames, (2 * radius + 1) ** 2
    area = sum(0.25 ** l for l in range(levels))
    return dict(bytes=px * (52 + 52) + ew * eh * ns * 52,
                flops=px / 3 * area * passes * 84 * (taps + 40 + (25 if iterations > 1 else 0)))


def work(case):
    if case["kind"] == "clip":
        n = case["frames"]
        return _still_work(case["w"], case["h"], case["ew"], case["eh"], n, case.get("styles", 1), case["radius"],
                           case["levels"], case["iterations"], 2 if n > 1 else 1)
    if case["kind"] == "steps":
        return _still_work(case["w"], case["h"], case["ew"], case["eh"], 1, 1, case["radius"], 1, case["iterations"],
                           1)
    if case["kind"] == "serve":
        each = [_still_work(w, h, e, e, 1, 1, 2, 3, 4, 1) for w, h, e in _request_sizes(case)]
        return dict(bytes=sum(e["bytes"] for e in each), flops=sum(e["flops"] for e in each))
    px = case["w"] * case["h"]
    return dict(bytes=8 * px, flops=4 * px * (2 * case["radius"] + 1))


def exact(case, seed):
    """The separable Gaussian (normalised weights, sigma = radius / 3, zero
    beyond the image) in 64 bits.  A synthesis has no 64-bit counterpart: its
    output is a chain of comparisons of nearly equal patch distances, which
    another rounding decides otherwise."""
    if case["kind"] != "blur":
        return None
    r, w, h = case["radius"], case["w"], case["h"]
    st = 5.0 * torch.rand((case["pitch"] * h,), generator=_dev(seed), device="cuda")
    a = st.view(h, case["pitch"])[:, :w].double()
    i = torch.arange(-r, r + 1, device="cuda", dtype=torch.float64)
    sigma = r / 3.0
    k = torch.exp(-i * i / (2 * sigma * sigma)) / (math.sqrt(2 * math.pi) * sigma)
    rows = sum(k[j] * torch.nn.functional.pad(a, (r, r))[:, j:j + w] for j in range(2 * r + 1))
    both = sum(k[j] * torch.nn.functional.pad(rows, (0, 0, r, r))[j:j + h] for j in range(2 * r + 1))
    out = torch.zeros((h, case["pitch"]), dtype=torch.float64, device="cuda")
    out[:, :w] = both
    return out
