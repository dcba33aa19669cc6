"""The work that users of gs300 have it do, as cases that can be timed and compared.

Every case goes through the package's public entry points on seeded synthetic scenes of the
distributions the tests and the benchmark use (positions N(0, 2^2), log-scales N(-4, 0.5^2), random
rotations, opacity sigmoid(N(0, 1)), SH coefficients N(0, 0.05^2)), made on the GPU and handed to the
viewer as host records, as a loader would.

Kinds:
  view    Viewer: one model, one camera, one frame a pass (camera update + render)
  stages  Preprocessor, RadixSorter and Renderer over buffers that the caller owns
  multi   MultiModelViewer: several transformed models in one frame
  batch   Batch: several views of resident models by one call
  sort    RadixSorter alone: 32-bit keys and values, the live count on the device
  ply     ply_convert: the vertex block of a PLY file into device records
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wgpu-3dgs-viewer_gb300"))

import gs300  # noqa: E402
from gs300 import records as R  # noqa: E402
from gs300 import scene as S  # noqa: E402

FORMATS = {"fp32": R.FORMAT_FP32, "fp16": R.FORMAT_HALF_SH_FP16, "bf16": R.FORMAT_HALF_SH_BF16}
MODES = {"splat": R.DISPLAY_SPLAT, "ellipse": R.DISPLAY_ELLIPSE, "point": R.DISPLAY_POINT}
RECORD_BYTES = {"fp32": 224, "fp16": 128, "bf16": 128}
BATCH_SIZES = ((640, 360), (1280, 720), (960, 540), (1920, 1080))

# FLOPs that one Gaussian cannot do without: two 4x4 products, the projected covariance and its
# axes, and the view direction; each SH band adds its basis and three channels of multiply-adds.
GAUSSIAN_FLOPS = 230
SH_FLOPS = (0, 20, 55, 120)
# FLOPs of a fragment: quad offset, squared radius, exp and alpha, three blended channels.
FRAGMENT_FLOPS = 29


def listed():
    return [
        # a thumbnail or preview of a small object: the smallest call, launches and latency count
        _view("thumb_5k_320x180", 5_000, 320, 180, radius=6.0),
        # the small scene of the parity tests at a window's size: an ordinary interactive frame
        _view("view_100k_640x360", 100_000, 640, 360),
        # a captured room or object at full HD
        _view("view_1m_1080p", 1_000_000, 1920, 1080),
        # the headline benchmark: a large scene at full HD
        _view("view_6m_1080p", 6_000_000, 1920, 1080),
        # a large compressed scene at 4K
        _view("view_3m_4k_bf16", 3_000_000, 3840, 2160, fmt="bf16"),
        # the camera inside the scene, as when flying through it: near splats cover many tiles
        _view("closeup_400k_1366x768_fp16", 400_000, 1366, 768, fmt="fp16", radius=3.0),
        # editing: a selection mask drawn as points in a ragged window
        _view("points_1501k_1283x717", 1_501_003, 1283, 717, mode="point", sh_deg=1, selected=0.6),
        # a host that owns its buffers and calls the stages itself; ellipse outlines, SH degree 2
        dict(_view("stages_ellipse_700k_1600x900_fp16", 700_001, 1600, 900, fmt="fp16", mode="ellipse", sh_deg=2, std=2.5), kind="stages"),
        # the four-model scene of the benchmark, 10 % translated Gaussians, one frame
        {"name": "multi_4x6m_1080p", "kind": "multi", "n": 6_000_000, "models": 4, "w": 1920, "h": 1080, "fmt": "fp32", "radius": 8.0},
        # a batch of views of two scenes at mixed sizes, as rendered offline or for training data
        {"name": "batch_12_views_2x600k", "kind": "batch", "n": 600_000, "models": 2, "views": 12, "fmt": "fp32", "radius": 8.0},
        # the sorter by itself, random 32-bit keys, a live count below the capacity
        {"name": "sort_2m", "kind": "sort", "n": 2_000_003, "live": 0.9, "key_bits": 32},
        # loading a scene: a standard degree-3 PLY into full-precision records
        {"name": "ply_1m_fp32", "kind": "ply", "n": 1_000_000, "fmt": "fp32", "sh_deg": 3},
    ]


def _view(name, n, w, h, fmt="fp32", mode="splat", sh_deg=3, std=3.0, radius=8.0, selected=1.0):
    return {"name": name, "kind": "view", "n": n, "w": w, "h": h, "fmt": fmt, "mode": mode, "sh_deg": sh_deg, "std": std,
            "radius": radius, "selected": selected}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["view"] * 10 + ["stages"] * 2 + ["multi"] * 2 + ["batch"] * 2 + ["sort"] * 2 + ["ply"] * 2)
    if kind == "sort":
        return {"kind": kind, "n": _log_int(rng, 1_000, 8_000_000), "live": round(rng.uniform(0.3, 1.0), 3),
                "key_bits": rng.choice([32, 32, 30, 24, 16])}
    if kind == "ply":
        return {"kind": kind, "n": _log_int(rng, 2_000, 2_000_000), "fmt": rng.choice(list(FORMATS)), "sh_deg": rng.choice([3, 3, 3, 2, 1, 0])}
    if kind == "batch":
        views = rng.randint(2, 16)
        return {"kind": kind, "n": _log_int(rng, 5_000, 600_000), "models": rng.randint(1, 3), "views": views,
                "fmt": rng.choice(list(FORMATS)), "radius": round(rng.uniform(5.0, 12.0), 2)}
    w = _log_int(rng, 160, 3840)
    h = max(64, min(2160, int(w * rng.choice([9 / 16, 9 / 16, 3 / 4, 1.0, 0.45]))))
    radius = round(rng.uniform(3.0, 12.0), 2)
    # no drawn frame costs more than the 6M / 1080p one: splats cover pixels / distance^2
    most = 6e6 * 1920 * 1080 / (w * h) * min(1.0, (radius / 8.0) ** 2)
    n = _log_int(rng, 2_000, max(4_000, min(6_000_000, int(most))))
    fmt = rng.choice(list(FORMATS))
    if kind == "multi":
        return {"kind": kind, "n": n, "models": rng.randint(2, 5), "w": w, "h": h, "fmt": fmt, "radius": radius}
    return {"kind": kind, "n": n, "w": w, "h": h, "fmt": fmt, "mode": rng.choice(["splat"] * 5 + ["ellipse", "point"]),
            "sh_deg": rng.choice([3, 3, 3, 2, 1, 0]), "std": rng.choice([3.0, 3.0, 2.5, 2.0]), "radius": radius,
            "selected": rng.choice([1.0, 1.0, 1.0, 0.5])}


# ---- inputs -----------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _attributes(n, g):
    """(positions, log-scales, quaternions x y z w, opacity logits, dc, sh) as FP32 CUDA tensors."""
    def normal(*shape):
        return torch.randn(shape, generator=g, device="cuda")

    pos, log_scale, quat = normal(n, 3) * 2.0, normal(n, 3) * 0.5 - 4.0, normal(n, 4)
    quat = quat / quat.norm(dim=1, keepdim=True)
    return pos, log_scale, quat, normal(n), normal(n, 3) * 0.2 + 0.5, normal(n, 45) * 0.05


def _cov3d(quat, scale):
    """(xx, xy, xz, yy, yz, zz) of R S S^T R^T in 64 bits."""
    x, y, z, w = quat.double().unbind(1)
    r = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], dim=1).view(-1, 3, 3)
    m = r * scale.double()[:, None, :]
    s = m @ m.transpose(1, 2)
    return torch.stack([s[:, 0, 0], s[:, 0, 1], s[:, 0, 2], s[:, 1, 1], s[:, 1, 2], s[:, 2, 2]], dim=1)


def _rgba(dc, logit):
    """RGBA8 packed into int64: rgb = 0.5 + SH_C0 dc, alpha = sigmoid(logit)."""
    rgb = (0.5 + S.SH_C0 * dc.double()).clamp(0.0, 1.0)
    rgba = torch.cat([rgb, torch.sigmoid(logit.double())[:, None]], dim=1)
    c = torch.round(rgba * 255.0).long()
    return c[:, 0] | (c[:, 1] << 8) | (c[:, 2] << 16) | (c[:, 3] << 24)


def _as_int32(v):
    return torch.where(v >= 1 << 31, v - (1 << 32), v).int()


def _records(n, seed, fmt, translated=0.0):
    """A seeded scene as device records in host memory (numpy)."""
    g = _generator(seed)
    pos, log_scale, quat, logit, dc, sh = _attributes(n, g)
    if translated:
        moved = torch.rand(n, generator=g, device="cuda") < translated
        pos = pos + moved[:, None] * torch.randn((n, 3), generator=g, device="cuda") * 0.1
    color, scale = _as_int32(_rgba(dc, logit)), log_scale.exp()
    if fmt == "fp32":
        rec = torch.zeros((n, 56), dtype=torch.int32, device="cuda")
        f = rec.view(torch.float32)
        f[:, 4:49] = sh
        for a in range(0, n, 1 << 20):
            f[a:a + (1 << 20), 49:55] = _cov3d(quat[a:a + (1 << 20)], scale[a:a + (1 << 20)]).float()
    else:
        rec = torch.zeros((n, 32), dtype=torch.int32, device="cuda")
        f, h = rec.view(torch.float32), rec.view(torch.float16)
        h[:, 8:12], h[:, 12:15] = quat.half(), scale.half()
        rec.view(torch.float16 if fmt == "fp16" else torch.bfloat16)[:, 15:60] = sh
    f[:, :3] = pos
    rec[:, 3] = color
    return rec.cpu().numpy().view(R.record_dtype(FORMATS[fmt])).reshape(-1)


def _camera(seed, w, h, radius):
    rng = random.Random(int(seed))
    cam = S.orbit_camera(rng.uniform(0.0, 120.0), radius=radius, pitch=rng.uniform(-0.3, 0.3))
    return gs300.CameraPod.new(cam, (w, h))


def _selection(n, seed, share):
    bits = np.random.default_rng(seed).random(((n + 31) // 32) * 32) < share
    return np.packbits(bits, bitorder="little").view(np.uint32)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _target(w, h):
    return torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")


def _model_sizes(n, models):
    parts = (0.5, 1.0, 1.5, 3.0, 0.75)[:models]
    return [max(1, int(n * p / sum(parts))) for p in parts]


def _multi_viewer(case, seed):
    mv, rng = gs300.MultiModelViewer(), np.random.default_rng(seed)
    keys = []
    for i, n in enumerate(_model_sizes(case["n"], case["models"])):
        key = f"model {i}"
        mv.insert_model(key, _records(n, seed * 16 + i, case["fmt"], translated=0.1), FORMATS[case["fmt"]])
        q = rng.normal(size=4)
        mv.update_model_transform(key, tuple(rng.normal(0.0, 0.5, 3)), tuple(q / np.linalg.norm(q)), (1.0, 1.0, 1.0))
        keys.append(key)
    return mv, keys


def _live(case):
    return max(1, int(case["n"] * case["live"]))


def _sort_pairs(case, seed):
    n, g = case["n"], _generator(seed)
    keys = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device="cuda").int()
    return keys, torch.randperm(n, generator=g, device="cuda").int()


_PLY_REST = (0, 9, 24, 45)  # f_rest properties of a degree 0..3 file


def _ply_vertices(case, seed):
    """(n, fields) FP32 vertices: x y z, normals, f_dc, f_rest (channel-major), opacity, scale, rot (w first)."""
    n = case["n"]
    pos, log_scale, quat, logit, dc, sh = _attributes(n, _generator(seed))
    length = torch.rand((n, 1), generator=_generator(seed + 1), device="cuda") + 0.5  # files hold unnormalised rotations
    rest = sh[:, :_PLY_REST[case["sh_deg"]]]
    return torch.cat([pos, torch.zeros_like(pos), dc, rest, logit[:, None], log_scale, quat[:, [3, 0, 1, 2]] * length], dim=1).contiguous()


def _ply_header(n, rest):
    names = ["x", "y", "z", "nx", "ny", "nz"] + [f"f_dc_{i}" for i in range(3)] + [f"f_rest_{i}" for i in range(rest)]
    names += ["opacity"] + [f"scale_{i}" for i in range(3)] + [f"rot_{i}" for i in range(4)]
    lines = ["ply", "format binary_little_endian 1.0", f"element vertex {n}"] + [f"property float {p}" for p in names]
    return ("\n".join(lines + ["end_header"]) + "\n").encode()


# ---- what a program has in hand before the call ---------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("view", "stages"):
        pod = _camera(seed, case["w"], case["h"], case["radius"])
        fmt, selected = FORMATS[case["fmt"]], case["selected"] < 1.0
        state = {"kind": kind, "pod": pod, "target": _target(case["w"], case["h"])}
        recs = _records(case["n"], seed, case["fmt"])
        bits = _selection(case["n"], seed, case["selected"]) if selected else None
        if kind == "view":
            viewer = state["viewer"] = gs300.Viewer(recs, fmt)
            viewer.update_gaussian_transform(1.0, MODES[case["mode"]], case["sh_deg"], False, case["std"])
            viewer.set_selection(bits)
            run(state)  # the program's first frame; the viewer grows its tile list where the frame needs it
            viewer.synchronize(_stream())
            return state
        n = case["n"]
        words = lambda k: torch.zeros(max(1, k), dtype=torch.int32, device="cuda")  # noqa: E731
        area = lambda k: torch.zeros(k, dtype=torch.uint8, device="cuda")  # noqa: E731
        gt = gs300.gaussian_transform_pod(1.0, MODES[case["mode"]], case["sh_deg"], False, case["std"])
        # room for the pairs of the largest splats: a multiple of the splats and of the tiles
        pairs = 24 * n + 64 * ((case["w"] + 15) // 16) * ((case["h"] + 15) // 16)
        state.update(
            n=n, fmt=fmt, records=torch.from_numpy(recs.view(np.uint8)).cuda(), control=words(8), indices=words(n),
            depths=words(gs300.Preprocessor.depth_capacity(n)), splats=torch.zeros(12 * n, device="cuda"), pairs=pairs,
            selection=None if bits is None else torch.from_numpy(bits.view(np.int32)).cuda(),
            uniforms=gs300.frame_uniforms(pod, gs300.model_transform_pod(), gt, (case["w"], case["h"])),
            pre=area(gs300.Preprocessor.scratch_bytes(n)), srt=area(gs300.RadixSorter.scratch_bytes(n)),
            ras=area(gs300.Renderer.scratch_bytes(n, case["w"], case["h"], pairs)))
        return state
    if kind == "multi":
        mv, keys = _multi_viewer(case, seed)
        state = {"kind": kind, "viewer": mv, "keys": keys, "pod": _camera(seed, case["w"], case["h"], case["radius"]),
                 "target": _target(case["w"], case["h"])}
        run(state)
        mv.synchronize(_stream())
        return state
    if kind == "batch":
        mv, keys = _multi_viewer(case, seed)
        views = []
        for i in range(case["views"]):
            w, h = BATCH_SIZES[i % len(BATCH_SIZES)]
            views.append((keys[i % len(keys)], _camera(seed * 64 + i, w, h, case["radius"]), _target(w, h)))
        state = {"kind": kind, "viewer": mv, "batch": gs300.Batch(mv, keys), "views": views}
        run(state)  # the shape's first render builds its graph
        state["batch"].synchronize(_stream())
        return state
    if kind == "sort":
        n, (keys, values) = case["n"], _sort_pairs(case, seed)
        nbytes = gs300.RadixSorter.scratch_bytes(n)
        return {"kind": kind, "n": n, "bits": case["key_bits"], "keys": keys, "values": values, "out_keys": torch.empty_like(keys),
                "out_values": torch.empty_like(values), "count": torch.tensor([_live(case)], dtype=torch.int32, device="cuda"),
                "scratch": torch.zeros(nbytes, dtype=torch.uint8, device="cuda"), "nbytes": nbytes}
    vertices = _ply_vertices(case, seed)
    layout = gs300.ply_parse_header(_ply_header(case["n"], _PLY_REST[case["sh_deg"]]))
    out = torch.zeros((case["n"], RECORD_BYTES[case["fmt"]] // 4), dtype=torch.int32, device="cuda")
    return {"kind": "ply", "vertices": vertices, "layout": layout, "fmt": case["fmt"], "records": out}


# ---- one pass -----------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "view":
        state["viewer"].update_camera_with_pod(state["pod"])
        state["viewer"].render(state["target"], _stream())
        return state["target"]
    if kind == "multi":
        state["viewer"].update_camera_with_pod(state["pod"])
        state["viewer"].render(state["target"], state["keys"], _stream())
        return state["target"]
    if kind == "batch":
        state["batch"].render(state["views"], _stream())
        return [target for _, _, target in state["views"]]
    if kind == "stages":
        s, st = state, _stream()
        control, target = s["control"].data_ptr(), s["target"]
        gs300.Preprocessor.preprocess(s["uniforms"], s["records"], s["fmt"], s["n"], control, control + 16, s["indices"], s["depths"],
                                      s["depths"].numel(), s["splats"], s["pre"], s["pre"].numel(), selection=s["selection"], stream=st)
        gs300.RadixSorter.sort(s["depths"], s["indices"], s["n"], s["srt"], s["srt"].numel(), count=control + 4, stream=st)
        gs300.Renderer.render(s["uniforms"], s["splats"], s["indices"], control + 4, s["n"], target, target.shape[1], target.shape[0],
                              target.stride(0), s["pairs"], s["ras"], s["ras"].numel(), stream=st)
        return {"frame": target, "indices": s["indices"], "control": s["control"]}
    if kind == "sort":
        state["out_keys"].copy_(state["keys"])  # the sort is in place: each pass sorts fresh keys
        state["out_values"].copy_(state["values"])
        gs300.RadixSorter.sort(state["out_keys"], state["out_values"], state["n"], state["scratch"], state["nbytes"],
                               count=state["count"], key_bits=state["bits"], stream=_stream())
        return {"keys": state["out_keys"], "values": state["out_values"]}
    gs300.ply_convert(state["vertices"].data_ptr(), state["layout"], FORMATS[state["fmt"]], state["records"].data_ptr(), _stream())
    rec = state["records"]
    f = rec.view(torch.float32)
    if state["fmt"] == "fp32":
        return {"pos": f[:, :3], "color": rec[:, 3], "sh": f[:, 4:49], "cov3d": f[:, 49:55]}
    h = rec.view(torch.float16)
    sh = h if state["fmt"] == "fp16" else rec.view(torch.bfloat16)
    return {"pos": f[:, :3], "color": rec[:, 3], "rot": h[:, 8:12], "scale": h[:, 12:15], "sh": sh[:, 15:60]}


# ---- what a pass cannot do without ----------------------------------------------------------------
def work(case):
    """Each input read once and each output written once: records in, frames out (depth keys, splats
    and tile lists are the implementation's own).  A frame's FLOPs: every Gaussian once, and one
    fragment for each pixel (more depend on the scene)."""
    kind, n = case["kind"], case["n"]
    if kind == "sort":
        return {"bytes": 16 * _live(case), "flops": 0}
    if kind == "ply":
        return {"bytes": n * (4 * (17 + _PLY_REST[case["sh_deg"]]) + RECORD_BYTES[case["fmt"]]), "flops": n * 120}
    rec = RECORD_BYTES[case["fmt"]]
    if kind == "batch":
        pixels = sum(w * h for w, h in (BATCH_SIZES[i % len(BATCH_SIZES)] for i in range(case["views"])))
        sizes = _model_sizes(n, case["models"])
        seen = sum(sizes[i % len(sizes)] for i in range(case["views"]))
        used = sum(sizes[:case["views"]])
        return {"bytes": rec * used + 4 * pixels, "flops": seen * (GAUSSIAN_FLOPS + SH_FLOPS[3]) + pixels * FRAGMENT_FLOPS}
    pixels = case["w"] * case["h"]
    drawn = n * case.get("selected", 1.0)
    flops = drawn * (GAUSSIAN_FLOPS + SH_FLOPS[case.get("sh_deg", 3)]) + pixels * FRAGMENT_FLOPS
    return {"bytes": rec * drawn + 4 * pixels, "flops": flops}


# ---- the same in 64 bits ---------------------------------------------------------------------------
def exact(case, seed):
    """Sorted pairs and converted records in 64 bits.  Frames are bytes (each blend rounds to 8 bits,
    in draw order) and have no 64-bit value of their own."""
    if case["kind"] == "sort":
        live, (keys, values) = _live(case), _sort_pairs(case, seed)
        order = torch.sort(keys[:live].long() & ((1 << case["key_bits"]) - 1), stable=True).indices
        return {"keys": torch.cat([keys[:live][order], keys[live:]]), "values": torch.cat([values[:live][order], values[live:]])}
    if case["kind"] != "ply":
        return None
    v = _ply_vertices(case, seed).double()
    rest = _PLY_REST[case["sh_deg"]]
    color = _as_int32(_rgba(v[:, 6:9], v[:, 9 + rest]))
    sh = torch.zeros((case["n"], 15, 3), dtype=torch.float64, device="cuda")
    if rest:
        sh[:, :rest // 3] = v[:, 9:9 + rest].view(-1, 3, rest // 3).transpose(1, 2)
    scale, rot = v[:, 10 + rest:13 + rest].exp(), v[:, 13 + rest:17 + rest][:, [1, 2, 3, 0]]
    rot = rot / rot.norm(dim=1, keepdim=True)
    out = {"pos": v[:, :3], "color": color, "sh": sh.view(-1, 45)}
    if case["fmt"] == "fp32":
        return dict(out, cov3d=_cov3d(rot, scale))
    return dict(out, rot=rot, scale=scale)
