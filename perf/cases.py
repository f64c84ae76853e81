"""Timed workloads of the compound-eye renderer, run through its C ABI.

The library holds one scene and its eyes at a time, as the reference does, so
a program loads a scene, sets up its eye once and then renders.  `prepare`
does that set-up (scene, eye, networks, batch handle, one warm render) and
restarts the eye's random streams, so that equal inputs give equal outputs;
`run` is one pass of the program's loop.

Scenes: `small` (ground and 64 boxes, 770 triangles), `textured` (the same
size with PNG textures and vertex colours), `terrain` (588,288-triangle
heightfield with plants, 200 m square).  Settings that differ from the
library's defaults are the ones its autotuner picks for that scene.
"""
import ctypes
import math
import os
import struct
import sys
import tempfile

import numpy as np
import torch

ROOT = os.getcwd()
sys.path.insert(0, os.path.join(ROOT, "compound-ray_gb300"))

import eyeRendererHelperFunctions as eh  # noqa: E402
import scenes  # noqa: E402

DEG = math.pi / 180.0


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The reference's speed test: a 1000-ommatidium eye at 32 samples, one
        # frame at a time, the image read after each (closed-loop agent).
        dict(name="frame_small", kind="frame", scene="small", n=1000, spp=32, proj="single_dimension_fast", w=1000,
             h=1, aa_lo=3.0, aa_hi=3.0, variant=0, cut=0),
        # The same loop in a natural scene with a full-size eye.
        dict(name="frame_terrain", kind="frame", scene="terrain", n=6000, spp=256, proj="single_dimension_fast",
             w=6000, h=1, aa_lo=1.5, aa_hi=4.0, variant=0, cut=0),
        # An image for a person to look at: the spherical projection, odd sizes.
        dict(name="frame_spherical", kind="frame", scene="small", n=20011, spp=4, proj="spherical_orientationwise",
             w=1023, h=511, aa_lo=2.0, aa_hi=2.0, variant=0, cut=0),
        # Dataset generation: a long trajectory of the natural scene with tuned
        # settings (the largest case).
        dict(name="trajectory_terrain", kind="device", scene="terrain", n=6000, spp=256, poses=1024, aa_lo=1.5,
             aa_hi=4.0, variant=2, cut=128),
        # A trajectory at few samples, default settings.
        dict(name="trajectory_low_spp", kind="device", scene="terrain", n=6000, spp=8, poses=256, aa_lo=1.5,
             aa_hi=4.0, variant=0, cut=0),
        # A trajectory of the small eye, default settings.
        dict(name="trajectory_small", kind="device", scene="small", n=1000, spp=32, poses=1000, aa_lo=3.0, aa_hi=3.0,
             variant=0, cut=0),
        # Host arrays in and out, textures, odd sizes, a sample count that
        # leaves half a warp.
        dict(name="host_textured", kind="host", scene="textured", n=1777, spp=48, poses=37, aa_lo=1.0, aa_hi=6.0,
             variant=0, cut=0),
        # Many uneven eyes in one launch.
        dict(name="batch_uneven", kind="batch", scene="small", eyes=24, n_min=500, n_max=30000, spp_max=512, poses=6,
             eye_seed=3, aa_lo=1.0, aa_hi=6.0, variant=2, cut=32),
        # The learned denoiser over a trajectory.
        dict(name="denoise_terrain", kind="denoise", scene="terrain", n=6000, spp=8, poses=250, aa_lo=1.5, aa_hi=4.0,
             variant=2, cut=128),
        # Learned sample allocation: a small eye over many poses, and a large
        # panoramic eye over few.
        dict(name="adaptive_small", kind="adaptive", scene="small", n=1000, spp=8, poses=1000, aa_lo=3.0, aa_hi=3.0,
             exponent=0.5, halvings=-1.0, variant=2, cut=0),
        dict(name="adaptive_terrain", kind="adaptive", scene="terrain", n=30000, spp=8, poses=16, aa_lo=0.5, aa_hi=5.0,
             exponent=0.625, halvings=-0.75, variant=2, cut=128),
        # A training job of the denoiser: rows from rendered poses, then Adam
        # steps, then the checkpoint.
        dict(name="train_denoiser", kind="train", scene="terrain", n=6000, spp=8, poses=8, target_spp=256, steps=200,
             batch=8192, aa_lo=1.5, aa_hi=4.0, variant=2, cut=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "device", "device", "host", "batch", "denoise", "adaptive", "train"])
    scene = rng.choice(["small", "textured", "terrain"])
    aa_lo = rng.uniform(0.5, 3.0)
    c = dict(kind=kind, scene=scene, aa_lo=aa_lo, aa_hi=aa_lo * rng.uniform(1.0, 2.5), variant=rng.choice([0, 0, 1, 2]),
             cut=rng.choice([0, 0, 32, 128]))
    if kind == "frame":
        proj = rng.choice(["single_dimension_fast", "single_dimension", "spherical_orientationwise",
                           "spherical_positionwise"])
        n = _log_int(rng, 100, 20000)
        c.update(n=n, spp=_log_int(rng, 1, 512), proj=proj)
        c.update(w=n, h=1) if proj == "single_dimension_fast" else c.update(w=rng.randint(200, 1100), h=rng.randint(100, 600))
    elif kind in ("device", "host"):
        n, spp = _log_int(rng, 100, 20000), _log_int(rng, 1, 700)
        c.update(n=n, spp=spp, poses=max(1, min(_log_int(rng, 1, 1000), int(3e8 / (n * spp)))))
    elif kind == "batch":
        c.update(scene="small", eyes=rng.randint(2, 24), n_min=200, n_max=_log_int(rng, 1000, 30000),
                 spp_max=rng.choice([64, 128, 256, 512]), poses=rng.randint(1, 6), eye_seed=rng.randint(1, 1000))
    elif kind == "denoise":
        n = _log_int(rng, 300, 20000)
        c.update(n=n, spp=rng.choice([4, 8, 8, 16]), poses=max(1, min(_log_int(rng, 1, 1000), int(2e6 / n))))
    elif kind == "adaptive":
        n = _log_int(rng, 300, 30000)
        c.update(n=n, spp=8, poses=max(1, min(_log_int(rng, 1, 1000), int(8e5 / n))),
                 exponent=rng.choice([0.5, 0.625, 0.75]), halvings=rng.choice([-1.0, -0.5, 0.0]))
    else:
        c.update(n=_log_int(rng, 1000, 8000), spp=8, poses=rng.randint(2, 8), target_spp=rng.choice([64, 256]),
                 steps=rng.randint(50, 200), batch=rng.choice([1000, 4096, 8192]))
    return c


# ---------------------------------------------------------------------------
# The program around the library: one scene, one set-up at a time
# ---------------------------------------------------------------------------
class _Program:
    def __init__(self):
        self.lib = eh.loadRenderer()
        self.lib.setVerbosity(False)
        self.lib.setOmmatidia.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
        self.stream = torch.cuda.Stream()
        self.dir = tempfile.mkdtemp(prefix="cr_cases_")
        self.infos = {}
        self.loaded = None
        self.batch = None  # handle, pose buffer, output buffer of the batch in force

    def check(self, rc=0):
        if rc != 0:
            raise RuntimeError(eh.lastError(self.lib) or "call failed")

    def info(self, scene, case):
        key = scene if scene != "batch" else (scene, case["eyes"], case["n_min"], case["n_max"], case["spp_max"],
                                              case["eye_seed"], case["aa_lo"], case["aa_hi"])
        if key not in self.infos:
            d = os.path.join(self.dir, "scene%d" % len(self.infos))
            if scene == "terrain":
                i = scenes.terrain_scene(d, poses=1)
            elif scene == "textured":
                i = scenes.textured_scene(d)
            elif scene == "small":
                i = scenes.small_scene(d)
            else:
                i = scenes.batch_scene(d, seed=scenes.SEED + case["eye_seed"], n_eyes=case["eyes"], poses_per_eye=1,
                                       n_min=case["n_min"], n_max=case["n_max"],
                                       spp_choices=tuple(range(16, case["spp_max"] + 1, 16)),
                                       aa_deg=(case["aa_lo"], case["aa_hi"]))
                i["boxes"] = scenes.small_scene(d + "_boxes", seed=scenes.SEED + case["eye_seed"])["boxes"]
            self.infos[key] = i
        return key, self.infos[key]

    def load(self, scene, case):
        key, info = self.info(scene, case)
        if self.loaded != key:
            self.batch = None
            self.lib.loadGlTFscene(info["gltf"].encode())
            err = eh.lastError(self.lib)
            if err:
                raise RuntimeError(err)
            eh.gotoFirstCompoundEye(self.lib)
            self.loaded = key
        self.lib.crSetStream(self.stream.cuda_stream)
        self.check(self.lib.crSetRenderVariant(case["variant"]))
        self.check(self.lib.crSetCutRadius(1.0 / case["cut"] if case["cut"] else 0.0))
        return info

    def eye(self, case, spp):
        """The case's eye on the current camera, its random streams restarted."""
        rng = np.random.default_rng(case["n"])
        omm = np.zeros((case["n"], 8), np.float32)
        if case["scene"] == "terrain" and case["kind"] != "adaptive":
            pos, d = scenes.droplet_eye(case["n"], rng)
        else:
            d = scenes.fibonacci_sphere(case["n"])
            pos = d * 0.001
        omm[:, 0:3], omm[:, 3:6] = pos, d
        omm[:, 6] = rng.uniform(case["aa_lo"] * DEG, case["aa_hi"] * DEG, case["n"])
        self.lib.setOmmatidia(omm.ctypes.data, case["n"])
        self.lib.setCurrentEyeSamplesPerOmmatidium(int(spp))


_program = None


def _prog():
    global _program
    if _program is None:
        _program = _Program()
    return _program


def _poses(case, info, count, seed, walk):
    """(count, 12) poses: a walk over the terrain or places between the boxes."""
    rng = np.random.default_rng([seed, 77])
    if case["scene"] == "terrain":
        hfn = info["height_fn"]
        if walk:
            return scenes.random_walk(hfn, count, rng)
        return scenes.random_poses(hfn, count, rng, 60.0)
    if "boxes" in info:
        return scenes.open_poses(info["boxes"], count, rng)
    return np.stack([scenes.pose_rows(np.array([rng.uniform(-8, 8), 2.2, rng.uniform(-8, 8)]),
                                      rng.uniform(0, 2 * math.pi)) for _ in range(count)])


def _p16(p12):
    p16 = np.zeros((len(p12), 16), np.float32)
    for k in range(4):
        p16[:, 4 * k:4 * k + 3] = p12[:, 3 * k:3 * k + 3]
    return torch.from_numpy(p16).cuda()


# Parameter vector of the networks: W1 [112 x 128], b1, W2 [128 x 128], b2,
# W3, b3, W4 [128 x 8], b4; a checkpoint is a 4-word header, the parameters
# and two vectors of Adam moments.
_SHAPES = [(112, 128), (128,), (128, 128), (128,), (128, 128), (128,), (128, 8), (8,)]
_COUNT = sum(int(np.prod(s)) for s in _SHAPES)


def _allocator_checkpoint(path):
    """An allocator that asks for more samples the wider an ommatidium's colour
    spread: a piecewise linear fit of log2(count) / 10, count = (512 sd)^(4/3)
    (the error of stratified samples falls faster than 1 / sqrt(count)), of the
    three spread features (4 sd of each channel), carried through the hidden
    layers by unit weights."""
    knots = np.array([0.0, 0.02, 0.08, 0.25, 0.7])
    sd = np.maximum(np.append(knots, 2.0) / 4.0, 1e-9)
    want = np.maximum(0.2, (4.0 / 3.0) * np.log2(np.maximum(512.0 * sd, 1.0)) / 10.0)
    slope = np.diff(want) / np.diff(np.append(knots, 2.0))
    p = [np.zeros(s, np.float32) for s in _SHAPES]
    for i, k in enumerate(knots):
        p[0][3:6, i] = 1.0 / 3.0
        p[1][i] = -k
        p[2][i, i] = p[4][i, i] = 1.0
        p[6][i, 0:3] = slope[i] - (slope[i - 1] if i else 0.0)
    p[7][0:3] = want[0]
    flat = np.concatenate([a.ravel() for a in p]).astype(np.float32)
    with open(path, "wb") as f:
        f.write(struct.pack("<4I", 0x4E445243, 1, _COUNT, 0))
        f.write(flat.tobytes())
        f.write(np.zeros(2 * _COUNT, np.float32).tobytes())


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def prepare(case, seed):
    g = _prog()
    lib = g.lib
    kind = case["kind"]
    s = {"case": case, "g": g}
    if kind == "batch":
        info = g.load("batch", case)
        n_eyes = case["eyes"]
        cams = np.arange(info["first_batch_camera"], info["first_batch_camera"] + n_eyes, dtype=np.int32)
        s["poses"] = _p16(_poses(case, info, n_eyes * case["poses"], seed, False))
        torch.cuda.synchronize()
        if g.batch is not None:
            lib.crBatchDestroy(g.batch[0])
        for i, c in enumerate(cams):  # restarts the streams; a batch recorded before ends here
            lib.gotoCamera(int(c))
            lib.setCurrentEyeSamplesPerOmmatidium(int(info["spp"][i]))
        d_poses = torch.empty_like(s["poses"])
        d_poses.copy_(s["poses"])
        d_out = torch.empty(sum(3 * case["poses"] * n for n in info["n"]), device="cuda")
        torch.cuda.synchronize()
        h = lib.crBatchCreate(cams, n_eyes, case["poses"], d_poses.data_ptr(), d_out.data_ptr())
        g.check(0 if h > 0 else -1)
        g.batch = (h, d_poses, d_out)
        g.check(lib.crBatchLaunch(h))
        g.check(lib.crSynchronize())
        return s
    info = g.load(case["scene"], case)
    if kind == "frame":
        lib.setCurrentEyeShaderName(case["proj"].encode())
        eh.setRenderSize(lib, case["w"], case["h"])
        g.eye(case, case["spp"])
        s["poses"] = _poses(case, info, 1, seed, False)
        s["pose"] = [float(v) for v in s["poses"][0]]
        lib.renderFrame()
        g.check(lib.crSynchronize())
        return s
    if kind in ("device", "host"):
        g.eye(case, case["spp"])
        s["poses"] = _poses(case, info, case["poses"], seed, True)
    else:
        g.eye(case, 32)
        s["poses"] = _poses(case, info, case["poses"], seed, kind == "denoise")
    shape = (case["poses"], case["n"], 3)
    if kind == "host":
        g.check(lib.crRenderPoses(s["poses"], 1, np.zeros(shape[1:], np.float32)))
        return s
    if kind == "train":
        s["path"] = os.path.join(g.dir, "denoiser.bin")
        s["loss"] = np.zeros(case["steps"], np.float32)
        return s
    s["d_poses"], s["out"] = _p16(s["poses"]), torch.empty(shape, device="cuda")
    torch.cuda.synchronize()
    if kind == "denoise":
        g.check(lib.crDenoiserInit(5))
    elif kind == "adaptive":
        path = os.path.join(g.dir, "allocator.bin")
        _allocator_checkpoint(path)
        lib.crDenoiserRelease()
        g.check(lib.crAllocatorLoad(path.encode()))
        g.check(lib.crSetAllocatorExponent(case["exponent"]))
        g.check(lib.crSetAllocatorHalvings(case["halvings"]))
        s["level"] = torch.empty(shape[:2], dtype=torch.uint8, device="cuda")
        s["rays"] = ctypes.c_double(0.0)
        torch.cuda.synchronize()
    _device_pass(s)
    g.check(lib.crSynchronize())
    return s


def _device_pass(s):
    lib, case, kind = s["g"].lib, s["case"], s["case"]["kind"]
    if kind == "device":
        s["g"].check(lib.crRenderPosesDevice(s["d_poses"].data_ptr(), case["poses"], s["out"].data_ptr()))
        return s["out"]
    if kind == "denoise":
        s["g"].check(lib.crDenoiserRenderPosesDevice(s["d_poses"].data_ptr(), case["poses"], case["spp"],
                                                     s["out"].data_ptr()))
        return s["out"]
    s["g"].check(lib.crAdaptiveRenderPosesDevice(s["d_poses"].data_ptr(), case["poses"], case["spp"],
                                                 s["out"].data_ptr(), s["level"].data_ptr(), ctypes.byref(s["rays"])))
    return {"colours": s["out"], "level": s["level"], "rays": s["rays"].value}


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def run(s):
    g, case, kind = s["g"], s["case"], s["case"]["kind"]
    lib = g.lib
    if kind == "frame":
        p = s["pose"]
        lib.setCameraPosition(p[0], p[1], p[2])
        lib.setCameraLocalSpace(*p[3:12])
        if lib.renderFrame() < 0:
            g.check(-1)
        return {"image": eh.getFrame(lib, case["w"], case["h"]), "colours": eh.getOmmatidialColours(lib)}
    if kind == "host":
        return eh.renderPoses(lib, s["poses"])
    if kind == "batch":  # the recorded batch reads its poses from a fixed buffer
        h, d_poses, d_out = g.batch
        with torch.cuda.stream(g.stream):
            d_poses.copy_(s["poses"])
        g.check(lib.crBatchLaunch(h))
        return d_out
    if kind == "train":
        g.check(lib.crDenoiserInit(5))
        g.check(lib.crDenoiserAddTrainingPoses(s["poses"], case["poses"], case["spp"], case["target_spp"]))
        g.check(lib.crDenoiserTrain(case["steps"], case["batch"], 1e-3, 1, s["loss"].ctypes.data))
        g.check(lib.crDenoiserSave(s["path"].encode()))
        state = np.fromfile(s["path"], np.float32, offset=16)
        return {"loss": s["loss"].copy(), "params": state[:_COUNT], "moments": state[_COUNT:]}
    return _device_pass(s)


# ---------------------------------------------------------------------------
# work, exact
# ---------------------------------------------------------------------------
# Flops of a ray with one box-free triangle test: two rotations and a frame
# change (75), the sheared triangle test (45), interpolation and the gamma
# curve (25), its share of the sum (5).  Flops of a network row, forward.
RAY_FLOPS = 150.0
NET_FLOPS = 2.0 * (112 * 128 + 2 * 128 * 128 + 128 * 8)
# Bytes of a scene that a pass reads once at most: nodes, triangles, shading
# records of the triangles its rays hit (the scene is far smaller than what
# the rays request, so few of them count).
OUT_BYTES = 12.0


def work(case):
    kind = case["kind"]
    if kind == "batch":
        _, info = _prog().info("batch", case)
        rays = float(case["poses"]) * sum(n * k for n, k in zip(info["n"], info["spp"]))
        rows = float(case["poses"]) * sum(info["n"])
        return {"bytes": rows * OUT_BYTES + 32.0 * sum(info["n"]) + 64.0 * rays / case["poses"], "flops": rays * RAY_FLOPS}
    P = float(case.get("poses", 1))
    rows = P * case["n"]
    rays = rows * case["spp"]
    state = 64.0 * case["n"] * case["spp"]  # generator states read and written once a call
    b = {"bytes": rows * OUT_BYTES + 64.0 * P + 32.0 * case["n"], "flops": rays * RAY_FLOPS}
    if kind in ("frame", "device", "host"):
        b["bytes"] += state + (4.0 * case["w"] * case["h"] if kind == "frame" else 0.0)
    elif kind == "denoise":
        b["flops"] += rows * NET_FLOPS
    elif kind == "adaptive":
        b["bytes"] += rows
        b["flops"] += rows * NET_FLOPS
    else:
        b["bytes"] = rows * (112 * 2 + 24.0) + 12.0 * _COUNT
        b["flops"] = rows * (case["spp"] + case["target_spp"]) * RAY_FLOPS + 3.0 * NET_FLOPS * case["steps"] * min(case["batch"], rows)
    return b


def exact(case, seed):
    """None: every output is a Monte-Carlo mean over cuRAND's streams (or a
    network fed with such means), which only the library draws."""
    return None
