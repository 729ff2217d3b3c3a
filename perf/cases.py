"""What a user of this framework has it do, as cases to be timed and compared.

Kinds of case (``case["kind"]``), each through the package's public classes:

* ``dropin``    ReconFlow: frames from host memory, solve, flow and points back to host
* ``flow``      CudaFlow: plain TV-L1 flow of a frame pair, host to host
* ``batch``     ReconFlowBatch: plain solve of pairs of several sizes, frames in HBM
* ``learned``   LearnedBatchSolver: features, network, warm state, refinement, energies
* ``sequence``  the next wave of frame sequences: the previous wave's depth carried
                into the new frames, warm state, refinement, energies
* ``network``   WarmStartNet.forward
* ``train``     WarmStartNet.backward and adam_step
* ``pose``      CameraPose: features, matching, essential matrix, pose, from host frames

Frames are made on the GPU from the seed: a smooth random texture of several
octaves is the second frame, and the first one samples it through the flow that a
piecewise-planar scene (inverse depth 0.1 .. 0.5 1/m) and a rigid motion give, with
N(0, 0.01) noise on both, as the package's own scene generator has them.
"""
import json
import math
import os

import numpy as np
import torch
import torch.nn.functional as F

import reconflow_gb300 as R
from reconflow_gb300 import autotune, warmstart
from reconflow_gb300.reconflow import CV_8U, CV_8UC3, CV_16U, CV_32F

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHECKPOINT = os.path.join(ROOT, "reconflow_gb300", "weights", "warmstart_f125.bin")
TILES_SINGLE = os.path.join(ROOT, "reconflow_gb300", "tuning", "gb300_720p_single.json")
TILES_BATCH = os.path.join(ROOT, "reconflow_gb300", "tuning", "gb300_720p_x64.json")
# the solver weights of the repository's workloads (theta = 0.33)
WEIGHTS = dict(lambda_=50.0, lambdaf=0.1, lambdams=100.0, alphaTv=1 / 0.33, alphaProj=60.0,
               tau=0.25, fix_quirks=1)
CV = {"f32": CV_32F, "u8": CV_8U, "u16": CV_16U, "rgb8": CV_8UC3}
# per pixel and inner iteration: 13 state planes read and written, 5 planes of the warp read
ITER_BYTES, ITER_FLOPS = 124, 420
# plain TV-L1: 6 state planes read and written, 3 planes of the warp read
FLOW_BYTES, FLOW_FLOPS = 60, 70


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest call: a thumbnail pair, a few iterations; launches and copies decide
        dict(name="dropin_96x72", kind="dropin", w=96, h=72, levels=3, warps=2, iters=5,
             method=14, input="f32"),
        # the 640x480 workload: 5 levels, 3 warps, 50 iterations
        dict(name="dropin_640x480", kind="dropin", w=640, h=480, levels=5, warps=3, iters=50,
             method=14, input="f32"),
        # the plain 720p workload: one pair, 6 levels, 5 warps, 100 iterations
        dict(name="dropin_1280x720", kind="dropin", w=1280, h=720, levels=6, warps=5, iters=100,
             method=14, input="f32"),
        # a video frame (8-bit colour) of ragged size with a prior flow from elsewhere
        dict(name="prior_451x333_rgb8", kind="dropin", w=451, h=333, levels=4, warps=3, iters=50,
             method=17, input="rgb8"),
        # flow only, 8-bit colour, the plain TV-L1 class
        dict(name="flow_640x480_rgb8", kind="flow", w=640, h=480, levels=5, warps=3, iters=50,
             input="rgb8"),
        # offline reconstruction of pairs of mixed sizes, plain schedule
        dict(name="batch_mixed_x12", kind="batch", sizes="320x240,640x480,1280x720,1920x1080",
             n=12, levels=6, warps=5, iters=100),
        # throughput serving: 64 720p pairs with the learned warm start, frames in HBM
        dict(name="learned_1280x720_x64", kind="learned", w=1280, h=720, n=64, level=1,
             iters="3,50", host=False),
        # one 720p pair at a time with the learned warm start, host to host: latency
        dict(name="learned_1280x720_x1", kind="learned", w=1280, h=720, n=1, level=1,
             iters="3,50", host=True),
        # two 4K sequences, one wave
        dict(name="sequence_3840x2160_x2", kind="sequence", w=3840, h=2160, n=2, level=3,
             iters="4,30,60,80"),
        # the network alone on the inputs of 64 720p pairs
        dict(name="network_160x90_x64", kind="network", w=160, h=90, n=64),
        # one training step at the training set's size and batch
        dict(name="train_160x120_x64", kind="train", w=160, h=120, n=64),
        # the pose front end, one 720p pair
        dict(name="pose_1280x720", kind="pose", w=1280, h=720),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "dropin", "flow", "batch", "learned", "learned", "sequence",
                       "network", "train", "pose"])
    if kind in ("dropin", "flow"):
        w, h = _log(rng, 80, 1280), 0
        h = max(60, min(720, int(w * rng.uniform(0.5, 1.0))))
        c = dict(kind=kind, w=w, h=h, levels=rng.randint(2, 5), warps=rng.randint(1, 5),
                 iters=_log(rng, 4, 100), input=rng.choice(["f32", "f32", "rgb8", "u8", "u16"]))
        if kind == "dropin":
            c["method"] = rng.choice([14, 14, 17, 20])
        return c
    if kind == "batch":
        n = rng.randint(2, 12)
        sizes = ",".join("%dx%d" % (_log(rng, 160, 1280), _log(rng, 120, 720))
                         for _ in range(rng.randint(1, 4)))
        return dict(kind=kind, sizes=sizes, n=n, levels=rng.randint(3, 5), warps=rng.randint(1, 4),
                    iters=_log(rng, 10, 100))
    if kind == "learned":
        w, h = rng.choice([(640, 480), (1280, 720), (1920, 1080),
                           (rng.randint(500, 1280), rng.randint(300, 720))])
        n = _log(rng, 1, 64) if w <= 1280 else _log(rng, 1, 16)
        level = 2 if w > 1280 else 1
        iters = [rng.randint(2, 6), rng.randint(20, 60), rng.randint(40, 80)][:level + 1]
        return dict(kind=kind, w=w, h=h, n=n, level=level, iters=",".join(map(str, iters)),
                    host=rng.random() < 0.3)
    if kind == "sequence":
        w, h = rng.choice([(1920, 1080), (1280, 720), (2560, 1440)])
        return dict(kind=kind, w=w, h=h, n=rng.randint(1, 4), level=2,
                    iters="%d,%d,%d" % (rng.randint(2, 6), rng.randint(20, 60),
                                        rng.randint(40, 80)))
    if kind == "network":
        return dict(kind=kind, w=rng.randint(60, 200), h=rng.randint(40, 120), n=_log(rng, 1, 64))
    if kind == "train":
        return dict(kind=kind, w=rng.randint(60, 160), h=rng.randint(45, 120),
                    n=rng.choice([8, 16, 32, 48, 64]))
    return dict(kind=kind, w=rng.randint(320, 1280), h=rng.randint(240, 720))


def _sizes(c):
    s = [tuple(map(int, t.split("x"))) for t in c["sizes"].split(",")]
    return [s[i % len(s)] for i in range(c["n"])]


def _level_sizes(w, h, levels):
    out = []
    for _ in range(levels):
        out.append((w, h))
        w, h = w // 2, h // 2
    return out


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _texture(w, h, g):
    """Random octaves, wavelengths 6 px to the image's size, in [0, 1]."""
    img = torch.zeros((1, 1, h, w), device="cuda")
    wave = 6.0
    while wave < max(w, h):
        gh, gw = max(2, int(h / wave) + 2), max(2, int(w / wave) + 2)
        grid = torch.randn((1, 1, gh, gw), device="cuda", generator=g)
        img += wave ** 0.5 * F.interpolate(grid, size=(h, w), mode="bicubic", align_corners=True)
        wave *= 1.9
    img = img[0, 0]
    return (0.5 + img / (5.0 * img.std())).clamp(0.0, 1.0)


def _rotation(axis, angle):
    a = axis / np.linalg.norm(axis)
    K = np.array([[0, -a[2], a[1]], [a[2], 0, -a[0]], [-a[1], a[0], 0]])
    return np.eye(3) + math.sin(angle) * K + (1 - math.cos(angle)) * (K @ K)


def _pair(w, h, seed, trans=0.1, max_deg=2.0):
    """One frame pair: frames (h, w) on the GPU, K, R, t and the first frame's inverse depth."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    f = 500.0 * w / 640.0
    K = np.array([[f, 0, w / 2.0], [0, f, h / 2.0], [0, 0, 1]])
    Rm = _rotation(rng.normal(size=3), math.radians(rng.uniform(0.0, max_deg)))
    t = rng.normal(size=3)
    t *= trans / np.linalg.norm(t)
    I1 = _texture(w, h, g)
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float32),
                          torch.arange(w, device="cuda", dtype=torch.float32), indexing="ij")
    # eight planes over a Voronoi partition of the image
    best = torch.full((h, w), float("inf"), device="cuda")
    rho = torch.zeros((h, w), device="cuda")
    for _ in range(8):
        cx, cy = rng.uniform(0, w), rng.uniform(0, h)
        a, b, c = rng.uniform(0.2, 0.4), rng.uniform(-0.1, 0.1) / w, rng.uniform(-0.1, 0.1) / h
        d = (x - cx) ** 2 + (y - cy) ** 2
        near = d < best
        best = torch.where(near, d, best)
        rho = torch.where(near, a + b * (x - w / 2) + c * (y - h / 2), rho)
    rho = rho.clamp(0.1, 0.5)
    A, b = K @ Rm @ np.linalg.inv(K), K @ t
    q = [A[i, 0] * x + A[i, 1] * y + A[i, 2] + rho * b[i] for i in range(3)]
    gx, gy = (q[0] / q[2] + 0.5) * (2.0 / w) - 1.0, (q[1] / q[2] + 0.5) * (2.0 / h) - 1.0
    I0 = F.grid_sample(I1[None, None], torch.stack([gx, gy], -1)[None], mode="bicubic",
                       padding_mode="reflection", align_corners=False)[0, 0]
    I0 = I0 + 0.01 * torch.randn((h, w), device="cuda", generator=g)
    I1 = I1 + 0.01 * torch.randn((h, w), device="cuda", generator=g)
    return I0, I1, K, Rm, t, rho


def _stride(w):
    return (w + 31) // 32 * 32


def _pinned(shape, dtype=torch.float32):
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _host_frame(img, kind):
    """A frame (h, w) in host memory as a capture card delivers it, rows padded to 32 pixels."""
    h, w = img.shape
    s = _stride(w)
    if kind == "f32":
        out = _pinned((h, s))
        out[:, :w] = img.cpu().numpy()
    elif kind == "u16":
        out = np.zeros((h, s), np.uint16)
        out[:, :w] = (img.clamp(0, 1) * 65535).round().cpu().numpy().astype(np.uint16)
    elif kind == "u8":
        out = np.zeros((h, s), np.uint8)
        out[:, :w] = (img.clamp(0, 1) * 255).round().cpu().numpy().astype(np.uint8)
    else:
        out = np.zeros((h, s, 3), np.uint8)
        gain = torch.tensor([0.9, 1.0, 0.8], device="cuda")
        out[:, :w] = (img[..., None].clamp(0, 1) * gain * 255).round().cpu().numpy().astype(np.uint8)
    return out


class _Plane:
    """Device memory of the library as an array that torch can view; `owner` lives as long."""

    def __init__(self, ptr, shape, strides, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(
            shape=shape, typestr="<f4", data=(int(ptr), False), version=3,
            strides=tuple(4 * s for s in strides))


def _view(ptr, shape, strides, owner):
    return torch.as_tensor(_Plane(ptr, shape, strides, owner), device="cuda")


def _table(path):
    """The tile shapes of a committed autotuner table."""
    with open(path) as f:
        return json.load(f)["levels"]


def _upload(batch, i, I0, I1):
    torch.cuda.synchronize()
    batch.copyImagesToDeviceFromDevice(i, I0.data_ptr(), I1.data_ptr(), I0.shape[1])
    batch.synchronize()


def _net_batch(c, seed):
    """Network inputs and targets as the features and the plain solver's results have them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n, h, w = c["n"], c["h"], c["w"]

    def smooth(ch, hh, ww, cell):
        a = torch.randn((n, ch, max(2, hh // cell), max(2, ww // cell)), device="cuda", generator=g)
        return F.interpolate(a, size=(hh, ww), mode="bilinear", align_corners=True)

    x = torch.cat([0.2 * smooth(2, h, w, 6), 1.2 * smooth(12, h, w, 4).abs(),
                   2.0 * smooth(2, h, w, 32)], 1).permute(0, 2, 3, 1).contiguous()
    h2, w2 = (h + 1) // 2, (w + 1) // 2

    def target(hh, ww, s):
        t = torch.zeros((n, hh, ww, 8), device="cuda")
        t[..., :2] = s * smooth(2, hh, ww, 12).permute(0, 2, 3, 1)
        t[..., 2] = (0.25 + 0.05 * smooth(1, hh, ww, 12)[:, 0]).clamp(0.1, 0.5)
        m = (torch.rand((n, hh, ww), device="cuda", generator=g) > 0.05).float()
        return t * m[..., None], m

    t8, m8 = target(h, w, 2.0)
    t16, m16 = target(h2, w2, 1.0)
    return x, t16, m16, t8, m8


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](dict(case), int(seed))


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _prepare_dropin(c, seed):
    I0, I1, K, Rm, t, rho = _pair(c["w"], c["h"], seed)
    s = dict(c, R=Rm, t=t, frames=[_host_frame(I, c["input"]) for I in (I0, I1)])
    f = R.ReconFlow()
    f.initializeR(c["w"], c["h"], 3 if c["input"] == "rgb8" else 1, c["levels"], 2.0, c["method"],
                  WEIGHTS["lambda_"], 0.0, WEIGHTS["lambdaf"], WEIGHTS["lambdams"],
                  WEIGHTS["alphaTv"], WEIGHTS["alphaProj"], 0.5, WEIGHTS["tau"], c["warps"],
                  c["iters"], cvType=CV[c["input"]], fix_quirks=1)
    f.setCameraMatrices(K, K)
    if (c["w"], c["h"], c["levels"]) == (1280, 720, 6):
        autotune.apply_single(f, _table(TILES_SINGLE), c["levels"])
    if c["method"] != 14:
        # a prior flow such as a network or a sparse matcher gives: the scene's, 0.3 px off
        h, w = c["h"], c["w"]
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed) + 1)
        y, x = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"),
                              indexing="ij")
        A, b = K @ Rm @ np.linalg.inv(K), K @ t
        q = [A[i, 0] * x + A[i, 1] * y + A[i, 2] + rho * b[i] for i in range(3)]
        uv = [q[0] / q[2] - x, q[1] / q[2] - y]
        uv = [p + 0.3 * torch.randn((h, w), device="cuda", generator=g) for p in uv]
        mask = None
        if c["method"] == 20:
            mask = np.zeros((h, _stride(w)), np.float32)
            mask[:, :w] = (torch.rand((h, w), device="cuda", generator=g) < 0.2).float().cpu().numpy()
        s["prior"] = [_host_frame(p, "f32") for p in uv] + [mask]
    s["flow"] = f
    s["out"] = [_pinned((c["h"], _stride(c["w"]))) for _ in range(5)]
    return s


def _run_dropin(s):
    f, o = s["flow"], s["out"]
    f.copyImagesToDevice(*s["frames"])
    if "prior" in s:
        f.copySparseOpticalFlowToDevice(*s["prior"])
    f.solveR(s["R"], s["t"], 5.0)
    f.copyOpticalFlowToHost(o[0], o[1])
    f.copy3dToHost(o[2], o[3], o[4])
    return dict(zip("uvXYZ", o))


def _prepare_flow(c, seed):
    I0, I1 = _pair(c["w"], c["h"], seed)[:2]
    f = R.CudaFlow()
    f.initialize(c["w"], c["h"], 3 if c["input"] == "rgb8" else 1, CV[c["input"]], c["levels"], 2.0,
                 lambda_=50.0, theta=0.33, tau=0.25, nWarpIters=c["warps"], nSolverIters=c["iters"])
    return dict(c, flow=f, frames=[_host_frame(I, c["input"]) for I in (I0, I1)],
                out=[_pinned((c["h"], _stride(c["w"]))) for _ in range(2)])


def _run_flow(s):
    f, o = s["flow"], s["out"]
    f.copyImagesToDevice(*s["frames"])
    f.solveOpticalFlow()
    f.copyOpticalFlowToHost(o[0], o[1])
    return {"u": o[0], "v": o[1]}


def _prepare_batch(c, seed):
    sizes = _sizes(c)
    b = R.ReconFlowBatch(sizes, c["levels"], method=14, nWarpIters=c["warps"],
                         nSolverIters=c["iters"], **WEIGHTS)
    Rs, ts = [], []
    for i, (w, h) in enumerate(sizes):
        I0, I1, K, Rm, t, _ = _pair(w, h, seed * 1000 + i)
        b.setCameraMatrices(i, K, K)
        _upload(b, i, I0, I1)
        Rs.append(Rm)
        ts.append(t)
    return dict(c, batch=b, pairs=sizes, R=Rs, t=ts)


def _run_batch(s):
    b = s["batch"]
    b.solveR(s["R"], s["t"])
    out = {}
    for i, (w, h) in enumerate(s["pairs"]):
        for k, p in zip("uvXYZ", b.deviceResults(i)):
            out["%s%d" % (k, i)] = _view(p, (h, w), (b.strides[i], 1), b)
    return out


def _batch_planes(b, w, h):
    """Every pair's u, v, X, Y, Z on the device: one (n, h, w) view per field."""
    first = b.deviceResults(0)
    step = (b.deviceResults(1)[0] - first[0]) // 4 if b.n > 1 else 1
    return {k: _view(p, (b.n, h, w), (step, b.strides[0], 1), b) for k, p in zip("uvXYZ", first)}


def _refinement(c, seed, levels=6):
    """A batch of pairs of one size, its scenes, and the network's handle."""
    w, h, n = c["w"], c["h"], c["n"]
    iters = [int(x) for x in c["iters"].split(",")]
    b = R.ReconFlowBatch([(w, h)] * n, levels, method=14, nWarpIters=1, nSolverIters=iters[0],
                         **WEIGHTS)
    autotune.apply(b, _table(TILES_BATCH))
    scenes = [_pair(w, h, seed * 1000 + i, *((0.05, 0.3) if c["kind"] == "sequence" else ()))
              for i in range(n)]
    for i, sc in enumerate(scenes):
        b.setCameraMatrices(i, sc[2], sc[2])
        _upload(b, i, sc[0], sc[1])
    return b, scenes, iters


def _prepare_learned(c, seed):
    b, scenes, iters = _refinement(c, seed)
    K = scenes[0][2]
    fac = warmstart.net_factor(K)
    net = warmstart.WarmStartNet(c["n"], c["h"] // fac, c["w"] // fac)
    net.load(CHECKPOINT)
    ls = warmstart.LearnedBatchSolver(net, b, (c["w"], c["h"]), K, warm_level=c["level"],
                                      warps=[1] * len(iters), iters=iters)
    s = dict(c, batch=b, solver=ls, K=[sc[2] for sc in scenes], R=[sc[3] for sc in scenes],
             t=[sc[4] for sc in scenes], net=net)
    if c["host"]:
        st = _stride(c["w"])
        s["in"] = [[_host_frame(sc[k], "f32") for sc in scenes] for k in (0, 1)]
        s["out"] = _pinned((6, c["n"], c["h"], st))
        s["ptrs"] = [[a.ctypes.data for a in col] for col in s["in"]] + \
                    [[s["out"][k, i].ctypes.data for i in range(c["n"])] for k in range(6)]
        s["pitch"] = st
    return s


def _run_learned(s):
    b = s["batch"]
    if s["host"]:
        b.uploadAll(s["ptrs"][0], s["ptrs"][1], s["pitch"])
    s["solver"].solve(s["K"], s["R"], s["t"])
    energy = b.energies()
    if s["host"]:
        b.downloadAll(s["pitch"], *s["ptrs"][2:])
        return {"results": s["out"], "energy": energy}
    return dict(_batch_planes(b, s["w"], s["h"]), energy=energy)


def _prepare_sequence(c, seed):
    b, scenes, iters = _refinement(c, seed)
    n, w, h = c["n"], c["w"], c["h"]
    fac = warmstart.net_factor(scenes[0][2])
    lw, lh, ls = b.levelDims(0, c["level"])
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    # the previous wave's solution: the scene's depth, 1% off, from 5 cm further back
    depth = [(1.0 / sc[5] + 0.05) * (1.0 + 0.01 * torch.randn((h, w), device="cuda", generator=g))
             for sc in scenes]
    s = dict(c, batch=b, depth=depth, K=[sc[2] for sc in scenes],
             R=[sc[3] for sc in scenes], t=[sc[4] for sc in scenes], factor=fac, lw=lw, lh=lh, ls=ls,
             R_prev=[_rotation(rng.normal(size=3), math.radians(0.2)) for _ in range(n)],
             t_prev=[np.array([0.0, 0.0, -0.05]) for _ in range(n)], iters_=iters,
             grid=torch.zeros((n, h // fac, w // fac, 3), device="cuda"),
             scratch=torch.zeros(2 * n * (h // fac) * (w // fac), dtype=torch.int32, device="cuda"),
             planes=[b.warmPlanes(i) for i in range(n)])
    s["K_level"] = [warmstart.level_intrinsics(K, c["level"]) for K in s["K"]]
    torch.cuda.synchronize()
    return s


def _run_sequence(s):
    b, st = s["batch"], s["batch"].stream()
    warmstart.propagate([d.data_ptr() for d in s["depth"]], s["w"], s["h"], s["w"], s["K"],
                        s["R_prev"], s["t_prev"], s["factor"], s["grid"], stream=st,
                        scratch=s["scratch"])
    warmstart.state(s["grid"], s["lw"], s["lh"], s["ls"], s["factor"] / 2.0 ** s["level"],
                    s["K_level"], s["R"], s["t"], s["planes"], st)
    b.solveWarm(s["level"], s["R"], s["t"], 1, s["iters_"])
    energy = b.energies()
    return dict(_batch_planes(b, s["w"], s["h"]), energy=energy, grid=s["grid"])


def _prepare_network(c, seed):
    net = warmstart.WarmStartNet(c["n"], c["h"], c["w"])
    net.load(CHECKPOINT)
    x = _net_batch(c, seed)[0]
    o16 = torch.empty((c["n"], (c["h"] + 1) // 2, (c["w"] + 1) // 2, 8), device="cuda")
    o8 = torch.empty((c["n"], c["h"], c["w"], 8), device="cuda")
    return dict(c, net=net, x=x, o16=o16, o8=o8)


def _run_network(s):
    s["net"].forward(s["x"], s["o16"], s["o8"])
    return {"o16": s["o16"], "o8": s["o8"]}


def _prepare_train(c, seed):
    net = warmstart.WarmStartNet(c["n"], c["h"], c["w"])
    net.load(CHECKPOINT)
    return dict(c, net=net, data=_net_batch(c, seed))


def _run_train(s):
    # a fine-tuning step; the gradients and the updated weights come back whole
    loss = s["net"].backward(*s["data"])
    s["net"].adam_step(1e-4)
    return {"loss": loss, "grads": s["net"].grads(), "params": s["net"].params()}


def _prepare_pose(c, seed):
    I0, I1, K = _pair(c["w"], c["h"], seed)[:3]
    p = R.CameraPose()
    p.initialize(K, 20.0)
    # the matches go into arrays for as many keypoints as a frame may have (1% of its pixels)
    most = c["w"] * c["h"] // 100 + 1
    return dict(c, pose=p, frames=[I.clamp(0, 1).cpu().numpy() for I in (I0, I1)],
                out=[np.zeros(most, t) for t in (np.int32, np.int32, np.float32, np.uint8)])


def _run_pose(s):
    found, Rm, t = s["pose"].solvePose_f32(*s["frames"])
    got = s["pose"].matches()
    for a, m in zip(s["out"], got):
        a[:len(m)] = m
        a[len(m):] = 0
    return {"found": int(found), "R": np.zeros((3, 3)) if Rm is None else Rm,
            "t": np.zeros(3) if t is None else t, "matches": len(got[0]),
            **dict(zip(("i0", "i1", "dist", "inlier"), s["out"]))}


# ---------------------------------------------------------------------------
# work: what a pass cannot do without
# ---------------------------------------------------------------------------

def _net_macs(c):
    p, q = c["n"] * c["h"] * c["w"], c["n"] * ((c["h"] + 1) // 2) * ((c["w"] + 1) // 2)
    return 9 * (p * (16 * 32 + 128 * 64 + 64 * 8) + q * (32 * 96 + 96 * 96 + 96 * 8))


def work(case):
    c, k = case, case["kind"]
    if k in ("dropin", "flow", "batch"):
        sizes = _sizes(c) if k == "batch" else [(c["w"], c["h"])]
        px = sum(w * h for w, h in sizes)
        it = c["warps"] * c["iters"] * sum(a * b for w, h in sizes
                                           for a, b in _level_sizes(w, h, c["levels"]))
        per = (FLOW_BYTES, FLOW_FLOPS) if k == "flow" else (ITER_BYTES, ITER_FLOPS)
        return {"bytes": it * per[0] + px * 4 * (4 if k == "flow" else 7), "flops": it * per[1]}
    if k in ("learned", "sequence"):
        px = c["w"] * c["h"] * c["n"]
        it = sum(int(n) * px / 4 ** l for l, n in enumerate(c["iters"].split(",")))
        flops = it * ITER_FLOPS
        if k == "learned":
            K = np.array([[500.0 * c["w"] / 640.0]])
            fac = warmstart.net_factor(K)
            flops += 2 * _net_macs(dict(n=c["n"], h=c["h"] // fac, w=c["w"] // fac))
        return {"bytes": it * ITER_BYTES + px * 4 * 7, "flops": flops}
    if k == "network":
        return {"bytes": c["n"] * c["h"] * c["w"] * 4 * (16 + 8 + 2), "flops": 2 * _net_macs(c)}
    if k == "train":
        return {"bytes": c["n"] * c["h"] * c["w"] * 4 * (16 + 9 + 9 // 4), "flops": 6 * _net_macs(c)}
    # pose: both frames in; four octaves of four box-filter layers, about 60 operations each
    px = c["w"] * c["h"]
    return {"bytes": 2 * px * 4, "flops": 2 * px * 4 * 60 * 4 / 3}


# ---------------------------------------------------------------------------
# exact: the same in 64 bits
# ---------------------------------------------------------------------------

def exact(case, seed):
    """The ReconFlow solves (dropin, batch, learned, sequence) have no value here: their 3x3
    point solves start from coincident points, so a solution in 64 bits is another one at many
    pixels (the flow of a cold start differs by hundreds of pixels at the worst of them).  The
    pose is a choice among seeded samples."""
    c, k = dict(case), case["kind"]
    if k == "flow":
        return _exact_flow(c, seed)
    if k == "network":
        o16, o8, _ = _net64(_params64(), _net_batch(c, seed)[0].double())
        return {"o16": o16, "o8": o8}
    if k == "train":
        return _exact_train(c, seed)
    return None


def _params64():
    with open(CHECKPOINT, "rb") as f:
        f.seek(28)
        return torch.from_numpy(np.frombuffer(f.read(), np.float32).copy()).cuda().double()


def _net64(p, x):
    """(out16, out8, layers): the network as convolutions over NCHW, parameters in one vector."""
    layers, off = [], 0
    for cin, cout in ((16, 32), (32, 96), (96, 96), (96, 8), (128, 64), (64, 8)):
        W = p[off:off + cout * 9 * cin].view(cout, 3, 3, cin).permute(0, 3, 1, 2)
        off += cout * 9 * cin
        layers.append((W, p[off:off + cout]))
        off += cout

    def conv(a, i, stride=1):
        # nine shifted matrix products: FP64 convolutions of the library are slow
        (W, b), (n, ch, h, w) = layers[i], a.shape
        ap = F.pad(a, (1, 1, 1, 1))
        ho, wo = (h + stride - 1) // stride, (w + stride - 1) // stride
        out = b[None, :, None, None]
        for ky in range(3):
            for kx in range(3):
                sl = ap[:, :, ky:ky + (ho - 1) * stride + 1:stride, kx:kx + (wo - 1) * stride + 1:stride]
                out = out + torch.einsum("oc,nchw->nohw", W[:, :, ky, kx], sl)
        return out

    h, w = x.shape[1:3]
    a1 = conv(x.permute(0, 3, 1, 2), 0).relu()
    a3 = conv(conv(a1, 1, 2).relu(), 2).relu()
    o16 = conv(a3, 3)
    up = a3.repeat_interleave(2, 2).repeat_interleave(2, 3)[:, :, :h, :w]
    o8 = conv(conv(torch.cat([up, a1], 1), 4).relu(), 5)
    return o16.permute(0, 2, 3, 1), o8.permute(0, 2, 3, 1), layers


def _exact_train(c, seed):
    x, t16, m16, t8, m8 = (a.double() for a in _net_batch(c, seed))
    wts = torch.tensor(warmstart.LOSS_WEIGHTS, device="cuda", dtype=torch.float64)
    p0 = _params64()
    grad, loss = torch.zeros_like(p0), 0.0
    for i in range(0, c["n"], 4):  # a few images at a time: the graph of 64 is large
        p = p0.clone().requires_grad_(True)
        part = 0.0
        o16, o8, _ = _net64(p, x[i:i + 4])
        for o, t, m in ((o16, t16, m16), (o8, t8, m8)):
            d = (o[..., :3] - t[i:i + 4, ..., :3]).abs() * wts * (m[i:i + 4, ..., None] > 0)
            part = part + d.sum() / m.numel()
        part.backward()
        grad += p.grad
        loss += float(part.detach())
    # the first Adam step
    m, v = 0.1 * grad, 0.001 * grad * grad
    params = p0 - 1e-4 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
    return {"loss": loss, "grads": grad, "params": params}


def _mirror(i, n):
    i = torch.remainder(i, 2 * n)
    return torch.where(i < n, i, 2 * n - 1 - i)


def _taps(tn, n):
    t = tn.abs().remainder(2.0)
    t = torch.where(t > 1.0, 2.0 - t, t) * n - 0.5
    i = t.floor()
    return _mirror(i.long(), n), _mirror(i.long() + 1, n), t - i


def _tex(img, xn, yn):
    """Bilinear samples at normalized coordinates, mirrored at the edges."""
    h, w = img.shape
    x0, x1, a = _taps(xn, w)
    y0, y1, b = _taps(yn, h)
    return ((1 - b) * ((1 - a) * img[y0, x0] + a * img[y0, x1])
            + b * ((1 - a) * img[y1, x0] + a * img[y1, x1]))


def _grid64(w, h):
    y, x = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float64),
                          torch.arange(w, device="cuda", dtype=torch.float64), indexing="ij")
    return x, y


def _deriv(a, dim):
    n = a.shape[dim]
    at = torch.arange(n, device="cuda")
    t = [a.index_select(dim, _mirror(at + k, n)) for k in (-2, -1, 1, 2)]
    return (t[0] - 8 * t[1] + 8 * t[2] - t[3]) / 12


def _median5(a):
    """5x5 median: a tap off one side takes the nearest pixel, one off both is zero."""
    h, w = a.shape
    p = F.pad(a[None, None], (2, 2, 2, 2), mode="replicate")[0, 0]
    p[:2, :2] = p[:2, w + 2:] = p[h + 2:, :2] = p[h + 2:, w + 2:] = 0
    return torch.stack([p[j:j + h, i:i + w] for j in range(5) for i in range(5)]).median(0).values


def _exact_flow(c, seed):
    w, h, lam, theta, tau = c["w"], c["h"], 50.0, 0.33, 0.25
    pyr = []
    for I in _pair(w, h, seed)[:2]:
        a = torch.from_numpy(_host_frame(I, c["input"])[:, :w].astype(np.float64)).cuda()
        if c["input"] == "rgb8":
            a = a.mean(-1)
        lv = [a / {"f32": 1.0, "u16": 65536.0}.get(c["input"], 256.0)]
        for lw, lh in _level_sizes(w, h, c["levels"])[1:]:
            x, y = _grid64(lw, lh)
            x, y, dx, dy = (x + 0.5) / lw, (y + 0.5) / lh, 0.25 / lw, 0.25 / lh
            f = lv[-1]
            lv.append(0.25 * (_tex(f, x - dx, y) + _tex(f, x + dx, y)
                              + _tex(f, x, y - dy) + _tex(f, x, y + dy)))
        pyr.append(lv)
    u = v = None
    for l in range(c["levels"] - 1, -1, -1):
        I0, I1 = pyr[0][l], pyr[1][l]
        lh, lw = I0.shape
        x, y = _grid64(lw, lh)
        xn, yn = (x + 0.5) / lw, (y + 0.5) / lh
        u = torch.zeros_like(I0) if u is None else 2 * _tex(u, xn, yn)
        v = torch.zeros_like(I0) if v is None else 2 * _tex(v, xn, yn)
        for _ in range(c["warps"]):
            W = _tex(I1, (x + u + 0.5) / lw, (y + v + 0.5) / lh)
            Ix, Iy = 0.5 * (_deriv(I0, 1) + _deriv(W, 1)), 0.5 * (_deriv(I0, 0) + _deriv(W, 0))
            It, mag = W - I0, Ix * Ix + Iy * Iy
            d = [torch.zeros_like(I0), torch.zeros_like(I0)]
            p = [torch.zeros_like(I0) for _ in range(4)]
            for _ in range(c["iters"]):
                r = Ix * d[0] + Iy * d[1] + It
                k = torch.where(r < -lam * theta * mag, lam * theta,
                                torch.where(r > lam * theta * mag, -lam * theta,
                                            torch.where(mag > 0, -r / mag.clamp_min(1e-300), 0.0)))
                for i, g in enumerate((Ix, Iy)):
                    div = p[2 * i] + p[2 * i + 1]
                    div[:, 1:] -= p[2 * i][:, :-1]
                    div[1:] -= p[2 * i + 1][:-1]
                    d[i] = d[i] + k * g + theta * div
                for i in range(2):
                    gx, gy = torch.zeros_like(I0), torch.zeros_like(I0)
                    gx[:, :-1] = d[i][:, 1:] - d[i][:, :-1]
                    gy[:-1] = d[i][1:] - d[i][:-1]
                    den = 1 + tau / theta * (gx * gx + gy * gy).sqrt()
                    p[2 * i] = (p[2 * i] + tau / theta * gx) / den
                    p[2 * i + 1] = (p[2 * i + 1] + tau / theta * gy) / den
            u, v = u + _median5(d[0]), v + _median5(d[1])
    out = []
    for a in (u, v):
        full = torch.zeros((h, _stride(w)), device="cuda", dtype=torch.float64)
        full[:, :w] = a
        out.append(full)
    return {"u": out[0], "v": out[1]}
