"""The work that a user of this library has it do, as timed cases over its public entry points.

Every case is a dict of plain values whose "kind" names one path of the library:

* ``frames``     the radiance-cache frame loop of a box room (Context.begin / frame), what a renderer
                 calls every frame: all of the timing table's methods, light and geometry events,
                 1 to 16 rays per point; the cache, the histories and the dependency masks come back
                 as the context's own device buffers
* ``mesh``       the same loop over a triangle mesh that the library prepared itself (static BVH,
                 hash-table cache points), the size of a street or of city blocks
* ``trace``      closest hits of caller-given rays against such a mesh (picking, visibility)
* ``taa``        the screen-space temporal accumulator's run, its error read every frame
* ``reference``  the converged references of a scene's states (scene preparation)
* ``paths``      one image of camera paths fed into the hash-grid cache, then the cache's resolve
* ``hashgrid``   one frame of samples inserted, accumulated and resolved in a hash-grid cache
* ``infer``      the learned cache's network at every cache point
* ``train``      the learned cache's training steps of one frame
* ``adjoint``    the gradient of the cached radiance with respect to every light

The box room and the city mesh are the library's own generators; the sizes are those of its
benchmark and of its scene files (10 k, 43 k, 170 k and 1.08 M cache points), or lie between them.
"""
import math
import os
import random
import tempfile

import numpy as np
import torch

from render_engine_gb300 import hashgrid as H
from render_engine_gb300 import methods as M
from render_engine_gb300 import mlp as MLP
from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

TIMING = {m.name: m for m in M.timing_methods()}
HEADLINE = "v4-A2C suivi 1/4"


def listed():
    return [
        # a small room's cache, the size of the reference's own box scenes: per-frame latency and
        # launches; twelve frames, a lamp goes out, four more
        {"name": "frames_small", "kind": "frames", "points": 10_728, "lights": 3, "method": HEADLINE, "seq": "0x12 1x4", "rays": 1.0},
        # the headline workload: 1.08 M points, 3 lights, dependencies tracked one frame in four,
        # a lamp switched off on the way
        {"name": "frames_1m", "kind": "frames", "points": 1_082_802, "lights": 3, "method": HEADLINE, "seq": "0x12 1x4", "rays": 1.0},
        # 8 lights, every frame tracked, the occluder moves: the event's own kernels and the
        # verification frames after it (per-zone sums, decision), at an odd size
        {"name": "frames_8_lights", "kind": "frames", "points": 213_457, "lights": 8, "method": "v3 complet", "seq": "1x4 2x8", "rays": 1.0},
        # a street-sized mesh prepared by the library: 250 k triangles, 8 lamps, half a million
        # points, the tree traversal ahead of every frame
        {"name": "mesh_250k", "kind": "mesh", "buildings": 100, "points": 500_000, "lamps": 8, "method": HEADLINE, "seq": "0x6 1x4"},
        # closest hits of a batch of incoherent rays given in host memory
        {"name": "trace_rays", "kind": "trace", "buildings": 100, "points": 60_000, "rays": 262_144},
        # the screen-space accumulator over the large room with the dependency mask: 24 frames, an
        # event in the middle, the error of each frame read back
        {"name": "taa_1m", "kind": "taa", "points": 1_082_802, "mask": 2, "seq": "0x12 1x12"},
        # the references of a 43 k-point room's five states at the preparation's own settings
        {"name": "reference_43k", "kind": "reference", "points": 43_000, "lights": 3, "K": 32, "block": 64},
        # one 1080p image of camera paths with two bounces, a rectangle light and a sun, into a
        # 2^22-entry hash grid with voxel light masks, and its resolve
        {"name": "paths_1080p", "kind": "paths", "width": 1920, "height": 1080, "points": 170_185, "log2_capacity": 22, "bounces": 2},
        # a frame of a large hash-grid cache: a million samples into 2^24 slots, half of them live
        {"name": "hashgrid_16m", "kind": "hashgrid", "log2_capacity": 24, "live": 0.5, "samples": 1_000_003, "event": False},
        # the learned cache served at every point of the large room
        {"name": "infer_1m", "kind": "infer", "n": 1_082_802, "n_out": 3},
        # the learned cache's four training steps of a frame, 2^16 samples each
        {"name": "train_64k", "kind": "train", "n": 65_536, "n_out": 3, "steps": 4},
        # dJ/dE of 16 lights over the large room: 16 frozen rays per point, 64 sweeps of each solve
        {"name": "adjoint_1m", "kind": "adjoint", "points": 1_082_802, "lights": 16, "K": 16, "iterations": 64},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["frames"] * 4 + ["mesh"] * 2 + ["trace", "taa", "reference", "paths", "hashgrid", "infer", "train", "adjoint"])
    if kind == "frames":
        lights = rng.choice([1, 2, 3, 3, 3, 4, 8, 16])
        # states 1 and 2 have light 0 off: a room of one light would stay dark
        seq = rng.choice(["0x16", "0x8 1x4", "2x3 3x8", "0x3 4x5 0x4"] + (["1x4 2x6"] if lights > 1 else []))
        return {"kind": kind, "points": _log(rng, 5_000, 1_082_802 if lights <= 4 else 400_000), "lights": lights,
                "method": rng.choice([m for m in TIMING if lights <= 8 or "v4" not in m]), "seq": seq,
                "rays": rng.choice([1.0, 1.0, 1.0, 2.0, 4.0])}
    if kind == "mesh":
        lamps = rng.choice([3, 3, 8, 16])
        return {"kind": kind, "buildings": rng.choice([9, 16, 36, 64, 100, 144]), "points": _log(rng, 20_000, 500_000), "lamps": lamps,
                "method": rng.choice([m for m in TIMING if lamps <= 8 or "v4" not in m]), "seq": rng.choice(["0x10", "0x4 1x6", "1x3 2x5"])}
    if kind == "trace":
        return {"kind": kind, "buildings": rng.choice([9, 16, 36, 64, 100]), "points": 60_000, "rays": _log(rng, 100, 262_144)}
    if kind == "taa":
        return {"kind": kind, "points": _log(rng, 10_000, 1_082_802), "mask": rng.randrange(5), "seq": rng.choice(["0x12 1x12", "0x6 2x6", "0x16"])}
    if kind == "reference":
        return {"kind": kind, "points": _log(rng, 5_000, 43_000), "lights": rng.choice([1, 2, 3]), "K": rng.choice([8, 16, 31, 32]), "block": rng.choice([16, 64])}
    if kind == "paths":
        w = rng.choice([320, 641, 960, 1280, 1920])
        return {"kind": kind, "width": w, "height": w * 9 // 16 + rng.randrange(3), "points": _log(rng, 10_000, 170_185),
                "log2_capacity": rng.choice([20, 21, 22]), "bounces": rng.choice([1, 2])}
    if kind == "hashgrid":
        b = rng.randrange(18, 25)
        return {"kind": kind, "log2_capacity": b, "live": rng.choice([0.1, 0.3, 0.5, 0.7]), "samples": _log(rng, 1_000, min(1_000_003, 1 << b)),
                "event": rng.random() < 0.3}
    if kind == "infer":
        return {"kind": kind, "n": _log(rng, 100, 1_082_802), "n_out": rng.choice([1, 2, 3])}
    if kind == "train":
        return {"kind": kind, "n": 128 * _log(rng, 1, 512), "n_out": rng.choice([1, 3]), "steps": rng.choice([1, 2, 4])}
    return {"kind": kind, "points": _log(rng, 10_000, 1_082_802), "lights": rng.choice([1, 2, 3, 4, 8, 16]), "K": rng.choice([8, 13, 16]),
            "iterations": rng.choice([16, 64])}


# ------------------------------------------------------------------------------- inputs
_ST = None


def _stream() -> torch.cuda.Stream:
    """The renderer's one stream, which every context of the program issues on."""
    global _ST
    if _ST is None:
        _ST = torch.cuda.Stream()
    return _ST


class _Dev:
    """A device buffer of a context, which stays open as long as the buffer is looked at."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "strides": None, "version": 3}


def _view(owner, ptr: int, shape, typestr: str) -> torch.Tensor:
    """A device buffer of the library as a tensor (no copy)."""
    return torch.as_tensor(_Dev(owner, ptr, tuple(shape), typestr), device="cuda")


def _seq(text: str) -> list:
    return M.sequence([tuple(int(x) for x in part.split("x")) for part in text.split()])


def _room_scene(points: int, lights: int, seed: int) -> S.Scene:
    """The room of that size (its boxes and point count follow the size alone) with the seed's
    albedo per point and light emissions."""
    sc = S.box_room(points=points, seed=points % 1009, lights=lights)
    rng = np.random.default_rng(seed)
    sc.A = rng.uniform(0.5, 0.8, sc.Np).astype(np.float32)
    gain = rng.uniform(0.7, 1.4, lights).astype(np.float32)
    for s in sc.states:
        s.inten = s.inten * gain
    return sc


def _open_room(points: int, lights: int, seed: int):
    ctx = N.Context(stream=_stream().cuda_stream)
    info = ctx.load_bytes(S.write(_room_scene(points, lights, seed)))
    ctx.build_states()
    ctx.sync()
    return ctx, info


def _open_city(buildings: int, points: int, lamps: int, seed: int):
    """A city mesh prepared by the library (tree, cache points, lamps; no references), with the
    seed's albedo per triangle."""
    V, alb, ds = S.city_mesh(buildings, buildings)
    alb = np.random.default_rng(seed).uniform(0.2, 0.8, len(alb)).astype(np.float32)
    ctx = N.Context(stream=_stream().cuda_stream)
    with tempfile.TemporaryDirectory() as d:
        with open(os.path.join(d, "m.msh"), "wb") as f:
            f.write(S.write_msh1(V, alb, ds))
        ctx.prep_mesh(os.path.join(d, "m.msh"), os.path.join(d, "s.bin"), points=points, lamps=lamps, seed=1, ref_iterations=-1)
    ctx.build_states()
    ctx.sync()
    return ctx, ctx.info(), V


def _signed(x: int) -> int:
    return x - (1 << 64) if x >= 1 << 63 else x


def _mix64(x: torch.Tensor) -> torch.Tensor:
    """The cell key's hash (splitmix64's finaliser) on int64 bit patterns."""
    def shr(v, s):
        return (v >> s) & ((1 << (64 - s)) - 1)
    x = (x ^ shr(x, 30)) * _signed(0xBF58476D1CE4E5B9)
    x = (x ^ shr(x, 27)) * _signed(0x94D049BB133111EB)
    return x ^ shr(x, 31)


def _net_inputs(n: int, g: torch.Generator):
    pos = torch.zeros(n, 4, device="cuda")
    pos[:, :3] = torch.rand(n, 3, device="cuda", generator=g) * torch.tensor([8.0, 4.0, 3.0], device="cuda")
    axis = torch.randint(0, 6, (n,), device="cuda", generator=g)
    nrm = torch.zeros(n, 4, device="cuda")
    nrm.scatter_(1, (axis % 3)[:, None], torch.where(axis < 3, 1.0, -1.0)[:, None])
    aux = torch.empty(n, 4, device="cuda")
    aux[:, 0] = 0.5 + 0.3 * torch.rand(n, device="cuda", generator=g)
    aux[:, 1:] = torch.empty(n, 3, device="cuda").exponential_(generator=g)
    return pos, nrm, aux


def _net_weights(seed: int, n_out: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    w = []
    for l, (k, n) in enumerate(MLP.LAYERS):
        a = rng.uniform(-1.0, 1.0, (n, k)) * math.sqrt(6.0 / k)
        if l == len(MLP.LAYERS) - 1:
            a[n_out:] = 0.0
        w.append(a.reshape(-1))
    return np.concatenate(w).astype(np.float32)


def _net_target(aux: torch.Tensor, n_out: int) -> torch.Tensor:
    """Radiance-like targets: albedo times (direct light of the point + a share of the others')."""
    return (aux[:, :1] * (aux[:, 1:1 + n_out] + 0.3 * aux[:, 1:].mean(dim=1, keepdim=True))).contiguous()


def prepare(case: dict, seed: int) -> dict:
    k = case["kind"]
    st = {"case": case, "seed": seed}
    if k == "frames":
        st["ctx"], st["info"] = _open_room(case["points"], case["lights"], seed)
        st["method"] = TIMING[case["method"]].replace(rays=case["rays"])
        st["seq"] = _seq(case["seq"])
    elif k == "mesh":
        st["ctx"], st["info"], _ = _open_city(case["buildings"], case["points"], case["lamps"], seed)
        st["method"] = TIMING[case["method"]]
        st["seq"] = _seq(case["seq"])
    elif k == "trace":
        st["ctx"], st["info"], V = _open_city(case["buildings"], case["points"], 3, seed)
        rng = np.random.default_rng(seed)
        lo, hi = V.reshape(-1, 3).min(axis=0), V.reshape(-1, 3).max(axis=0)
        d = rng.normal(size=(case["rays"], 3))
        st["rays"] = np.concatenate([rng.uniform(lo, hi, (case["rays"], 3)), d / np.linalg.norm(d, axis=1, keepdims=True)], axis=1).astype(np.float32)
    elif k == "taa":
        sc = _room_scene(case["points"], 3, seed)
        rng = np.random.default_rng(seed)
        for i, s in enumerate(sc.states):   # stand-in references (smooth in space, dimmer with the lamp off)
            s.ref = ((1.0 if i in (0, 4) else 0.5) * (0.6 + 0.3 * np.sin(s.P @ rng.uniform(0.2, 1.0, 3)))).astype(np.float32)
            s.valid = np.ones(sc.Np, np.uint8)
            s.Pw = np.zeros((sc.Np, sc.NL), np.float32)
        st["ctx"] = N.Context(stream=_stream().cuda_stream)
        st["info"] = st["ctx"].load_bytes(S.write(sc))
        st["ctx"].build_states()
        st["ctx"].sync()
        st["seq"] = _seq(case["seq"])
    elif k == "reference":
        st["ctx"], st["info"] = _open_room(case["points"], case["lights"], seed)
    elif k == "paths":
        st["ctx"], st["info"] = _open_room(case["points"], 3, seed)
        st["hg"] = H.HashGrid(H.make_config(cell=0.05, capacity=1 << case["log2_capacity"], max_depth=4, tracing_distance=50.0, stream=_stream().cuda_stream))
        st["hg"].voxels_init(128)
        rng = np.random.default_rng(seed)
        st["cam"] = N.camera((0.5 + 0.3 * rng.random(), 0.5 + 0.3 * rng.random(), 1.6), (6.0, 3.0, 1.0), width=case["width"], height=case["height"], fov_y_deg=75.0)
        st["image"] = torch.zeros(case["height"], case["width"], 3, device="cuda")
        st["counts"] = torch.zeros(3, dtype=torch.int32, device="cuda")
        st["frame"] = 0
    elif k == "hashgrid":
        g = torch.Generator(device="cuda").manual_seed(seed)
        cap = 1 << case["log2_capacity"]
        hg = H.HashGrid(H.make_config(capacity=cap, cell=0.02, max_depth=4, acc_frames=64, stale_frames=60_000, tracing_distance=50.0, stream=_stream().cuda_stream))
        nx, ny, nz = 400, 200, 150
        want = int(cap * case["live"])
        # distinct random (cell, normal bucket) pairs: a random start and stride, coprime to their number
        total = nx * ny * nz * 6
        step = 1_000_003 + 2 * int(torch.randint(0, 100_000, (1,), generator=g, device="cuda"))
        while math.gcd(step, total) != 1:
            step += 2
        ids = (torch.arange(want, device="cuda", dtype=torch.int64) * step + int(torch.randint(0, total, (1,), generator=g, device="cuda"))) % total
        b, cx, cy, cz = ids % 6, ids // 6 % nx, ids // (6 * nx) % ny, ids // (6 * nx * ny)
        keys = ((((cx << 20 | cy) << 20 | cz) << 3) | b) + 1
        home = _mix64(keys) & (cap - 1)
        home, order = torch.sort(home)
        rank = torch.arange(want, device="cuda")
        slot = rank + torch.cummax(home - rank, 0).values   # linear probing, keys in order of their home slot
        ok = slot < cap
        slot, order = slot[ok], order[ok]
        table = _view(hg, hg.array_ptr(H.A_KEYS)[0], (cap,), "<i8")
        table[slot] = keys[order]
        for bank in (H.A_BANK0, H.A_BANK1):
            m = _view(hg, hg.array_ptr(bank)[0], (cap, 4), "<i4")
            m[slot] = 1 << torch.randint(0, 31, (len(slot), 4), generator=g, device="cuda", dtype=torch.int32)
        pick = order[torch.randint(0, len(order), (case["samples"],), generator=g, device="cuda")]
        cell = torch.stack([cx[pick], cy[pick], cz[pick]], 1).to(torch.float32)
        st["pos"] = ((cell + 0.25 + 0.5 * torch.rand(cell.shape, generator=g, device="cuda")) * 0.02).contiguous()
        nrm = torch.zeros(case["samples"], 3, device="cuda")
        nrm.scatter_(1, (b[pick] // 2)[:, None], torch.where(b[pick] % 2 == 0, 1.0, -1.0)[:, None])
        st["nrm"] = nrm
        st["rgb"] = torch.empty(case["samples"], 3, device="cuda").exponential_(generator=g)
        st["entry"] = torch.zeros(case["samples"], dtype=torch.int32, device="cuda")
        st["counts"] = torch.zeros(3, dtype=torch.int32, device="cuda")
        st["resolved"] = _view(hg, hg.array_ptr(H.A_RESOLVED)[0], (cap, 4), "<i4")
        st["inv"] = [1 << (seed % 32), 0, 0, 0] if case["event"] else [0, 0, 0, 0]
        st["hg"] = hg
    elif k in ("infer", "train"):
        g = torch.Generator(device="cuda").manual_seed(seed)
        st["net"] = MLP.Mlp(n_out=case["n_out"], lr=1e-2, seed=seed & 0xFFFF, max_batch=max(128, case["n"] if k == "train" else 128), stream=_stream().cuda_stream)
        st["net"].set_weights(_net_weights(seed, case["n_out"]))
        if k == "infer":
            st["pos"], st["nrm"], st["aux"] = _net_inputs(case["n"], g)
            st["out"] = torch.zeros(case["n"], 4, device="cuda")
        else:
            st["pos"], st["nrm"], st["aux"] = _net_inputs(4 * case["n"], g)
            st["target"] = _net_target(st["aux"], case["n_out"])
            st["idx"] = [torch.randint(0, 4 * case["n"], (case["n"],), generator=g, device="cuda", dtype=torch.int32) for _ in range(case["steps"])]
            st["loss"] = torch.zeros(1, device="cuda")
    elif k == "adjoint":
        st["ctx"], st["info"] = _open_room(case["points"], case["lights"], seed)
        rng = np.random.default_rng(seed)
        w = np.zeros(st["info"]["np"], np.float32)
        n = min(4096, len(w) // 2)
        w[rng.choice(len(w), n, replace=False)] = 1.0 / n
        st["weights"] = w
    else:
        raise ValueError("kind %r" % k)
    return st


# ------------------------------------------------------------------------------- one pass
AREA = ((3.5, 1.5, 2.95), (1.0, 0.0, 0.0), (0.0, -1.0, 0.0), (4.0, 3.5, 3.0))
SUN = ((0.3, 0.2, 1.0), (0.5, 0.5, 0.45))


def run(st: dict):
    case = st["case"]
    k = case["kind"]
    if k in ("frames", "mesh"):
        ctx, info = st["ctx"], st["info"]
        ctx.begin(st["method"], st["seq"][0], st["seed"])
        for s in st["seq"]:
            ctx.frame(s)
        n, lcs = info["np"], (info["nl"] + 3) // 4 * 4
        return {"cache": _view(ctx, ctx.device_ptr(N.A_LC), (n, lcs), "<f4"), "history": _view(ctx, ctx.device_ptr(N.A_N), (n,), "<f4"),
                "masks": _view(ctx, ctx.device_ptr(N.A_CUR), (info["nw"], n), "<i4")}
    if k == "trace":
        prim, t = st["ctx"].trace_rays(0, st["rays"])
        return {"prim": prim, "t": t}
    if k == "taa":
        ctx = st["ctx"]
        ctx.taa_begin(0.1, 1.0, case["mask"], st["seq"][0], 5000 + st["seed"] % 1000)
        errs = [ctx.taa_frame(s, want_err=True) for s in st["seq"]]
        return {"errors": np.array(errs, np.float32), "history": ctx.taa_array(N.T_H), "react": ctx.taa_array(N.T_REACT)}
    if k == "reference":
        ctx = st["ctx"]
        noise, iters = ctx.build_reference(K=case["K"], warmup=16, block=case["block"], max_iter=case["block"], noise_target=0.03)
        return {"noise": np.array(noise, np.float32), "iterations": np.array(iters, np.int32),
                "ref": [ctx.state_array(s, N.SA_REF) for s in range(st["info"]["ns"])], "valid": [ctx.state_array(s, N.SA_VALID) for s in range(st["info"]["ns"])]}
    if k == "paths":
        hg, f = st["hg"], st["frame"]
        st["frame"] += 1
        hg.begin_frame(f, 16)
        hg.camera_paths(st["ctx"], 0, H.path_params(st["cam"], bounces=case["bounces"], seed=1, frame=f, area=AREA, sun=SUN), st["image"])
        hg.resolve(None, st["counts"])
        cap = 1 << case["log2_capacity"]
        return {"image": st["image"], "counts": st["counts"], "resolved": _view(hg, hg.array_ptr(H.A_RESOLVED)[0], (cap, 4), "<i4"),
                "masks": _view(hg, hg.array_ptr(H.A_BANK0)[0], (cap, 4), "<i4")}
    if k == "hashgrid":
        hg = st["hg"]
        hg.insert(st["pos"], st["nrm"], st["entry"])
        hg.accumulate(st["entry"], st["rgb"])
        hg.resolve(st["inv"], st["counts"])
        return {"entry": st["entry"], "resolved": st["resolved"], "counts": st["counts"]}
    if k == "infer":
        st["net"].infer(st["pos"], st["nrm"], st["aux"], st["out"])
        return {"radiance": st["out"]}
    if k == "train":
        with torch.cuda.stream(_stream()):
            st["loss"].zero_()
        for idx in st["idx"]:
            st["net"].train(st["pos"], st["nrm"], st["aux"], st["target"], idx=idx, loss=st["loss"])
        return {"gradients": st["net"].gradients(), "loss": st["loss"]}
    g, res = st["ctx"].adjoint(0, st["weights"], K=case["K"], seed=st["seed"] & 0xFFFF, iterations=case["iterations"])
    return {"gradient": g, "J": res["J"], "back": res["back"], "max_incoming": res["max_incoming"]}


# ------------------------------------------------------------------------------- needed work
FLOP_PER_RAY = 400.0     # direction, a handful of plane or box tests, one exact triangle test, the walk


def work(case: dict) -> dict:
    """Bytes that a pass has to read and write once, and its arithmetic (a ray at FLOP_PER_RAY)."""
    k = case["kind"]
    if k in ("frames", "mesh"):
        m = TIMING[case["method"]]
        n, nl = case["points"], case.get("lights", case.get("lamps"))
        lcs, frames = (nl + 3) // 4 * 4, len(_seq(case["seq"]))
        rays = m.budget * case.get("rays", 1.0)
        # position, normal, own cache in and out, history in and out; per ray the hit's albedo and
        # direct light and its cache; tracked frames the mask in and out and the hit's voxels
        per = 32 + 8 * lcs + 8 + rays * (4 * ((nl + 4) // 4 * 4) + 4 * lcs)
        tracked = (32 + 16 * rays) / m.track_every if m.deps else 0.0
        return {"bytes": n * frames * (per + tracked), "flops": n * frames * rays * FLOP_PER_RAY}
    if k == "trace":
        return {"bytes": 32.0 * case["rays"], "flops": case["rays"] * 4 * FLOP_PER_RAY}
    if k == "taa":
        n, f = case["points"], len(_seq(case["seq"]))
        # position, normal, the hit's record and reference, history in and out, statistics, the masks
        return {"bytes": n * f * (32.0 + 20 + 8 + 8 + 8 + 5 + (48 if case["mask"] in (2, 3) else 0)), "flops": n * f * FLOP_PER_RAY}
    if k == "reference":
        its = 2 * (16 + case["block"]) * 5
        lcs = (case["lights"] + 3) // 4 * 4
        return {"bytes": case["points"] * its * (32.0 + 8 * lcs + case["K"] * (16 + 4 * lcs)), "flops": case["points"] * its * case["K"] * FLOP_PER_RAY}
    if k == "paths":
        v = case["width"] * case["height"] * (case["bounces"] + 1)
        # a vertex record and its sample written, then read for the marks; the table once
        return {"bytes": v * (64.0 + 36 + 64 + 40) + 72.0 * (1 << case["log2_capacity"]), "flops": v * 2 * FLOP_PER_RAY}
    if k == "hashgrid":
        cap = 1 << case["log2_capacity"]
        return {"bytes": 8.0 * cap + case["live"] * cap * 96 + case["samples"] * (24 + 8 + 4 + 4 + 12 + 32), "flops": 20.0 * case["live"] * cap}
    if k == "infer":
        return {"bytes": case["n"] * (48.0 + 4 * case["n_out"]), "flops": 2.0 * case["n"] * (168 * 64 + 3 * 64 * 64 + 64 * case["n_out"])}
    if k == "train":
        return {"bytes": case["steps"] * (case["n"] * (52.0 + 4 * case["n_out"]) + 24_576 * 24.0),
                "flops": case["steps"] * 6.0 * case["n"] * (168 * 64 + 3 * 64 * 64 + 64 * case["n_out"])}
    rays = float(case["points"] * case["K"])
    return {"bytes": case["iterations"] * (8.0 * rays + 40.0 * case["points"]), "flops": rays * (FLOP_PER_RAY + 4.0 * case["iterations"])}


# ------------------------------------------------------------------------------- in 64 bits
def _features(pos, nrm, aux):
    p = (pos[:, :3].double() / torch.tensor([8.0, 4.0, 3.0], device="cuda", dtype=torch.float64)).clamp(0, 1)
    n, x = nrm[:, :3].double(), aux.double()
    f = []
    for a in range(3):
        for o in range(12):
            f += [torch.sin(2.0 ** o * math.pi * p[:, a]), torch.cos(2.0 ** o * math.pi * p[:, a])]
    for a in range(3):
        for o in range(4):
            f += [torch.sin(2.0 ** o * math.pi * n[:, a]), torch.cos(2.0 ** o * math.pi * n[:, a])]
    for a in range(3):
        f += [(1 - (p[:, a] * 16 - (j + 0.5)).abs()).clamp(min=0) for j in range(16)]
    for a in range(3):
        f += [(1 - ((n[:, a] * 0.5 + 0.5) * 4 - (j + 0.5)).abs()).clamp(min=0) for j in range(4)]
    f += [p[:, 0], p[:, 1], p[:, 2], n[:, 0], n[:, 1], n[:, 2], x[:, 1], x[:, 2], x[:, 3], x[:, 0]]
    f.append(torch.ones_like(f[0]))
    f += [torch.zeros_like(f[0])] * (176 - len(f))
    return torch.stack(f, 1)


def _layers(w: torch.Tensor) -> list:
    out, o = [], 0
    for a, b in ((176, 64), (64, 64), (64, 64), (64, 64), (64, 16)):
        out.append(w[o:o + a * b].reshape(b, a))
        o += a * b
    return out


def _net(w: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    ws = _layers(w)
    for a in ws[:-1]:
        x = torch.relu(x @ a.T)
    return x @ ws[-1].T


def exact(case: dict, seed: int):
    """The network's outputs and its training gradients in 64 bits.  The other kinds return integers,
    or values that follow random walks whose every step is an integer decision (which point a ray
    reaches), so they have no value in 64 bits apart from their own arithmetic."""
    k = case["kind"]
    if k not in ("infer", "train"):
        return None
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.from_numpy(_net_weights(seed, case["n_out"])).to("cuda").double()
    if k == "infer":
        pos, nrm, aux = _net_inputs(case["n"], g)
        out = torch.zeros(case["n"], 4, device="cuda", dtype=torch.float64)
        for i in range(0, case["n"], 1 << 17):
            s = slice(i, i + (1 << 17))
            out[s, :case["n_out"]] = _net(w, _features(pos[s], nrm[s], aux[s]))[:, :case["n_out"]]
        return {"radiance": out}
    pos, nrm, aux = _net_inputs(4 * case["n"], g)
    target = _net_target(aux, case["n_out"]).double()
    idx = [torch.randint(0, 4 * case["n"], (case["n"],), generator=g, device="cuda", dtype=torch.int32) for _ in range(case["steps"])]
    m1, m2, loss = torch.zeros_like(w), torch.zeros_like(w), torch.zeros(1, device="cuda", dtype=torch.float64)
    for t, i in enumerate(idx, 1):
        i = i.long()
        wi = w.clone().requires_grad_(True)
        y = _net(wi, _features(pos[i], nrm[i], aux[i]))[:, :case["n_out"]]
        e = (y - target[i]) ** 2 / (y.detach() ** 2 + 0.01)
        (e.sum() / e.numel()).backward()
        grad = wi.grad
        loss += e.detach().sum()
        m1 = 0.9 * m1 + 0.1 * grad
        m2 = 0.99 * m2 + 0.01 * grad * grad
        w = w - 1e-2 * (m1 / (1 - 0.9 ** t)) / ((m2 / (1 - 0.99 ** t)).sqrt() + 1e-8)
    return {"gradients": grad.cpu().numpy(), "loss": loss}
