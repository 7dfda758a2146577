"""The work that a user of this framework has it do, as cases to measure.

Every case goes through the public entry points (photonmap.Context, .Batch) with
the settings that the repository's workloads, tests and benchmark use: the room,
the heightfield room and the stress room of photonmap.scenes.WORKLOADS, the
instance ranges of scenes.batch_instances, the learned frame's settings of
photonmap.learned.  A case's `kind` says which call it is:

  frame     Context.frame: photon pass + grid + eye pass + gather + resolve
  dynamic   set_scene with the device BVH builder, then a frame: geometry that
            changes every frame
  render    Context.render on a resident photon map: a camera that moves
  map       a photon list that the caller has (set_photons), grid, kNN queries
  knn       kNN queries on a resident map
  split     one rank's share of a frame split over ranks: trace_paths of its
            path range, set_photons, build_grid, render_rows of its band
  batch     Batch.frame: many scene instances per frame
  gradient  cache_gradient: forward and backward of the radiance cache
  infer     cache_infer: its forward
  learned   render_learned: the frame answered by a trained cache

prepare() makes what such a program holds before the call (scene on the device,
resident map, trained cache, sample arrays) from the seed; run() is the call.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-photon-mapping_b200"))

import photonmap  # noqa: E402
from photonmap import learned, scenes  # noqa: E402

BOX = [-1.0, -1.0, -1.0, 1.0, 1.0, 1.0]
OUT_SCALE = 0.5          # the cache's output unit in the gradient and infer cases
LAYERS, DIM = 5, 64


def listed():
    return [
        # the smallest frame (workload cornell_small): a preview, where launches and host waits count
        dict(name="frame_room_100k", kind="frame", scene="room", photons=100_000, caustic=0, bounces=8, width=320,
             height=240, k=100, radius=0.1, k_caustic=0),
        # an ordinary frame with both photon maps, at an odd image size
        dict(name="frame_caustics_1m", kind="frame", scene="room", photons=1_000_003, caustic=120_011, bounces=8,
             width=641, height=361, k=64, radius=0.1, k_caustic=50),
        # the headline workload cornell_hf_1080p
        dict(name="frame_hf_10m_1080p", kind="frame", scene="hf", photons=10_000_000, caustic=0, bounces=10,
             width=1920, height=1080, k=64, radius=0.05, k_caustic=0),
        # the largest workload, cornell_stress_4k
        dict(name="frame_stress_100m_4k", kind="frame", scene="stress", photons=100_000_000, caustic=0, bounces=16,
             width=3840, height=2160, k=200, radius=0.02, k_caustic=0),
        # geometry that changes every frame: device BVH build, photons, grid and image
        dict(name="dynamic_hf_250k", kind="dynamic", scene="hf", photons=250_000, caustic=0, bounces=8, width=640,
             height=360, k=64, radius=0.1, k_caustic=0),
        # a camera that moves through a resident map
        dict(name="render_resident_2m", kind="render", scene="hf", photons=2_000_000, caustic=0, bounces=10,
             width=1280, height=720, k=128, radius=0.05, k_caustic=0),
        # a photon file's list brought in, its grid and a ragged number of queries with their ids
        dict(name="map_3m_k200", kind="map", photons=3_000_017, queries=100_003, k=200, radius=0.05),
        # a few queries on a small resident map: latency
        dict(name="knn_1k", kind="knn", photons=100_000, queries=1_021, k=16, radius=0.1),
        # one of four ranks of a split 1080p frame
        dict(name="split_rank_of_4", kind="split", scene="hf", paths=600_001, bounces=10, width=1920, height=1080,
             rank=1, ranks=4, k=64, radius=0.05),
        # sixteen instances of the batched workload
        dict(name="batch_16", kind="batch", instances=16, layout=0),
        # one training batch of the learned frame, forward and backward
        dict(name="gradient_262k", kind="gradient", samples=262_144),
        # the learned frame: cache inference, exact probes and per-tile fallback
        dict(name="learned_1080p", kind="learned", scene="hf", photons=4_000_000, bounces=10, width=1920, height=1080,
             k=64, radius=0.05),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "dynamic", "render", "map", "knn", "split", "batch", "gradient",
                       "infer", "learned"])
    if kind == "batch":
        return dict(kind=kind, instances=rng.randint(2, 16), layout=rng.randint(1, 1000))
    if kind in ("gradient", "infer"):
        return dict(kind=kind, samples=_log(rng, 500, 1_100_000))
    if kind in ("map", "knn"):
        photons = _log(rng, 20_000, 4_000_000 if kind == "map" else 1_000_000)
        return dict(kind=kind, photons=photons, queries=_log(rng, 300, 200_000), k=rng.randint(1, 256),
                    radius=rng.choice([0.03, 0.05, 0.1]))
    scene = rng.choice(["room", "hf"])
    width = _log(rng, 128, 1920)
    c = dict(kind=kind, scene=scene, bounces=rng.choice([8, 10, 16]), width=width,
             height=max(96, int(width * rng.uniform(0.5, 1.0))), k=rng.choice([32, 50, 64, 100, 128, 200]),
             radius=rng.choice([0.05, 0.1]))
    if kind == "split":
        ranks = rng.choice([2, 4, 8])
        c.update(paths=_log(rng, 20_000, 1_500_000), ranks=ranks, rank=rng.randrange(ranks))
        return c
    if kind == "learned":
        c.update(photons=_log(rng, 300_000, 6_000_000), k=64)
        return c
    c.update(photons=_log(rng, 50_000, 20_000_000 if kind == "frame" else 4_000_000), caustic=0, k_caustic=0)
    if kind != "render" and rng.random() < 0.4:
        c.update(caustic=max(1_000, c["photons"] // rng.randint(8, 40)), k_caustic=rng.choice([20, 50, 100]))
    return c


# ------------------------------------------------------------------ scenes --
@functools.lru_cache(maxsize=8)
def _scene(name, terrain=0):
    return {"room": lambda: scenes.cornell(sphere_level=3, seed=terrain),
            "hf": lambda: scenes.cornell(sphere_level=3, heightfield_n=256, seed=terrain),
            "stress": lambda: scenes.cornell(sphere_level=3, stress=True, seed=terrain)}[name]()


@functools.lru_cache(maxsize=4)
def _instances(n, layout):
    return scenes.batch_instances(n, seed=layout)


def _camera(case, rng):
    """The workloads' camera, moved a little as the seed says."""
    cs = scenes.default_camera(case["width"], case["height"])
    dx, dy = rng.uniform(-0.1, 0.1, 2)
    return photonmap.camera_setup((float(dx), float(dy), 3.5), cs.direction, cs.up, cs.fov_deg, cs.width, cs.height)


def _rays(case):
    """Eye-path hits of a frame: about 0.6 per pixel with this camera."""
    return 0.6 * case["width"] * case["height"]


# ------------------------------------------------------- photons of a list --
def _cloud(n, gen):
    """A photon map as a caller may have it: photons on the walls of the room
    and on two spheres, arriving from above, equal power."""
    dev = "cuda"
    p = torch.rand((n, 3), generator=gen, device=dev) * 2 - 1
    which = torch.randint(0, 14, (n,), generator=gen, device=dev)
    d = torch.randn((n, 3), generator=gen, device=dev)
    d = d / d.norm(dim=1, keepdim=True).clamp_min(1e-6)
    nrm = torch.zeros((n, 3), device=dev)
    for side, (axis, val) in enumerate(((1, -1.0), (1, 1.0), (2, -1.0), (0, -1.0), (0, 1.0))):
        on = (which >= 2 * side) & (which < 2 * side + 2)
        p[:, axis] = torch.where(on, torch.full_like(p[:, axis], val), p[:, axis])
        nrm[:, axis] = torch.where(on, torch.full_like(nrm[:, axis], -val), nrm[:, axis])
    for c, pick in (((-0.4, -0.7, 0.2), 10), ((0.45, -0.7, -0.3), 12)):
        on = ((which == pick) | (which == pick + 1))[:, None]
        p = torch.where(on, torch.tensor(c, device=dev) + 0.3 * d, p)
        nrm = torch.where(on, d, nrm)
    inc = torch.randn((n, 3), generator=gen, device=dev)
    inc = inc / inc.norm(dim=1, keepdim=True).clamp_min(1e-6)
    facing = (inc * nrm).sum(1, keepdim=True)
    inc = torch.where(facing > 0, -inc, inc)               # photons arrive against the normal
    power = torch.full((n, 3), 1.0 / n, device=dev) * torch.tensor([1.0, 0.8, 0.6], device=dev)
    return p.contiguous(), power.contiguous(), inc.contiguous(), nrm.contiguous()


def _map_inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    pos, power, inc, _ = _cloud(case["photons"], gen)
    qpos, _, _, qnrm = _cloud(case["queries"], gen)
    return pos, power, inc, qpos, qnrm


def _samples(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    n = case["samples"]
    pos, _, _, nrm = _cloud(n, gen)
    lit = 0.5 + 0.4 * torch.sin(3 * pos) * torch.cos(2 * pos.roll(1, 1)) + 0.1 * nrm
    return pos, nrm, (lit * torch.rand((n, 3), generator=gen, device="cuda") * 0.4).contiguous()


# ------------------------------------------------------- the cache's network --
def _encode(pos, nrm, dtype):
    lo = torch.tensor(BOX[:3], dtype=dtype, device=pos.device)
    u = (pos.to(dtype) - lo) * 0.5
    n = nrm.to(dtype)
    a = n.abs().sum(1)
    a = torch.where(a > 0, a, torch.ones_like(a))
    o = n[:, :2] / a[:, None]
    s = torch.where(o >= 0, torch.ones_like(o), -torch.ones_like(o))
    o = torch.where((n[:, 2] < 0)[:, None], (1 - o.flip(1).abs()) * s, o) * 0.5 + 0.5
    x = torch.cat([u, o], 1)
    ang = math.pi * x[:, :, None] * (2.0 ** torch.arange(6, dtype=dtype, device=pos.device))
    f = torch.stack([ang.sin(), ang.cos()], -1).reshape(pos.shape[0], 60)
    return torch.nn.functional.pad(f, (0, 4))


def _weights(seed):
    """Parameters in the library's layout (He-uniform, padding zero)."""
    rng = np.random.default_rng(seed)
    w = np.zeros((LAYERS, DIM, DIM), np.float32)
    for l in range(LAYERS):
        fan = 60 if l == 0 else DIM
        outs = 3 if l == LAYERS - 1 else DIM
        b = (0.5 if l == LAYERS - 1 else 1.0) * math.sqrt(6.0 / fan)
        w[l, :outs, :fan] = rng.uniform(-b, b, (outs, fan))
    return w


def _forward(w, feats):
    x = feats
    for l in range(LAYERS - 1):
        x = torch.relu(x @ w[l].T)
    return (x @ w[LAYERS - 1][:3].T)


def _fit(pool, seed, steps=250, batch=16384, lr=3e-3):
    """Weights fitted to a training pool in plain torch, so that the same seed
    gives the same weights whoever renders with them."""
    w = torch.tensor(_weights(seed), device="cuda").requires_grad_(True)
    live = (w.detach() != 0).float()
    feats, target = _encode(pool.pos, pool.nrm, torch.float32), pool.target / pool.scale
    m, v = torch.zeros_like(live), torch.zeros_like(live)
    at = 0
    for step in range(1, steps + 1):
        if at + batch > feats.shape[0]:
            at = 0
        loss = (_forward(w, feats[at:at + batch]) - target[at:at + batch]).square().mean()
        (g,) = torch.autograd.grad(loss, w)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.99 * v + 0.01 * g * g
            w -= lr * live * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.99 ** step)).sqrt() + 1e-8)
        at += batch
    return w.detach().cpu().numpy().reshape(-1)


# ---------------------------------------------------------------- interface --
def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    st = dict(case=case, seed=int(seed))
    if kind == "batch":
        inst = []
        for i, p in enumerate(_instances(case["instances"], case["layout"])):
            cs = p["camera_spec"]
            cam = photonmap.camera_setup(cs.position, cs.direction, cs.up, cs.fov_deg, cs.width, cs.height)
            inst.append(dict(scene=p["scene"], camera=cam, seed=int(seed) * 1000 + i, photons=p["photons"],
                             max_bounces=p["max_bounces"], k=p["k"], radius=p["radius"], max_depth=p["max_depth"]))
        st["batch"] = photonmap.Batch(inst)
        return st
    ctx = st["ctx"] = photonmap.Context(0)
    if kind in ("map", "knn"):
        st["in"] = _map_inputs(case, seed)
        if kind == "knn":
            ctx.set_photons(photonmap.PM_MAP_GLOBAL, *st["in"][:3])
            ctx.build_grid(aabb=BOX)
        return st
    if kind in ("gradient", "infer"):
        st["in"] = _samples(case, seed)
        ctx.cache_init(seed=1, out_scale=OUT_SCALE, aabb=BOX)
        ctx.cache_set_params(_weights(seed))
        return st
    if kind == "dynamic":
        st["scene"] = _scene(case["scene"], int(seed) % 1000)
        ctx.set_bvh_builder("device_lbvh")
    else:
        ctx.set_scene(_scene(case["scene"]))
    st["cam"] = _camera(case, rng)
    if kind in ("render", "learned"):
        ctx.trace_photons(int(seed), case["bounces"], case["photons"])
        ctx.build_grid()
    if kind == "learned":
        pool = learned.training_pool(ctx, st["cam"], case["k"], case["radius"], n=1 << 17, seed=1)
        ctx.cache_init(seed=0, out_scale=pool.scale, aabb=BOX)
        ctx.cache_set_params(_fit(pool, seed))
    return st


def _padded(x, rows):
    out = torch.zeros((rows,) + tuple(x.shape[1:]), dtype=x.dtype, device=x.device)
    out[:x.shape[0]] = x
    return out


def run(state):
    c, seed = state["case"], state["seed"]
    kind = c["kind"]
    if kind == "batch":
        b = state["batch"]
        b.frame(1)
        return [b.image(i) for i in range(b.n)]
    ctx = state["ctx"]
    if kind in ("frame", "dynamic"):
        if kind == "dynamic":
            ctx.set_scene(state["scene"])
        return ctx.frame(seed, c["bounces"], c["photons"], state["cam"], c["k"], c["radius"],
                         caustic_capacity=c["caustic"], k_caustic=c["k_caustic"])[:2]
    if kind == "render":
        return ctx.render(state["cam"], c["k"], c["radius"])
    if kind in ("map", "knn"):
        pos, power, inc, qpos, qnrm = state["in"]
        if kind == "map":
            ctx.set_photons(photonmap.PM_MAP_GLOBAL, pos, power, inc)
            ctx.build_grid(aabb=BOX, k_hint=c["k"])
        rad, ids, cnt = ctx.gather(qpos, qnrm, c["k"], c["radius"], want_ids=True)
        return dict(rad=rad, ids=ids, cnt=cnt)
    if kind == "split":
        first = c["rank"] * c["paths"]
        t = ctx.trace_paths(seed, c["bounces"], c["paths"], first, first + c["paths"])
        power = torch.from_numpy(ctx.light_intensity / np.float32(c["paths"])).cuda().expand_as(t["g_pos"])
        ctx.set_photons(photonmap.PM_MAP_GLOBAL, t["g_pos"], power, t["g_dir"])
        ctx.build_grid()
        h = c["height"]
        y0, y1 = h * c["rank"] // c["ranks"], h * (c["rank"] + 1) // c["ranks"]
        rgb, rad = ctx.render_rows(state["cam"], c["k"], c["radius"], 4, y0, y1)
        w = c["width"]
        # the records leave for the other ranks padded to one size, as the exchange sends them
        out = {key: _padded(t[key], 3 * c["paths"] // (2 if key[0] == "g" else 4))
               for key in ("g_pos", "g_dir", "c_pos", "c_dir")}
        return dict(out, counts=t["counts"], rgb=rgb[3 * w * y0:3 * w * y1], rad=rad[w * y0:w * y1])
    if kind == "gradient":
        g, loss = ctx.cache_gradient(*state["in"])
        return dict(grad=g, loss=loss)
    if kind == "infer":
        return ctx.cache_infer(*state["in"][:2])
    rgb, rad, stats = ctx.render_learned(state["cam"], c["k"], c["radius"], **learned.FRAME_SETTINGS)
    return dict(rgb=rgb, rad=rad, fallback_tiles=stats["fallback_tiles"],
                fallback_requests=stats["fallback_requests"])


# per ray of the photon pass and the eye pass: about 11 BVH nodes of two boxes
# (2 x 20 flops) and 4 triangle tests (86 flops); 1.4 rays per stored photon.
# Per kNN query: a distance and a filter term (30 flops) for each of its k.
RAY_FLOPS = 11 * 40 + 4 * 86
TRIANGLES = {"room": 2_572, "hf": 132_620, "stress": 89_612}


def work(case):
    """Bytes: each input read once and each output written once (scene: 116
    bytes per triangle; photon of a resident or given map: position, power,
    direction; image: 3 bytes and 12 of radiance per pixel)."""
    kind = case["kind"]
    if kind == "batch":
        inst = _instances(case["instances"], case["layout"])
        px = sum(p["camera_spec"].width ** 2 for p in inst)
        photons = sum(p["photons"] for p in inst)
        flops = 1.4 * photons * RAY_FLOPS
        flops += sum(p["camera_spec"].width ** 2 * (RAY_FLOPS + p["k"] * 30.0) for p in inst)
        return dict(bytes=3.0 * px + 116.0 * TRIANGLES["room"] * len(inst), flops=flops)
    if kind in ("gradient", "infer"):
        n = case["samples"]
        per = 2.0 * (60 * DIM + 3 * DIM * DIM + DIM * 3)
        return dict(bytes=36.0 * n, flops=per * n * (3 if kind == "gradient" else 1))
    if kind in ("map", "knn"):
        q, k = case["queries"], case["k"]
        return dict(bytes=(36.0 * case["photons"] if kind == "map" else 36.0 * min(case["photons"], q * k)) +
                    q * (24.0 + 12 + 4 + 4 * k), flops=30.0 * q * k)
    px = case["width"] * case["height"]
    scene = 116.0 * TRIANGLES[case["scene"]]
    hits = _rays(case)
    if kind == "split":
        photons = 1.1 * case["paths"]
        return dict(bytes=scene + photons * 24 + case["paths"] * 8 + 15.0 * px / case["ranks"],
                    flops=1.4 * photons * RAY_FLOPS + hits / case["ranks"] * (RAY_FLOPS + 30.0 * case["k"]))
    image = scene + 15.0 * px
    if kind == "learned":
        per = 2.0 * (60 * DIM + 3 * DIM * DIM + DIM * 3)
        return dict(bytes=image + 28.0 * case["k"] * px / 32, flops=px * RAY_FLOPS + hits * per)
    gather = hits * 30.0 * (case["k"] + case["k_caustic"])
    if kind == "render":
        return dict(bytes=image + 28.0 * min(case["photons"], hits * case["k"]), flops=px * RAY_FLOPS + gather)
    return dict(bytes=image, flops=(1.4 * (case["photons"] + case["caustic"]) + px) * RAY_FLOPS + gather)


# -------------------------------------------------------------------- exact --
def _knn64(pos, power, inc, qpos, qnrm, k, radius):
    """The k nearest within radius and the filtered density estimate, in 64 bits."""
    dev = pos.device
    P, Q = pos.double(), qpos.double()
    n = int(math.ceil(2.0 / radius)) + 4
    cell_of = lambda x: ((x + 1.0) / radius + 2).long().clamp(1, n - 2)  # noqa: E731
    pc, qc = cell_of(P), cell_of(Q)
    pid = pc[:, 0] + n * (pc[:, 1] + n * pc[:, 2])
    order = torch.argsort(pid, stable=True)
    starts = torch.searchsorted(pid[order], torch.arange(n ** 3 + 1, device=dev))
    runs = torch.tensor([n * (dy + n * dz) for dy in (-1, 0, 1) for dz in (-1, 0, 1)], device=dev)
    qid = (qc[:, 0] + n * (qc[:, 1] + n * qc[:, 2]))[:, None] + runs
    a, b = starts[qid - 1], starts[qid + 2]                 # three cells along x are one run
    total = (b - a).sum(1)
    if float(total.sum()) > 2e9:
        return None
    out = torch.zeros((Q.shape[0], 3), dtype=torch.float64, device=dev)
    by_size = torch.argsort(total)
    at = 0
    while at < Q.shape[0]:
        take = by_size[at:at + 65536]
        most = int(total[take].max())
        take = take[:max(1, 20_000_000 // max(most, 1))]
        most = int(total[take].max())
        at += take.numel()
        if most == 0:
            continue
        length = (b - a)[take]
        ends = length.cumsum(1)
        col = torch.arange(most, device=dev).expand(take.numel(), most).contiguous()
        run = torch.searchsorted(ends, col, right=True).clamp_max(8)
        slot = a[take].gather(1, run) + col - (ends - length).gather(1, run)
        ok = col < ends[:, -1:]
        ph = order[slot.clamp(0, P.shape[0] - 1)]
        d = (P[ph] - Q[take][:, None, :]).square().sum(-1).sqrt()
        d = torch.where(ok & (d <= radius), d, torch.full_like(d, math.inf))
        kk = min(k, most)
        dk, at_k = torch.topk(d, kk, dim=1, largest=False)
        found = torch.isfinite(dk)
        rk = torch.where(found, dk, torch.zeros_like(dk)).amax(1, keepdim=True)
        ph = ph.gather(1, at_k)
        facing = (inc.double()[ph] * qnrm.double()[take][:, None, :]).sum(-1) < 0
        f = 1.818 * (1 - (1 - torch.exp(-1.953 * dk ** 2 / (2 * rk ** 2))) / (1 - math.exp(-1.953)))
        f = torch.where(found & facing, f, torch.zeros_like(f))
        est = (power.double()[ph] * f[..., None]).sum(1) / (math.pi * rk ** 2)
        out[take] = torch.where(rk > 0, est, torch.zeros_like(est))
    return out


def exact(case, seed):
    """64-bit answers where plain torch has them: estimates of the kNN queries,
    the network's outputs and gradients.  Frames have none: their paths take
    decisions on 32-bit draws and distances that 64 bits would take otherwise."""
    kind = case["kind"]
    if kind in ("map", "knn"):
        rad = _knn64(*_map_inputs(case, seed), case["k"], case["radius"])
        return None if rad is None else dict(rad=rad, ids=None, cnt=None)
    if kind in ("gradient", "infer"):
        pos, nrm, target = _samples(case, seed)
        w = torch.tensor(_weights(seed), dtype=torch.float64, device="cuda")
        if kind == "infer":
            return _forward(w, _encode(pos, nrm, torch.float64)) * OUT_SCALE
        w.requires_grad_(True)
        y = _forward(w, _encode(pos, nrm, torch.float64))
        loss = (y - target.double() / OUT_SCALE).square().mean()
        (g,) = torch.autograd.grad(loss, w)
        return dict(grad=g.reshape(-1).cpu().numpy(), loss=float(loss))
    return None
