"""Performance cases: the work that programs have this library do, through its public entry points.

A case is a dict of plain values; `prepare` makes what a program has in hand before the call (a
resident model, the rays or rows on the device or in page-locked host memory), `run` is one pass.

Models. `sphere`: the 65,536-triangle displaced sphere with its 1,024-leaf cut and the committed
trained weights (16 levels x 2 features x 2^19 entries, 4 points, 64 x 4 MLP). `refdef`: the same
mesh and cut with the reference renderer's default encoding (8 levels x 4 features x 2^18, 3
points); no trained weights of it are committed, so its table holds seeded values whose outputs lie
on both sides of the visibility threshold. A program keeps its models between calls, so a model
that a pass only reads is built once per process.
"""

import math
import os

import numpy as np
import torch

import nbvh_gb300 as nb
from nbvh_gb300 import abi, scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TRAINED = os.path.join(ROOT, "bench_data", "sphere65k_cut1024_trained.npz")
FLT_MAX = 3.4028234663852886e38
PRECISIONS = {"fp16": 0, "bf16": 1, "fp8": 2}

# leaf segments the network answers per ray (nbvh_last_query_stats on these models)
SEGMENTS_PER_RAY = {"uniform": 0.57, "camera": 1.08, "surface": 1.4}


def listed():
    return [
        # a cursor pick or a handful of probe rays per frame: latency alone
        {"name": "pick_17", "kind": "closest", "model": "sphere", "n": 17, "depth": 1},
        # one interactive frame of primary rays (run-inference at 512 x 512)
        {"name": "frame_512", "kind": "frame", "model": "sphere", "width": 512, "height": 512},
        # the benchmark's batch: 2^22 rays from the 1.5x scene box, closest hit
        {"name": "closest_4m", "kind": "closest", "model": "sphere", "n": 1 << 22, "depth": 1},
        # secondary visibility (shadow) rays of an odd-sized batch with the reference's default encoding
        {"name": "visibility_refdef_1m", "kind": "visibility", "model": "refdef", "n": 1000003, "depth": 2},
        # a host renderer's batch: rays in and records out in page-locked host memory
        {"name": "host_1m", "kind": "host", "model": "sphere", "n": 1 << 20, "depth": 1},
        # a path-traced preview frame: 4 bounces, ground plane, sky
        {"name": "path_960x540", "kind": "path", "model": "sphere", "width": 960, "height": 540, "spp": 1, "bounces": 4},
        # the non-neural BLAS on the benchmark's batch, and on a small odd batch
        {"name": "classic_4m", "kind": "classic", "n": 1 << 22, "any": False},
        {"name": "classic_20k", "kind": "classic", "n": 20011, "any": False},
        # the network alone on encoded rows (a program with its own encoder)
        {"name": "mlp_1m", "kind": "mlp", "n": 1 << 20, "precision": "fp16"},
        # encoding + network on explicit points: a few thousand samples per call
        {"name": "network_3k", "kind": "network", "n": 3001, "precision": "fp16"},
        # forward + loss + backward of the default training batch, gradients out
        {"name": "gradients_262k", "kind": "gradients", "n": 1 << 18, "precision": "fp16"},
        # run-optimisation's step in a program's own loop: sampled batch, gradients, Adam
        {"name": "train_step_262k", "kind": "train", "n": 1 << 18, "precision": "fp16"},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["closest", "closest", "visibility", "frame", "host", "path", "classic", "mlp", "network",
                       "gradients", "train"])
    c = {"kind": kind}
    if kind in ("closest", "visibility"):
        c.update(model=rng.choice(["sphere", "sphere", "refdef"]), n=_log_uniform(rng, 1, 1 << 22),
                 depth=rng.choice([1, 2]))
    elif kind == "host":
        c.update(model="sphere", n=_log_uniform(rng, 100, 1 << 20), depth=rng.choice([1, 2]))
    elif kind == "frame":
        c.update(model=rng.choice(["sphere", "refdef"]), width=_log_uniform(rng, 16, 1920),
                 height=_log_uniform(rng, 16, 1080))
    elif kind == "path":
        c.update(model="sphere", width=_log_uniform(rng, 64, 960), height=_log_uniform(rng, 64, 540),
                 spp=rng.choice([1, 1, 2]), bounces=rng.randint(0, 4))
    elif kind == "classic":
        c.update(n=_log_uniform(rng, 1, 1 << 22), any=rng.random() < 0.3)
    elif kind in ("mlp", "network"):
        c.update(n=_log_uniform(rng, 1, 1 << 20), precision=rng.choice(["fp16", "fp16", "bf16", "fp8"]))
    elif kind == "gradients":
        c.update(n=_log_uniform(rng, 64, 1 << 18), precision=rng.choice(["fp16", "fp16", "bf16", "fp8"]))
    else:
        c.update(n=1 << rng.randint(10, 18), precision=rng.choice(["fp16", "fp16", "bf16"]))
    return c


# ------------------------------------------------------------------------------------------------
# Models
# ------------------------------------------------------------------------------------------------

_cache = {}


def _once(key, make):
    if key not in _cache:
        _cache[key] = make()
    return _cache[key]


def _mesh():
    v, f = scenes.fbm_sphere(7, seed=1)
    return v, f, scenes.palette_albedo(len(f), 1)


def _trained_params():
    return np.load(TRAINED)["params_f16"].view(np.float16).astype(np.float32)


def _refdef_params(layout):
    # Xavier-uniform matrices and a table of uniform values: outputs on both sides of the threshold
    rng = np.random.default_rng(7)
    p = rng.uniform(-0.6, 0.6, layout.n_params).astype(np.float32)
    rows, cols, o = [64, 64, 64, 64, 16], [layout.n_inputs, 64, 64, 64, 64], 0
    for r, c in zip(rows, cols):
        p[o:o + r * c] *= math.sqrt(6.0 / (c + min(r, 64))) / 0.6
        o += r * c
    p[o - 8 * 64:o] = 0.0  # padding rows of the output matrix
    return p


def _build(model, precision="fp16", batch=1 << 18):
    cfg = nb.reference_default_config() if model == "refdef" else nb.default_config()
    cfg.network.precision = PRECISIONS[precision]
    cfg.neural_bvh_max_depth = 10
    cfg.batch_size = batch
    h = nb.NBVH(cfg)
    v, f, alb = _once("mesh", _mesh)
    h.set_mesh(v, f, alb)
    h.build_classic()
    h.build_neural_cut()
    h.set_params(_refdef_params(h.layout) if model == "refdef" else _once("trained", _trained_params))
    return h


def _model(model, precision="fp16"):
    return _once(("model", model, precision), lambda: _build(model, precision))


# ------------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _uniform_rays(n, seed):
    """Origins uniform in the scene box scaled by 1.5, directions uniform on the sphere."""
    g = _gen(seed)
    v = _once("mesh", _mesh)[0]
    lo, hi = (torch.from_numpy(b).cuda() for b in (v.min(0), v.max(0)))
    o = lo + (torch.rand((n, 3), device="cuda", generator=g) * 1.5 - 0.25) * (hi - lo)
    d = torch.randn((n, 3), device="cuda", generator=g)
    return _rays(o, d)


def _surface_rays(n, seed):
    """Secondary rays: from just above the surface into the outer hemisphere."""
    g = _gen(seed)
    v, f, _ = _once("mesh", _mesh)
    vt, ft = torch.from_numpy(v).cuda(), torch.from_numpy(f.astype(np.int64)).cuda()
    tri = vt[ft[torch.randint(len(f), (n,), device="cuda", generator=g)]]
    w = torch.rand((n, 2), device="cuda", generator=g)
    w = torch.where(w.sum(1, keepdim=True) > 1, 1 - w, w)
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    p = tri[:, 0] + w[:, :1] * e1 + w[:, 1:] * e2
    nrm = torch.nn.functional.normalize(torch.linalg.cross(e1, e2), dim=1)
    out = p - vt.mean(0)
    nrm = torch.where((nrm * out).sum(1, keepdim=True) < 0, -nrm, nrm)
    d = torch.nn.functional.normalize(torch.randn((n, 3), device="cuda", generator=g), dim=1) + nrm
    return _rays(p + 1e-3 * nrm, d)


def _rays(o, d):
    r = torch.empty((o.shape[0], 8), device="cuda")
    r[:, 0:3] = o
    r[:, 3] = 1e-4
    r[:, 4:7] = torch.nn.functional.normalize(d, dim=1)
    r[:, 7] = FLT_MAX
    return r.contiguous()


def _segment_points(n, seed):
    """Encoded points of n leaf segments near the surface: 4 stratified points of a short segment."""
    g = _gen(seed)
    v = _once("mesh", _mesh)[0]
    vt = torch.from_numpy(v).cuda()
    mid = vt[torch.randint(len(v), (n,), device="cuda", generator=g)]
    d = torch.nn.functional.normalize(torch.randn((n, 3), device="cuda", generator=g), dim=1)
    length = 0.02 + 0.06 * torch.rand((n, 1), device="cuda", generator=g)
    t = (torch.arange(4, device="cuda") + 0.5) / 4 - torch.rand((n, 1), device="cuda", generator=g)
    p = mid[:, None, :] + (t * length)[:, :, None] * d[:, None, :]
    lo, hi = vt.amin(0), vt.amax(0)
    return ((p - 0.5 * (lo + hi)) / (hi - lo) + 0.5).clamp(0.0, 1.0).contiguous()


def _feature_rows(case, seed):
    """Encoded rows of real segments, in the MLP's type."""
    dt = torch.bfloat16 if case["precision"] == "bf16" else torch.float16
    table = _network()[1]
    return torch.cat([_grid_features(p, table).to(dt) for p in _segment_points(case["n"], seed).split(1 << 16)])


def _targets(n, seed):
    """Labels of a batch: about half the segments hit; depth, normal and albedo in [0, 1]."""
    g = _gen(seed + 77)
    t = torch.rand((n, 8), device="cuda", generator=g)
    t[:, 0] = (t[:, 0] < 0.5).float()
    return (t * t[:, :1]).contiguous()


def _camera(case, seed):
    v = _once("mesh", _mesh)[0]
    o, tgt, up = scenes.orbit_camera(v.min(0), v.max(0), seed=int(seed))
    return nb.render_request(case["width"], case["height"], o, tgt, up, sample_idx=int(seed) % 1000)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("closest", "visibility"):
        rays = _uniform_rays(case["n"], seed) if case["depth"] == 1 else _surface_rays(case["n"], seed)
        return {"case": case, "h": _model(case["model"]), "rays": rays,
                "out": torch.empty((case["n"], 12), dtype=torch.int32, device="cuda")}
    if kind == "host":
        rays = _uniform_rays(case["n"], seed) if case["depth"] == 1 else _surface_rays(case["n"], seed)
        return {"case": case, "h": _model(case["model"]), "rays": nb.pinned_copy(rays.cpu().numpy()),
                "out": nb.pinned_empty(case["n"], nb.NEURAL_HIT_DTYPE)}
    if kind == "classic":
        return {"case": case, "h": _model("sphere"), "rays": _uniform_rays(case["n"], seed),
                "out": torch.empty((case["n"], 4), dtype=torch.int32, device="cuda")}
    if kind == "frame":
        return {"case": case, "h": _model(case["model"]), "req": _camera(case, seed)}
    if kind == "path":
        req = nb.path_request(_camera(case, seed), spp=case["spp"], max_bounces=case["bounces"],
                              seed=int(seed) & 0xFFFF, ground_height=-0.01)
        return {"case": case, "h": _model(case["model"]), "req": req}
    if kind == "mlp":
        return {"case": case, "h": _model("sphere", case["precision"]), "x": _feature_rows(case, seed)}
    if kind == "network":
        return {"case": case, "h": _model("sphere", case["precision"]), "pos": _segment_points(case["n"], seed)}
    if kind == "gradients":
        return {"case": case, "h": _model("sphere", case["precision"]), "pos": _segment_points(case["n"], seed),
                "tgt": _targets(case["n"], seed)}
    # a training program's own model: its weights change with every pass
    return {"case": case, "h": _build("sphere", case["precision"], batch=case["n"]), "step": int(seed) % 4096}


def run(state):
    case, h = state["case"], state["h"]
    kind = case["kind"]
    if kind == "closest":
        return _hits(h.query_closest_neural(state["rays"], case["depth"], state["out"]).view(torch.float32))
    if kind == "visibility":
        return _hits(h.query_visibility_neural(state["rays"], case["depth"], state["out"]).view(torch.float32))
    if kind == "host":
        r = h.query_closest_neural_host(state["rays"], case["depth"], state["out"])
        return {k: r[k] for k in ("t", "normal", "albedo", "visibility", "flags", "segments")}
    if kind == "frame":
        return _hits(h.run_inference(state["req"]).view(torch.float32))
    if kind == "path":
        img, traced = h.render_path(state["req"])
        return {"image": img, "rays": traced}
    if kind == "classic":
        q = h.query_any_classic if case["any"] else h.query_closest_classic
        r = q(state["rays"], state["out"])
        f = r.view(torch.float32)
        return {"t": f[:, 0], "u": f[:, 1], "v": f[:, 2], "prim": r[:, 3]}
    if kind == "mlp":
        return h.mlp_inference(state["x"])
    if kind == "network":
        return h.network_inference(state["pos"])
    if kind == "gradients":
        g, loss = h.compute_gradients(state["pos"], state["tgt"])
        return {"gradient": g, "loss": loss}
    pos, tgt, nodes = h.generate_training_batch(state["step"] + h.training_step, case["n"])
    g, loss = h.compute_gradients(pos, tgt)
    h.adam_step(g)
    return {"positions": pos, "targets": tgt, "nodes": nodes, "gradient": g, "loss": loss}


def _hits(f):
    i = f.view(torch.int32)
    return {"t": f[:, 0], "normal": f[:, 1:4], "albedo": f[:, 4:7], "visibility": f[:, 7], "flags": i[:, 8],
            "segments": i[:, 9], "prim": i[:, 10]}


# ------------------------------------------------------------------------------------------------
# Work a pass cannot do without
# ------------------------------------------------------------------------------------------------

TABLE = {"sphere": 6098120 * 4, "refdef": 1348096 * 8}  # bytes of the 16-bit table
MLP_FLOPS = {"sphere": 43008, "refdef": 38912}          # 2 x weights, per segment
CLASSIC_BVH = 73831 * 32 + 65536 * 48


def work(case):
    kind = case["kind"]
    if kind in ("closest", "visibility", "host", "frame"):
        n = case["width"] * case["height"] if kind == "frame" else case["n"]
        rays_in = 0 if kind == "frame" else 32 * n
        seg = n * SEGMENTS_PER_RAY["camera" if kind == "frame" else "uniform" if case["depth"] == 1 else "surface"]
        return {"bytes": rays_in + 48 * n + min(TABLE[case["model"]], 2048 * seg), "flops": seg * MLP_FLOPS[case["model"]]}
    if kind == "path":
        n = case["width"] * case["height"] * case["spp"]
        rays = n * (1 + 0.4 * case["bounces"])
        return {"bytes": 16 * case["width"] * case["height"] + min(TABLE["sphere"], 2048 * rays),
                "flops": rays * SEGMENTS_PER_RAY["camera"] * MLP_FLOPS["sphere"]}
    if kind == "classic":
        return {"bytes": 48 * case["n"] + min(CLASSIC_BVH, 2048 * case["n"]), "flops": 1000 * case["n"]}
    n = case["n"]
    if kind == "mlp":
        return {"bytes": n * (256 + 32) + 43008, "flops": n * 43008}
    if kind == "network":
        return {"bytes": n * (48 + 32) + min(TABLE["sphere"], 2048 * n) + 43008, "flops": n * (43008 + 4 * 16 * 8 * 4)}
    n_params = 12217744
    b = n * (48 + 32) + min(TABLE["sphere"], 2048 * n) + 4 * n_params
    if kind == "train":
        b += n * 4 + (4 * 4 + 3 * 4 + 2) * n_params  # Adam: gradient, weights and moments in, out again
    return {"bytes": b, "flops": n * 3 * (43008 + 4 * 16 * 8 * 4)}


# ------------------------------------------------------------------------------------------------
# 64-bit values
# ------------------------------------------------------------------------------------------------

def _grid_features(pos, table):
    """Multiresolution hash grid of the sphere model (16 levels x 2 features x 2^19, 16 .. 2048)."""
    n = pos.shape[0] * pos.shape[1]
    x = pos.reshape(n, 3).double()
    scale1 = float(np.float32((2048.0 / 16.0) ** (1.0 / 15.0)))
    out, off = [], 0
    for l in range(16):
        s = float(np.float32(2.0 ** (l * float(np.log2(np.float32(scale1)))) * 16 - 1))
        res = int(math.ceil(s)) + 1
        dense = (res ** 3 + 7) // 8 * 8
        size = min(dense, 1 << 19)
        p = x * s + 0.5
        fl = torch.floor(p)
        w, g = p - fl, fl.long()
        acc = torch.zeros((n, 2), dtype=torch.float64, device=pos.device)
        for c in range(8):
            b = torch.tensor([c & 1, (c >> 1) & 1, (c >> 2) & 1], device=pos.device)
            q = g + b
            if dense > size:
                m = 0xFFFFFFFF
                i = (q[:, 0] ^ ((q[:, 1] * 2654435761) & m) ^ ((q[:, 2] * 805459861) & m)) & (size - 1)
            else:
                i = (q[:, 0] + q[:, 1] * res + q[:, 2] * res * res) % size
            wc = torch.where(b.bool(), w, 1 - w).prod(1, keepdim=True)
            acc = acc + wc * table[off + i]
        out.append(acc)
        off += size
    return torch.stack(out, 1).reshape(pos.shape[0], -1)  # point-major, then level


def _network():
    """The trained matrices and table in 64 bits."""
    p = torch.from_numpy(_once("trained", _trained_params)).cuda().double()
    ws, o = [], 0
    for r, c in ((64, 128), (64, 64), (64, 64), (64, 64), (16, 64)):
        ws.append(p[o:o + r * c].reshape(r, c).clone())
        o += r * c
    return ws, p[o:].reshape(-1, 2).clone()


def _mlp(x, ws):
    for w in ws[:-1]:
        x = torch.relu(x @ w.T)
    return torch.sigmoid(x @ ws[-1][:8].T)


def _classic_exact(rays):
    """Closest hit of every ray against every triangle (Moller-Trumbore) in 64 bits."""
    v, f, _ = _once("mesh", _mesh)
    tri = torch.from_numpy(v).cuda().double()[torch.from_numpy(f.astype(np.int64)).cuda()]
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    res = []
    for r in rays.double().split(1024):
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        pv = torch.linalg.cross(d, e2[None])
        inv = 1.0 / (e1[None] * pv).sum(2)
        tv = o - v0[None]
        u = (tv * pv).sum(2) * inv
        qv = torch.linalg.cross(tv, e1[None])
        w = (d * qv).sum(2) * inv
        t = (e2[None] * qv).sum(2) * inv
        ok = (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (t >= r[:, None, 3])
        t, k = torch.where(ok, t, torch.full_like(t, FLT_MAX)).min(1)
        hit = t < FLT_MAX
        z = torch.zeros_like(t)
        res.append((t, torch.where(hit, u.gather(1, k[:, None])[:, 0], z), torch.where(hit, w.gather(1, k[:, None])[:, 0], z)))
    return [torch.cat(c) for c in zip(*res)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "classic" and case["n"] <= 1 << 15 and not case["any"]:
        t, u, v = _classic_exact(_uniform_rays(case["n"], seed))
        return {"t": t, "u": u, "v": v, "prim": None}
    if kind not in ("mlp", "network", "gradients"):
        return None
    ws, table = _network()
    if kind == "mlp":
        return torch.cat([_mlp(c.double(), ws) for c in _feature_rows(case, seed).split(1 << 18)])
    pos = _segment_points(case["n"], seed)
    if kind == "network":
        return torch.cat([_mlp(_grid_features(c, table), ws) for c in pos.split(1 << 16)])
    if case["precision"] != "fp16":  # the batch sum cancels: 8-bit mantissas say nothing about 64-bit values
        return None
    tgt = _targets(case["n"], seed).double()
    leaves = [w.requires_grad_() for w in ws] + [table.requires_grad_()]
    total = torch.zeros((), dtype=torch.float64, device="cuda")
    for p, t in zip(pos.split(1 << 15), tgt.split(1 << 15)):
        y = _mlp(_grid_features(p, table), ws)
        value, dy = _loss(y.detach(), t, 8 * case["n"])
        total += value
        y.backward(dy)
    return {"gradient": torch.cat([w.grad.reshape(-1) for w in leaves]), "loss": total}


def _loss(y, t, n_total):
    """The default composite loss (BCE visibility, L1 depth, L1 linear normal, relative L2 albedo;
    channels 1 .. 7 only where the target is visible): its value and d value / d y."""
    p = y[:, :1].clamp(1e-5, 1 - 1e-5)
    vis = -(t[:, :1] * p.log() + (1 - t[:, :1]) * (1 - p).log())
    dvis = -(t[:, :1] - p) / (p - p * p)
    dd = y[:, 1:2] - t[:, 1:2]
    lin = (y[:, 2:5] * 2 - 1) / 0.1 * 0.5 + 0.5 - t[:, 2:5]
    da = y[:, 5:8] - t[:, 5:8]
    den = y[:, 5:8] ** 2 + 1e-2
    on = (t[:, :1] >= 0.5).double()
    value = torch.cat([vis, on * dd.abs(), on * lin.abs(), on * da * da / den], 1).sum() / n_total
    one = torch.ones_like
    sgn = lambda x: torch.copysign(one(x), x)  # noqa: E731
    return value, torch.cat([dvis, on * sgn(dd), on * sgn(lin) * 10.0, on * 2 * da / den], 1) / n_total
