"""The work a program has this framework do, as measurable cases.

Every case goes through the framework's public entry points: the methods of
GpuSpace, or the C ABI of include/ilg.h for device-resident batches. Sizes are
those of the repository's own workloads (the 1,048,576-triangle heightfield
with 4,194,304 rays, the icosphere field, the box scene, the batch of uneven
scenes, the radiance cache's 16,384-row training batches) and of its tests.

  op         entry point                         what a case gives
  closest    ilg_intersect, device arrays        prim, t, u, v of every ray
  any        ilg_occluded, device arrays         0 / 1 of every segment
  host       GpuSpace.intersects, numpy arrays   prim, t, u, v of every ray
  rebuild    GpuSpace.build + ilg_intersect      counts of the tree, hits of a few rays
  render     GpuSpace.render                     the image
  batch      GpuSpace.render_batch               every scene's image
  viewer     GpuSpace.render with the cache,     the frame and the displayed image
             then accumulate and tonemap
  infer      ilg_mlp_infer, device arrays        the network's outputs
  grads      ilg_mlp_grads, device arrays        loss and weight gradients
"""
from __future__ import annotations

import math

import numpy as np
import torch

from illuminaprt_b200 import scenes
from illuminaprt_b200.ilg import ILG_DEVICE_PTRS, ILG_MLP_RAW, GpuSpace

DEV = "cuda:0"
FLT_MAX = float(np.finfo(np.float32).max)

# the cache network: 96 encoded columns -> 64 x 5 (ReLU) -> 8 (3 used), no biases
MLP_DIMS = [(96, 64)] + [(64, 64)] * 4 + [(64, 8)]
MLP_WEIGHTS = sum(i * o for i, o in MLP_DIMS)
GRID_LEVELS, GRID_SIZE = 16, 1 << 15
GRID_RES = [int(math.floor(16.0 * 2.0 ** (7.0 * l / 15.0))) for l in range(GRID_LEVELS)]


def listed():
    return [
        # a tool picking or probing a small mesh: one call, host arrays, latency is all of it
        {"name": "pick", "op": "host", "nx": 64, "ny": 32, "rays": 1000, "kind": "incoherent", "watertight": False},
        # a host program's batch from ordinary (pageable) arrays, watertight test, ragged count
        {"name": "host_batch", "op": "host", "nx": 256, "ny": 128, "rays": 300001, "kind": "coherent",
         "watertight": True},
        # the headline ray batch: camera rays, then diffuse bounce rays, on 1,048,576 triangles
        {"name": "camera_rays", "op": "closest", "nx": 1024, "ny": 512, "rays": 4194304, "kind": "coherent",
         "watertight": False},
        {"name": "bounce_rays", "op": "closest", "nx": 1024, "ny": 512, "rays": 4194304, "kind": "incoherent",
         "watertight": False},
        # ambient occlusion: short segments, any hit, ragged count on a mid-size mesh
        {"name": "occlusion", "op": "any", "nx": 397, "ny": 211, "rays": 1000003, "kind": "segments",
         "watertight": False},
        # an animated mesh: the tree is built again, then queried
        {"name": "rebuild", "op": "rebuild", "nx": 512, "ny": 256, "rays": 65536, "fast": False},
        # the box scene at its quoted size, image to the host
        {"name": "box_image", "op": "render", "scene": "box", "side": 0, "subdiv": 0, "width": 256, "height": 256,
         "spp": 16, "depth": 6, "one_launch": False},
        # a frame of the icosphere field (5.2 M triangles), depth 12, image stays on the device
        {"name": "field_image", "op": "render", "scene": "field", "side": 8, "subdiv": 6, "width": 1920,
         "height": 1080, "spp": 4, "depth": 12, "one_launch": False},
        # independent scenes of uneven size in one launch
        {"name": "batch_images", "op": "batch", "scenes": 12, "tris": 200000, "most": 320, "one_launch": True},
        # an interactive viewer: one sample a frame with the learned cache, trained as it goes
        {"name": "viewer_frame", "op": "viewer", "side": 8, "subdiv": 5, "width": 960, "height": 540,
         "encoding": "hashgrid", "tail": 1, "steps": 4, "tone": "drago"},
        # the cache network by itself: a 1080p frame's queries, and one training batch's gradients
        {"name": "cache_queries", "op": "infer", "rows": 2073600, "encoding": "freq12"},
        {"name": "cache_grads", "op": "grads", "rows": 16384, "encoding": "hashgrid"},
    ]


def _spread(rng, lo, hi):
    """A whole number, spread over the logarithm of the range, odd ones as likely as even."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["host", "closest", "closest", "any", "rebuild", "render", "render", "batch", "viewer", "infer",
                     "grads"])
    if op in ("host", "closest", "any"):
        nx = _spread(rng, 32, 1024)
        return {"op": op, "nx": nx, "ny": max(16, nx // 2 - rng.randrange(8)),
                "rays": _spread(rng, 500, 400_000 if op == "host" else 4_000_000),
                "kind": "segments" if op == "any" else rng.choice(["coherent", "incoherent", "incoherent"]),
                "watertight": op != "any" and rng.random() < 0.25}
    if op == "rebuild":
        nx = _spread(rng, 64, 700)
        return {"op": op, "nx": nx, "ny": max(16, nx // 2 - rng.randrange(8)), "rays": _spread(rng, 1000, 65536),
                "fast": rng.random() < 0.3}
    if op == "render":
        if rng.random() < 0.4:
            w = _spread(rng, 32, 400)
            return {"op": op, "scene": "box", "side": 0, "subdiv": 0, "width": w, "height": max(16, w - rng.randrange(16)),
                    "spp": rng.choice([1, 4, 16]), "depth": rng.randint(3, 8), "one_launch": rng.random() < 0.3}
        w = _spread(rng, 160, 1280)
        return {"op": op, "scene": "field", "side": rng.randint(2, 8), "subdiv": rng.randint(3, 6), "width": w,
                "height": w * 9 // 16, "spp": rng.choice([1, 2, 4]), "depth": rng.randint(4, 12),
                "one_launch": rng.random() < 0.25}
    if op == "batch":
        return {"op": op, "scenes": rng.randint(2, 12), "tris": _spread(rng, 20_000, 200_000),
                "most": _spread(rng, 96, 320), "one_launch": rng.random() < 0.6}
    if op == "viewer":
        w = _spread(rng, 160, 960)
        return {"op": op, "side": rng.randint(3, 8), "subdiv": rng.randint(3, 5), "width": w, "height": w * 9 // 16,
                "encoding": rng.choice(["hashgrid", "hashgrid", "freq12"]), "tail": rng.choice([0, 1, 2]),
                "steps": rng.choice([2, 4]), "tone": rng.choice(["global", "auto", "drago"])}
    if op == "infer":
        return {"op": op, "rows": _spread(rng, 500, 2_000_000), "encoding": rng.choice(["freq12", "hashgrid"])}
    return {"op": op, "rows": _spread(rng, 500, 32768), "encoding": rng.choice(["freq12", "hashgrid"])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cpu")
    g.manual_seed(seed)
    return g


def _rays(case, pos, idx, seed):
    """(n, 4) origins and directions on the CPU: camera rays in image order
    from a moving eye, or diffuse rays off random triangles (segments: of a
    finite length, for ambient occlusion)."""
    n, g = case["rays"], _gen(seed)
    u = torch.rand(n, 4, generator=g, dtype=torch.float64)
    if case["kind"] == "coherent":
        side = max(1, int(math.ceil(math.sqrt(n))))
        j = torch.rand(3, generator=g, dtype=torch.float64) * 0.1
        eye = np.array([0.45 + float(j[0]), -0.6 + float(j[1]), 0.75 + float(j[2])])
        o4, d4 = scenes.pinhole_rays(side, side, eye, (0.5, 0.5, 0.0), (0, 0, 1), 60.0)
        return torch.from_numpy(o4[:n]), torch.from_numpy(d4[:n])
    p = torch.from_numpy(pos).double()[torch.from_numpy(idx.astype(np.int64))]
    tri = torch.randint(0, idx.shape[0], (n,), generator=g)
    p0, p1, p2 = p[tri].unbind(1)
    su = u[:, :1].sqrt()
    at = (1 - su) * p0 + u[:, 1:2] * su * p1 + (su - u[:, 1:2] * su) * p2
    w = torch.linalg.cross(p1 - p0, p2 - p0)
    w = w / w.norm(dim=1, keepdim=True)
    w = torch.where(w[:, 2:] < 0, -w, w)
    a = torch.where(w[:, :1].abs() > w[:, 1:2].abs(), torch.tensor([[0.0, 1.0, 0.0]], dtype=torch.float64),
                    torch.tensor([[1.0, 0.0, 0.0]], dtype=torch.float64))
    x = torch.linalg.cross(a, w)
    x = x / x.norm(dim=1, keepdim=True)
    y = torch.linalg.cross(w, x)
    r, phi = u[:, 2:3].sqrt(), 2 * math.pi * u[:, 3:4]
    d = r * phi.cos() * x + r * phi.sin() * y + (1 - u[:, 2:3]).sqrt() * w
    o4, d4 = torch.zeros(n, 4), torch.empty(n, 4)
    o4[:, :3] = at + 1e-4 * w
    d4[:, :3] = d / d.norm(dim=1, keepdim=True)
    d4[:, 3] = 0.1 if case["kind"] == "segments" else FLT_MAX
    return o4, d4


def _network(seed, encoding):
    """Weights with zero unused output columns, and grid features large enough to matter."""
    g = _gen(seed)
    w = []
    for i, o in MLP_DIMS:
        m = (2 * torch.rand(i, o, generator=g) - 1) * math.sqrt(6.0 / (i + o))
        if o == 8:
            m[:, 3:] = 0.0
        w.append(m)
    grid = (torch.rand(GRID_LEVELS, GRID_SIZE, 2, generator=g) * 0.6 - 0.3) if encoding == "hashgrid" else None
    return w, grid


def _queries(rows, seed):
    """Vertices as the path tracer hands them to the cache, and radiance targets."""
    g = _gen(seed + 77)
    raw = torch.zeros(rows, ILG_MLP_RAW)
    raw[:, :3] = torch.rand(rows, 3, generator=g)
    v = torch.randn(rows, 2, 3, generator=g)
    raw[:, 3:9] = (v / v.norm(dim=2, keepdim=True)).reshape(rows, 6)
    raw[:, 9] = torch.where(torch.rand(rows, generator=g) < 0.5, torch.ones(rows), 0.05 + 0.45 * torch.rand(rows, generator=g))
    raw[:, 10:13] = 0.1 + 0.8 * torch.rand(rows, 3, generator=g)
    return raw, torch.exp(torch.randn(rows, 3, generator=g) - 1.0)


def _mesh(case, seed):
    return scenes.heightfield(case["nx"], case["ny"], 0.2, seed)


def _batch(case):
    return scenes.batch_workload(case["scenes"], seed=9, tri_range=(10_000, case["tris"]),
                                 side_range=(64, case["most"]))


def prepare(case, seed):
    op, s = case["op"], {"case": case, "seed": seed}
    if op in ("host", "closest", "any", "rebuild"):
        pos, idx = _mesh(case, seed)
        sp = s["space"] = GpuSpace(device=0, fast_build=bool(case.get("fast")))
        sp.initialise(pos, idx)
        sp.build()
        o4, d4 = _rays({"kind": "incoherent", **case}, pos, idx, seed)
        if op == "host":
            s["o4"], s["d4"] = np.ascontiguousarray(o4.numpy()), np.ascontiguousarray(d4.numpy())
        else:
            n = case["rays"]
            s["o4"], s["d4"] = o4.to(DEV), d4.to(DEV)
            if op == "any":
                s["occ"] = torch.empty(n, dtype=torch.uint8, device=DEV)
            else:
                s["hit"] = (torch.empty(n, dtype=torch.int32, device=DEV),
                            *(torch.empty(n, dtype=torch.float32, device=DEV) for _ in range(3)))
    elif op == "render" and case["scene"] == "box":
        sp = s["space"] = GpuSpace(device=0)
        box = scenes.load_box_scene(sp)
        s["camera"] = dict(box["camera"], aspect=case["width"] / case["height"])
        s["sky"] = (0.0, 0.0, 0.0)
    elif op in ("render", "viewer"):
        w, h = case["width"], case["height"]
        f = scenes.sphere_field(case["side"], case["subdiv"], seed=seed, width=w, height=h)
        sp = s["space"] = GpuSpace(device=0)
        scenes.load_sphere_field(sp, f)
        s["camera"], s["sky"] = f["camera"], f["sky"]
        s["out"] = torch.empty((h, w, 3), dtype=torch.float32, device=DEV)
        if op == "viewer":
            s["mean"], s["shown"] = torch.empty_like(s["out"]), torch.empty_like(s["out"])
            sp.mlp_init(seed=seed, lr=1e-2, encoding=case["encoding"])
    elif op == "batch":
        # sizes do not depend on the seed; every scene is seen from a place of its own
        move = torch.rand(case["scenes"], 3, generator=_gen(seed), dtype=torch.float64).numpy() - 0.5
        s["spaces"], s["items"] = [], []
        for k, f in enumerate(_batch(case)):
            f["camera"]["eye"] = tuple(float(x) for x in np.array(f["camera"]["eye"]) + move[k])
            sp = GpuSpace(device=0)
            scenes.load_sphere_field(sp, f)
            s["spaces"].append(sp)
            s["items"].append({"space": sp, "camera": f["camera"], "width": f["width"], "height": f["height"],
                               "spp": min(f["spp"], 16), "max_depth": f["max_depth"], "seed": seed + k, "sky": f["sky"],
                               "out": torch.empty((f["height"], f["width"], 3), dtype=torch.float32, device=DEV)})
        s["space"] = GpuSpace(device=0)
    else:
        sp = s["space"] = GpuSpace(device=0)
        sp.mlp_init(seed=1, lr=1e-2, encoding=case["encoding"])
        w, grid = _network(seed, case["encoding"])
        sp.mlp_set_params(torch.cat([m.reshape(-1) for m in w]).numpy())
        if grid is not None:
            sp.mlp_set_grid(grid.reshape(-1).numpy())
        raw, target = _queries(case["rows"], seed)
        s["raw"] = raw.to(DEV)
        if op == "infer":
            s["out"] = torch.empty(case["rows"], 3, device=DEV)
        else:
            s["target"] = target.to(DEV)
            s["grad"], s["loss"] = torch.empty(MLP_WEIGHTS, device=DEV), torch.empty(1, device=DEV)
    torch.cuda.synchronize()  # the space's stream does not wait for torch's
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case, sp = s["case"], s["space"]
    op = case["op"]
    if op == "host":
        return sp.intersects(s["o4"], s["d4"], watertight=case["watertight"])
    if op == "closest":
        sp.intersects_into(s["o4"], s["d4"], *s["hit"], device_ptrs=True, watertight=case["watertight"])
        return s["hit"]
    if op == "any":
        sp.occluded_into(s["o4"], s["d4"], s["occ"], device_ptrs=True)
        return s["occ"]
    if op == "rebuild":
        sp.build()
        sp.intersects_into(s["o4"], s["d4"], *s["hit"], device_ptrs=True)
        st = sp.stats()
        return (st["n_tris"], st["n_nodes"], st["max_depth"], *s["hit"])
    if op == "render":
        out = None if case["scene"] == "box" else s["out"]
        return sp.render(s["camera"], case["width"], case["height"], case["spp"], max_depth=case["depth"],
                         seed=s["seed"], sky=s["sky"], out=out, one_launch=case["one_launch"])
    if op == "batch":
        return sp.render_batch(s["items"], device_ptrs=True, one_launch=case["one_launch"])
    if op == "viewer":
        sp.render(s["camera"], case["width"], case["height"], 1, max_depth=12, seed=s["seed"], sky=s["sky"],
                  out=s["out"], cache_depth=1, train_tail=case["tail"], train_steps=case["steps"])
        sp.accumulate(s["out"], s["mean"])
        sp.tonemap(s["mean"], case["tone"], s["shown"])
        return s["out"], s["shown"]
    if op == "infer":
        sp._check(sp.L.ilg_mlp_infer(sp.h, s["raw"].data_ptr(), case["rows"], s["out"].data_ptr(), ILG_DEVICE_PTRS))
        return s["out"]
    sp._check(sp.L.ilg_mlp_grads(sp.h, s["raw"].data_ptr(), s["target"].data_ptr(), case["rows"],
                                 s["grad"].data_ptr(), s["loss"].data_ptr(), ILG_DEVICE_PTRS))
    return s["loss"], s["grad"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    op = case["op"]
    if op in ("host", "closest", "any", "rebuild"):
        # the mesh (36 bytes of vertices a triangle) once, 32 bytes of ray in, 16 bytes (any hit: 1) of hit out;
        # a ray has at least one triangle test of about 50 operations
        tris = 2 * case["nx"] * case["ny"]
        return {"bytes": 36 * tris + case["rays"] * (33 if op == "any" else 48), "flops": 50 * case["rays"]}
    if op in ("render", "viewer"):
        tris = 36 if case.get("scene") == "box" else case["side"] ** 2 * 20 * 4 ** case["subdiv"]
        pixels = case["width"] * case["height"]
        paths = pixels * (case["spp"] if op == "render" else 1)
        # the mesh and the image once; a path has at least a camera ray's triangle test
        more = 2 * pixels * sum(i * o for i, o in MLP_DIMS) if op == "viewer" else 0
        return {"bytes": 36 * tris + pixels * (12 if op == "render" else 48), "flops": 50 * paths + more}
    if op == "batch":
        items = _batch(case)
        return {"bytes": sum(36 * f["idx"].shape[0] + 12 * f["width"] * f["height"] for f in items),
                "flops": sum(50 * f["width"] * f["height"] * min(f["spp"], 16) for f in items)}
    macs = sum(i * o for i, o in MLP_DIMS)
    grid = 4 * GRID_LEVELS * GRID_SIZE * 2 if case["encoding"] == "hashgrid" else 0
    if op == "infer":
        return {"bytes": case["rows"] * 76 + grid + 4 * macs, "flops": 2 * macs * case["rows"]}
    return {"bytes": case["rows"] * 76 + 2 * grid + 8 * macs, "flops": 6 * macs * case["rows"]}


# ---------------------------------------------------------------------------
# results in 64 bits
# ---------------------------------------------------------------------------
def _encode64(raw, grid):
    """The 96 input columns in float64 (grid None: the 12-band frequency encoding)."""
    x = raw[:, :3].double()
    one = torch.ones(x.shape[0], 1, dtype=torch.float64, device=x.device)
    bands = 12 if grid is None else 4
    arg = x[:, :, None] * (math.pi * 2.0 ** torch.arange(bands, device=x.device, dtype=torch.float64))
    wave = torch.stack([arg.sin(), arg.cos()], 3).reshape(x.shape[0], -1)
    f = raw.double()
    if grid is None:
        cols = [wave, f[:, 3:13], one]
    else:
        feats = []
        for l, res in enumerate(GRID_RES):
            p = x.clamp(0, 1) * res
            i = p.floor().long().clamp(max=res - 1)
            fr = p - i
            acc = 0
            for c in range(8):
                b = torch.tensor([(c >> k) & 1 for k in range(3)], device=x.device)
                at, w = i + b, torch.where(b.bool(), fr, 1 - fr).prod(1, keepdim=True)
                if (res + 1) ** 3 <= GRID_SIZE:
                    e = at[:, 0] + (res + 1) * (at[:, 1] + (res + 1) * at[:, 2])
                else:
                    e = (at[:, 0] ^ (at[:, 1] * 2654435761) ^ (at[:, 2] * 805459861)) & (GRID_SIZE - 1)
                acc = acc + w * grid[l][e]
            feats.append(acc)
        a, b, c = f[:, 3], f[:, 4], f[:, 5]
        sh = torch.stack([0.28209479177387814 + 0 * a, -0.48860251190291987 * b, 0.48860251190291987 * c,
                          -0.48860251190291987 * a, 1.0925484305920792 * a * b, -1.0925484305920792 * b * c,
                          0.94617469575755997 * c * c - 0.31539156525251999, -1.0925484305920792 * a * c,
                          0.54627421529603959 * (a * a - b * b), 0.59004358992664352 * b * (3 * a * a - b * b),
                          2.8906114426405538 * a * b * c, 0.45704579946446572 * b * (5 * c * c - 1),
                          0.3731763325901154 * c * (5 * c * c - 3), 0.45704579946446572 * a * (5 * c * c - 1),
                          1.4453057213202769 * c * (a * a - b * b), 0.59004358992664352 * a * (a * a - 3 * b * b)], 1)
        cols = [*feats, wave, sh, f[:, 6:9], f[:, 9:13], one]
    out = torch.cat(cols, 1)
    return torch.cat([out, torch.zeros(x.shape[0], 96 - out.shape[1], dtype=torch.float64, device=x.device)], 1)


def _net64(x, w):
    for m in w[:-1]:
        x = (x @ m).relu()
    return x @ w[-1]


def exact(case, seed):
    op = case["op"]
    if op in ("host", "closest") and not case["watertight"] and 2 * case["nx"] * case["ny"] * case["rays"] <= 2e8:
        # the plane-and-edges test of every triangle, smallest t in the window [1e-5, max]
        pos, idx = _mesh(case, seed)
        o4, d4 = _rays(case, pos, idx, seed)
        o, d = o4[:, :3].double().to(DEV), d4[:, :3].double().to(DEV)
        v = torch.from_numpy(pos).double()[torch.from_numpy(idx.astype(np.int64))].to(DEV)
        e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        n = torch.linalg.cross(e1, e2)
        ts, us, vs = [], [], []
        for k in range(0, o.shape[0], 512):
            oo, dd = o[k:k + 512, None], d[k:k + 512, None]
            den = (n * dd).sum(2)
            e = v[:, 0] - oo
            t = (n * e).sum(2) / den
            q = torch.linalg.cross(dd.expand_as(e), e)
            b, c = -(q * e2).sum(2) / den, (q * e1).sum(2) / den
            t = torch.where((t >= 1e-5) & (b >= 0) & (c >= 0) & (b + c <= 1), t, torch.inf)
            t, at = t.min(1, keepdim=True)
            hit = t.isfinite()
            ts.append(t)
            us.append(torch.where(hit, b.gather(1, at), 0.0))
            vs.append(torch.where(hit, c.gather(1, at), 0.0))
        return (None, *(torch.cat(x)[:, 0] for x in (ts, us, vs)))
    if op not in ("infer", "grads"):
        return None  # a Monte Carlo image, or a search over more triangles than a plain loop can take
    w, grid = _network(seed, case["encoding"])
    w = [m.double().to(DEV) for m in w]
    grid = None if grid is None else grid.double().to(DEV)
    raw, target = (x.to(DEV) for x in _queries(case["rows"], seed))
    if op == "infer":
        return torch.cat([_net64(_encode64(r, grid), w)[:, :3] for r in raw.split(1 << 18)])
    w = [m.requires_grad_() for m in w]
    y = _net64(_encode64(raw, grid), w)[:, :3]
    loss = ((y - target.double()) ** 2 / (y.detach() ** 2 + 0.01)).mean()
    grads = torch.autograd.grad(loss, w)
    return loss.detach().reshape(1), torch.cat([m.reshape(-1) for m in grads])
