"""The workloads whose speed this repository is judged by, each through the public
entry points that a user's program calls.

    listed()              the named cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   what the program holds before the call, on the GPU
    run(state)            one pass; its outputs, whole
    work(case)            bytes and operations a pass cannot do without
    exact(case, seed)     the outputs in 64 bits, where they have such a value

A case is a dict of plain values; "kind" is one of
    trace   closest-hit or any-hit queries over rays in device or in host memory
    render  one frame of a scene by one of the shaders
    batch   many small frames of one scene in one pass
    ltc     polygon-light shading of a G-buffer
    infer   the light-selection network over shading points
    train   Adam steps of that network over recorded light samples
"""
from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

from chakumrender_gb300 import ckr
from chakumrender_gb300 import scene as S
from chakumrender_gb300.batch import Batch, BatchTuning, Job, box_jobs
from chakumrender_gb300.proposal import NPARAMS, Proposal

ROOM = dict(nemit=128, nclusters=64)  # the small many-light room of the network cases


def listed():
    return [
        # An offline ray-query service over a scanned mesh: the repository's headline
        # batch, half camera rays and half incoherent ones.
        {"name": "closest_1310k_8m", "kind": "trace", "any": False, "host": "", "subdiv": 8, "nsph": 0, "n": 1 << 23,
         "rays": "mixed"},
        # Visibility queries of a lighting pass: any hit over a mid-size mesh, with the
        # ray lengths of shadow rays; an odd count.
        {"name": "any_82k_1m", "kind": "trace", "any": True, "host": "", "subdiv": 6, "nsph": 0, "n": 1000003,
         "rays": "incoherent"},
        # A picking or collision query: few rays, a small mesh with a few spheres, latency.
        {"name": "closest_1280_1k", "kind": "trace", "any": False, "host": "", "subdiv": 3, "nsph": 3, "n": 1013,
         "rays": "mixed"},
        # A caller that holds its rays in host memory, as every caller of the reference
        # does: pinned buffers, copies inside the call.
        {"name": "host_closest_328k_2m", "kind": "trace", "any": False, "host": "pinned", "subdiv": 7, "nsph": 0,
         "n": 1 << 21, "rays": "mixed"},
        # The path tracer on the box scene at the size of its scene file.
        {"name": "box_path_256", "kind": "render", "scene": "box", "shader": S.SHADER_PATH, "width": 256, "height": 256,
         "spp": 16, "depth": 4, "n_light": 1, "n_brdf": 1, "env": False},
        # The reference's default shader with its default sample counts.
        {"name": "box_miscv_512", "kind": "render", "scene": "box", "shader": S.SHADER_DIRECT_MISCV, "width": 512,
         "height": 512, "spp": 4, "depth": 1, "n_light": 10, "n_brdf": 60, "env": False},
        # An interactive preview: one sample per pixel, direct light with an environment
        # map, a window of no round size.
        {"name": "box_mis_env_preview", "kind": "render", "scene": "box", "shader": S.SHADER_DIRECT_MIS, "width": 163,
         "height": 121, "spp": 1, "depth": 1, "n_light": 1, "n_brdf": 2, "env": True},
        # A final frame of the many-light scene, 1.3M triangles and 4,096 emitters.
        {"name": "manylight_nee_1080p", "kind": "render", "scene": "manylight", "subdiv": 8, "shader": S.SHADER_PATH_NEE,
         "width": 1920, "height": 1080, "spp": 8, "depth": 6, "n_light": 1, "n_brdf": 1, "env": False},
        # Thumbnails and parameter sweeps: many small frames of one scene in one pass.
        {"name": "batch_512_small", "kind": "batch", "njobs": 512, "size_lo": 32, "size_hi": 64},
        # Deferred shading of a frame under rectangular lights.
        {"name": "ltc_1024_8quads", "kind": "ltc", "width": 1024, "height": 1024, "quads": 8},
        # The light-selection network over the vertices of one bounce, and its training on
        # the records of a bounce (65,536 records in minibatches of 4,096).
        {"name": "proposal_infer_256k", "kind": "infer", "n": 1 << 18},
        {"name": "proposal_train_64k", "kind": "train", "n": 65536, "minibatch": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "render", "render", "render", "batch", "ltc", "ltc", "infer", "train"])
    if kind == "trace":
        host = rng.choice(["", "", "", "pinned", "pageable"])
        return {"kind": "trace", "any": rng.random() < 0.4, "host": host, "subdiv": rng.randint(2, 8),
                "nsph": rng.choice([0, 0, 1, 3, 6]), "n": _log_int(rng, 32, 1 << (21 if host else 23)),
                "rays": rng.choice(["mixed", "primary", "incoherent"])}
    if kind == "render":
        if rng.random() < 0.3:
            return {"kind": "render", "scene": "manylight", "subdiv": rng.randint(3, 8), "shader": S.SHADER_PATH_NEE,
                    "width": _log_int(rng, 64, 1920), "height": _log_int(rng, 36, 1080), "spp": rng.randint(1, 8),
                    "depth": rng.randint(2, 6), "n_light": 1, "n_brdf": 1, "env": False}
        shader = rng.choice([S.SHADER_PATH, S.SHADER_PATH, S.SHADER_DIRECT_MISCV, S.SHADER_DIRECT_MIS,
                             S.SHADER_DIRECT_CV, S.SHADER_EXPLICIT])
        many = shader in (S.SHADER_DIRECT_MISCV, S.SHADER_DIRECT_MIS) and rng.random() < 0.5
        return {"kind": "render", "scene": "box", "shader": shader, "width": _log_int(rng, 32, 512),
                "height": _log_int(rng, 32, 512), "spp": rng.choice([1, 2, 3, 4, 8, 16]) if not many else rng.randint(1, 4),
                "depth": rng.randint(2, 6) if shader in (S.SHADER_PATH, S.SHADER_EXPLICIT) else 1,
                "n_light": 10 if many else rng.randint(1, 3), "n_brdf": 60 if many else rng.randint(1, 6),
                "env": shader in (S.SHADER_PATH, S.SHADER_DIRECT_MIS) and rng.random() < 0.4}
    if kind == "batch":
        lo = rng.randint(24, 64)
        return {"kind": "batch", "njobs": _log_int(rng, 4, 512), "size_lo": lo, "size_hi": lo + rng.randint(1, 64)}
    if kind == "ltc":
        return {"kind": "ltc", "width": _log_int(rng, 8, 1400), "height": _log_int(rng, 8, 1024),
                "quads": _log_int(rng, 1, 16)}
    if kind == "infer":
        return {"kind": "infer", "n": _log_int(rng, 16, 1 << 20)}
    return {"kind": "train", "n": _log_int(rng, 64, 65536), "minibatch": rng.choice([1024, 3000, 4096, 16384])}


# ---- inputs ------------------------------------------------------------------------
def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _mesh(case, seed):
    return ckr.icosphere(case["subdiv"], 0.05, 6, 1 + seed % 1000)


def _spheres(case, seed):
    rng = np.random.default_rng(seed)
    n = case["nsph"]
    return np.concatenate([rng.uniform(-1.4, 1.4, (n, 3)), rng.uniform(0.05, 0.4, (n, 1))], 1).astype(np.float32)


FAR = 100.0  # tmax of rays without an end of their own


def _rays(case, seed, device="cuda"):
    """n rays (ox oy oz tmin dx dy dz tmax): camera rays of a 40 degree pinhole at
    distance 3, then rays with origins in the mesh's box and uniform directions."""
    n, kind = case["n"], case["rays"]
    n_prim = {"mixed": n // 2, "primary": n, "incoherent": 0}[kind]
    g = _gen(seed, device)
    r = torch.zeros(n, 8, device=device)
    if n_prim:
        side = max(1, math.isqrt(n_prim))
        i = torch.arange(n_prim, device=device)
        half = math.tan(math.radians(20.0))
        u = ((i % side) + 0.5) / side * 2 - 1
        v = 1 - (torch.div(i, side, rounding_mode="floor") % side + 0.5) / side * 2
        turn = 2 * math.pi * ((seed % 997) / 997.0)
        c, s = math.cos(turn), math.sin(turn)
        d = _unit(torch.stack([u * half, v * half, -torch.ones_like(u)], 1))
        r[:n_prim, 0], r[:n_prim, 2] = 3 * s, 3 * c
        r[:n_prim, 4], r[:n_prim, 5], r[:n_prim, 6] = c * d[:, 0] + s * d[:, 2], d[:, 1], -s * d[:, 0] + c * d[:, 2]
    m = n - n_prim
    if m:
        r[n_prim:, 0:3] = torch.rand(m, 3, device=device, generator=g) * 2.1 - 1.05
        r[n_prim:, 4:7] = _unit(torch.randn(m, 3, device=device, generator=g))
    r[:, 7] = FAR
    if case["any"] and m:
        r[n_prim:, 7] = 0.1 + 1.9 * torch.rand(m, device=device, generator=g)
    return r


def _gbuffer(case, seed):
    """G-buffer rows (pos, alpha, n, f0, v, spec): positions in [-1, 1]^3, normals on the
    upper hemisphere, views cosine-distributed about them; and the quads' triangles."""
    n, g = case["width"] * case["height"], _gen(seed)

    def rand(*shape):
        return torch.rand(*shape, device="cuda", generator=g)

    x = rand(n, 3) * 2 - 1
    nz, ph = rand(n), rand(n) * 2 * math.pi
    st = (1 - nz * nz).clamp_min(0).sqrt()
    nn = _unit(torch.stack([st * ph.cos(), st * ph.sin(), nz], 1))
    v = _unit(_unit(torch.randn(n, 3, device="cuda", generator=g)) * 0.999 + nn)
    rows = torch.cat([x, 0.05 + 0.95 * rand(n, 1), nn, 0.02 + 0.88 * rand(n, 1), v, rand(n, 1)], 1).contiguous()
    q = case["quads"]
    side, c = 0.2 + 0.8 * rand(q, 1), torch.cat([rand(q, 2) * 4 - 2, 1 + 2 * rand(q, 1)], 1)
    corner = torch.tensor([[-0.5, -0.5, 0], [0.5, -0.5, 0], [0.5, 0.5, 0], [-0.5, 0.5, 0]], device="cuda")
    p = c[:, None, :] + side[:, None, :] * corner[None]
    tri = torch.stack([p[:, [0, 2, 1]], p[:, [0, 3, 2]]], 1).reshape(2 * q, 9).contiguous()
    rgb = (2 + 6 * rand(q, 1, 3)).expand(q, 2, 3).reshape(2 * q, 3).contiguous()
    return rows, tri, rgb


def _params(seed):
    rng = np.random.default_rng(seed)
    w = rng.normal(size=NPARAMS)
    w[:64 * 96] *= math.sqrt(2.0 / 96)
    w[64 * 96:] *= math.sqrt(2.0 / 64)
    w[-(64 * 64 + 64):] *= 0.5
    return w.astype(np.float32)


def _records(n, seed):
    """Shading points of the room with a cluster and the radiance its light sample
    brought (a quarter of them blocked)."""
    g = _gen(seed)
    r = torch.zeros(n, 12, device="cuda")
    r[:, 0:3] = torch.rand(n, 3, device="cuda", generator=g) * 9 - 4.5
    r[:, 3] = 0.1 + 0.7 * torch.rand(n, device="cuda", generator=g)
    r[:, 4:7] = _unit(torch.randn(n, 3, device="cuda", generator=g))
    r[:, 8:11] = _unit(_unit(torch.randn(n, 3, device="cuda", generator=g)) * 0.999 + r[:, 4:7])
    w = torch.exp(torch.randn(n, device="cuda", generator=g))
    r[:, 7] = torch.where(torch.rand(n, device="cuda", generator=g) < 0.25, torch.zeros_like(w), w)
    near = (r[:, 0] + 4.5) / 9 * 40 + torch.rand(n, device="cuda", generator=g) * 24
    r[:, 11] = near.to(torch.int32).clamp(0, 63).view(torch.float32)
    return r


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _env_image(seed, h=32, w=64):
    rng = np.random.default_rng(seed)
    sky = np.linspace(1.0, 0.2, h)[:, None, None] * np.array([0.5, 0.7, 1.0])
    img = np.broadcast_to(sky, (h, w, 3)) * rng.uniform(0.6, 1.4, (h, w, 1))
    img[h // 5, w // 3] += 40.0
    return img.astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "trace":
        st["scene"] = ckr.Scene(_mesh(case, seed), _spheres(case, seed) if case["nsph"] else None)
        rays, n = _rays(case, seed), case["n"]
        if not case["host"]:
            st["rays"] = rays
            if case["any"]:
                st["occ"] = torch.empty(n, dtype=torch.uint8, device="cuda")
            else:
                st["id"] = torch.empty(n, dtype=torch.int32, device="cuda")
                st["t"] = torch.empty(n, dtype=torch.float32, device="cuda")
        elif case["host"] == "pageable":
            st["rays"] = rays.cpu().numpy()
        else:
            st["rays"] = rays.cpu().pin_memory()
            if case["any"]:
                st["occ"] = torch.empty(n, dtype=torch.uint8).pin_memory()
            else:
                st["id"] = torch.empty(n, dtype=torch.int32).pin_memory()
                st["t"] = torch.empty(n, dtype=torch.float32).pin_memory()
    elif kind == "render":
        if case["scene"] == "box":
            sd = S.load_xml(S.SCENES / "box.xml")
            if case["env"]:
                sd.set_env(_env_image(seed), n_samples=2)
        else:
            sd = S.manylight_scene(S.manylight_spec(subdiv=case["subdiv"], rough_seed=3 + seed % 1000,
                                                    width=case["width"], height=case["height"]))
        cam = sd.camera
        cam.width, cam.height = case["width"], case["height"]
        st["scene"], st["cam"] = S.RenderScene(sd), cam
        st["cfg"] = S.render_cfg(shader=case["shader"], spp=case["spp"], max_depth=case["depth"],
                                 n_light=case["n_light"], n_brdf=case["n_brdf"], seed=seed)
        st["rgb"] = torch.empty(case["height"], case["width"], 3, device="cuda")
    elif kind == "batch":
        sd = S.load_xml(S.SCENES / "box.xml")
        sizes = tuple(sorted({case["size_lo"], (case["size_lo"] + case["size_hi"]) // 2, case["size_hi"]}))
        # The jobs' sizes are the case's; their random streams are the seed's.
        params, mats = box_jobs(sd, case["njobs"], 4, sizes, (1, 2, 4), (3, 6))
        px = [p["cam"].width * p["cam"].height for p in params]
        st["rgb"] = torch.empty(sum(px), 3, device="cuda")
        at, jobs = st["rgb"].data_ptr(), []
        for p, k in zip(params, px):
            jobs.append(Job(p["cam"], p["spp"], p["max_depth"], seed * 4096 + p["seed"], p["material_set"], 0, at))
            at += 12 * k
        # The tuning that the autotuner finds for batches of this kind, kept by the program.
        st["batch"] = Batch(S.RenderScene(sd), jobs, mats, tuning=BatchTuning(256, 1 << 21, 0.0, 0, 0))
    elif kind == "ltc":
        st["gbuf"], st["tri"], st["rgb_light"] = _gbuffer(case, seed)
        st["rgb"] = torch.empty(case["width"] * case["height"], 3, device="cuda")
    else:
        sd = S.manylight_scene(S.manylight_spec(subdiv=2, width=16, height=9, **ROOM))
        st["prop"] = Proposal(S.RenderScene(sd), seed=1, lr=1e-3)
        st["prop"].set_params(_params(seed))
        st["rec"] = _records(case["n"], seed)
        if kind == "infer":
            st["probs"] = torch.empty(case["n"], 64, dtype=torch.float16, device="cuda")
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "trace":
        n, sc = case["n"], st["scene"]
        if case["host"] == "pageable":
            if case["any"]:
                return sc.trace_any_host(st["rays"])
            ids, t = sc.trace_closest_host(st["rays"])
            return ids.view(np.int32), t
        if case["host"]:
            if case["any"]:
                ckr.check(ckr.lib().ckr_trace_any_host(sc.handle, st["rays"].data_ptr(), n, st["occ"].data_ptr(), _stream()),
                          "ckr_trace_any_host")
                return st["occ"]
            ckr.check(ckr.lib().ckr_trace_closest_host(sc.handle, st["rays"].data_ptr(), n, st["id"].data_ptr(),
                                                       st["t"].data_ptr(), _stream()), "ckr_trace_closest_host")
            return st["id"], st["t"]
        if case["any"]:
            sc.trace_any(st["rays"].data_ptr(), n, st["occ"].data_ptr(), _stream())
            return st["occ"]
        sc.trace_closest(st["rays"].data_ptr(), n, st["id"].data_ptr(), st["t"].data_ptr(), _stream())
        return st["id"], st["t"]
    if kind == "render":
        st["scene"].render(st["cam"], st["cfg"], st["rgb"].data_ptr(), None, _stream())
        return st["rgb"]
    if kind == "batch":
        st["batch"].render(_stream())
        return st["rgb"]
    if kind == "ltc":
        ckr.ltc_shade(st["gbuf"].data_ptr(), st["gbuf"].shape[0], st["tri"].data_ptr(), st["rgb_light"].data_ptr(),
                      st["tri"].shape[0], st["rgb"].data_ptr(), _stream())
        return st["rgb"]
    if kind == "infer":
        st["prop"].infer(st["rec"].data_ptr(), case["n"], st["probs"].data_ptr(), _stream())
        return st["probs"]
    for off in range(0, case["n"], case["minibatch"]):
        st["prop"].train_step(st["rec"][off:].data_ptr(), min(case["minibatch"], case["n"] - off), _stream())
    return st["prop"].params()


# ---- work --------------------------------------------------------------------------
BOX_TEST, TRI_TEST, SPHERE_TEST = 16, 60, 30  # operations of one test
VERTEX = 400                                  # of shading one vertex with one light and one BRDF sample


def _ray_ops(ntri, nsph):
    return BOX_TEST * 2 * math.log2(max(2, ntri)) + TRI_TEST + SPHERE_TEST * nsph


def work(case):
    kind = case["kind"]
    if kind == "trace":
        ntri = 20 * 4 ** case["subdiv"]
        return {"bytes": case["n"] * (32 + (1 if case["any"] else 8)) + 36 * ntri + 16 * case["nsph"],
                "flops": case["n"] * _ray_ops(ntri, case["nsph"])}
    if kind == "render":
        px = case["width"] * case["height"]
        box = case["scene"] == "box"
        ntri, nsph = (13, 3) if box else (20 * 4 ** case["subdiv"] + 12 + 4096, 0)
        # Camera rays all meet something; a path goes on with probability 0.7.
        vertices = sum(0.7 ** k for k in range(case["depth"]))
        direct = case["n_light"] + (case["n_brdf"] if case["shader"] in (0, 1) else 1)
        rays = 1 + (0 if case["shader"] == S.SHADER_DIRECT_MISCV else case["n_light"])
        ops = px * case["spp"] * vertices * (rays * _ray_ops(ntri, nsph) + 0.5 * VERTEX * direct)
        return {"bytes": 12 * px + (36 + 4) * ntri, "flops": ops}
    if kind == "batch":
        px = case["njobs"] * ((case["size_lo"] + case["size_hi"]) / 2) ** 2
        return {"bytes": 12 * px, "flops": px * 7 / 3 * 2.5 * (2 * _ray_ops(13, 3) + VERTEX)}
    if kind == "ltc":
        n = case["width"] * case["height"]
        return {"bytes": 60 * n + 96 * case["quads"], "flops": n * (90 + 2 * case["quads"] * 267)}
    layers = 2 * (96 * 64 + 3 * 64 * 64)
    if kind == "infer":
        return {"bytes": case["n"] * (48 + 128) + 43008, "flops": case["n"] * layers}
    steps = -(-case["n"] // case["minibatch"])
    return {"bytes": 48 * case["n"] + steps * 24 * NPARAMS, "flops": 3 * case["n"] * layers}


# ---- 64-bit values -----------------------------------------------------------------
def exact(case, seed):
    """trace: every ray against every triangle and sphere, where that is quick enough;
    ltc: the closed form; the network: its definition and Adam's.  A rendered frame has
    no such value: it is an estimate over its own random paths, and a path that 64 bits
    send past the other side of an edge is another path."""
    kind = case["kind"]
    if kind == "trace":
        if case["any"] or case["n"] * 20 * 4 ** case["subdiv"] > 2e10:
            return None
        return [None, _exact_trace(case, seed)]
    if kind == "ltc":
        return _exact_ltc(case, seed)
    if kind == "infer":
        centre, scale = _encoding()
        w = torch.from_numpy(_params(seed)).cuda().double()
        rec = _records(case["n"], seed)
        return torch.cat([torch.softmax(_logits(w, r, centre, scale), 1) for r in rec.split(1 << 16)])
    if kind == "train":
        return _exact_train(case, seed)
    return None


def _exact_trace(case, seed):
    tri = torch.from_numpy(_mesh(case, seed)).cuda().double().reshape(-1, 3, 3)
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    an = (a * nrm).sum(1)
    rays = _rays(case, seed).double()
    best = rays[:, 7].clone()
    step = max(1, int(4e7) // len(tri))
    for lo in range(0, len(rays), step):
        o, d = rays[lo:lo + step, 0:3], rays[lo:lo + step, 4:7]
        t = (an - o @ nrm.T) / (d @ nrm.T)
        # Barycentric coordinates (Moller and Trumbore 1997) with the products of ray and
        # triangle taken apart, so that they are matrix products.
        m = torch.linalg.cross(o, d)
        det = -(d @ nrm.T)
        ae1, ae2 = torch.linalg.cross(a, e1), torch.linalg.cross(a, e2)
        u = (m @ e2.T + d @ ae2.T) / det
        v = -(m @ e1.T + d @ ae1.T) / det
        eps = 1e-11
        ok = (u >= -eps) & (v >= -eps) & (u + v <= 1 + eps) & (t > rays[lo:lo + step, 3:4]) & (t < best[lo:lo + step, None])
        near = torch.where(ok, t, torch.full_like(t, math.inf)).amin(1)
        best[lo:lo + step] = torch.minimum(best[lo:lo + step], near)
    for c in torch.from_numpy(_spheres(case, seed)).double().cuda():
        op = c[:3] - rays[:, 0:3]
        b = (op * rays[:, 4:7]).sum(1)
        det = b * b - (op * op).sum(1) + c[3] * c[3]
        s = det.clamp_min(0).sqrt()
        for t in (b + s, b - s):
            best = torch.where((det >= 0) & (t > 1e-4) & (t < best), t, best)
    return best


def _edge(p, q):
    c = (p * q).sum(1).clamp(-1, 1)
    th = torch.acos(c)
    return torch.linalg.cross(p, q) * torch.where(c < 1 - 1e-15, th / torch.sin(th).clamp_min(1e-300), torch.ones_like(th))[:, None]


def _polygon(corners, n):
    """|sum of the edge integrals about n| of unit corners, each (N, 3)."""
    k = len(corners)
    s = sum(_edge(corners[i], corners[(i + 1) % k]) for i in range(k))
    return (s * n).sum(1).abs()


def _lobe(P, n):
    """|integral| about n of a triangle with corners P[0..2] relative to the point, cut at
    the horizon as the reference cuts it: of the three edges, those that cross give a
    segment each, in order; two are needed; on the edge CA corners of equal x do not cross."""
    E = [_unit(p) for p in P]
    h = [(p * n).sum(1) for p in P]
    up, down = (h[0] > 0) & (h[1] > 0) & (h[2] > 0), (h[0] < 0) & (h[1] < 0) & (h[2] < 0)
    full = _polygon(E, n)
    hits = torch.zeros_like(h[0], dtype=torch.int64)
    dead = torch.zeros_like(up)
    seg = [torch.zeros_like(P[0]) for _ in range(4)]
    for i in range(3):
        j = (i + 1) % 3
        dh = h[i] - h[j]
        flat = dh * dh <= 1e-15
        dead |= flat & (h[i] * h[i] < 1e-15)
        d = -h[i] / torch.where(flat, torch.ones_like(dh), dh)
        cross = ~flat & (d > -1) & (d < 0)
        if i == 2:
            cross &= P[0][:, 0] != P[2][:, 0]
        x = (P[i] - P[j]) * d[:, None] + P[i]
        first, second = torch.where((h[i] < 0)[:, None], x, P[i]), torch.where((h[i] < 0)[:, None], P[j], x)
        for slot in (0, 1):
            m = (cross & (hits == slot))[:, None]
            seg[2 * slot], seg[2 * slot + 1] = torch.where(m, first, seg[2 * slot]), torch.where(m, second, seg[2 * slot + 1])
        hits += cross
    cut = _polygon([p / p.norm(dim=1, keepdim=True).clamp_min(1e-300) for p in seg], n)
    cut = torch.where((hits > 1) & ~dead, cut, torch.zeros_like(cut))
    return torch.where(up, full, torch.where(down, torch.zeros_like(full), cut))


def _ltc_table():
    raw = (Path(ckr.PKG) / "data" / "ltc_ggx.bin").read_bytes()
    n = 64 * 64
    inv = np.frombuffer(raw, np.float64, 9 * n, 16 + 72 * n).reshape(n, 9)
    amp = np.frombuffer(raw, np.float32, n, 16 + 144 * n)
    # Rows hold the matrix's columns: slots 0, 2, 4, 6, 8 of the transpose.
    return torch.from_numpy(np.column_stack([inv[:, [0, 6, 4, 2, 8]], amp]).copy()).cuda()


def _exact_ltc(case, seed):
    tab = _ltc_table()
    gb, tri, rgb = (t.double() for t in _gbuffer(case, seed))
    out = []
    for g in gb.split(1 << 18):
        x, al, n, v, spec = g[:, 0:3], g[:, 3], g[:, 4:7], g[:, 8:11], g[:, 11]
        c = (n * v).sum(1)
        tf = torch.acos(c.clamp(-1, 1)) / (0.5 * 3.14159265359) * 64
        t0 = tf.floor().clamp(0, 63).long()
        t1 = (t0 + 1).clamp(max=63)
        a = (al.sqrt() * 64).floor().clamp(0, 63).long()
        f = torch.where(t0 == t1, torch.zeros_like(tf), tf - t0)[:, None]
        m = tab[a + t0 * 64] * (1 - f) + tab[a + t1 * 64] * f
        T1 = _unit(v - n * c[:, None])
        T2 = _unit(torch.linalg.cross(n, T1))
        rows = (m[:, 0:1] * T1 + m[:, 1:2] * n, m[:, 2:3] * T2, m[:, 3:4] * T1 + m[:, 4:5] * n)
        z = torch.zeros_like(n)
        z[:, 2] = 1
        acc_s, acc_d = torch.zeros_like(x), torch.zeros_like(x)
        for k in range(len(tri)):
            P = [tri[k, 3 * i:3 * i + 3] - x for i in range(3)]
            Q = [torch.stack([(r * p).sum(1) for r in rows], 1) for p in P]
            acc_s += _lobe(Q, z)[:, None] * rgb[k]
            acc_d += _lobe(P, n)[:, None] * rgb[k]
        out.append((acc_s * (m[:, 5] * spec)[:, None] + acc_d * (1 - spec)[:, None]) / (2 * 3.14159265359))
    return torch.cat(out)


def _encoding():
    """The position normalisation: the scene's box to [-1, 1] along its longest side."""
    tri = S.manylight_scene(S.manylight_spec(subdiv=2, width=16, height=9, **ROOM)).tri9.reshape(-1, 3).astype(np.float64)
    lo, hi = tri.min(0), tri.max(0)
    return torch.from_numpy((lo + hi) / 2).cuda(), 2.0 / float((hi - lo).max())


def _split(w):
    p, at = [], 0
    for shape in ((64, 96), (64, 64), (64,), (64, 64), (64,), (64, 64), (64,)):
        k = math.prod(shape)
        p.append(w[at:at + k].reshape(shape))
        at += k
    return p


def _logits(w, rec, centre, scale):
    W1, W2, b2, W3, b3, W4, b4 = _split(w)
    r = rec.double()
    p = (r[:, 0:3] - centre) * scale
    arg = p[:, :, None] * (math.pi * 2.0 ** torch.arange(12, device="cuda", dtype=torch.float64))
    wave = torch.stack([arg.sin(), arg.cos()], 3).reshape(len(r), 72)
    f = torch.cat([wave, r[:, 4:7], r[:, 8:11], r[:, 3:4], torch.ones_like(r[:, :1]), torch.zeros(len(r), 16, device="cuda", dtype=torch.float64)], 1)
    h = torch.relu(f @ W1.T)
    h = torch.relu(h @ W2.T + b2)
    h = torch.relu(h @ W3.T + b3)
    return h @ W4.T + b4


def _exact_train(case, seed):
    centre, scale = _encoding()
    w = torch.from_numpy(_params(seed)).cuda().double()
    rec = _records(case["n"], seed)
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    for k, r in enumerate(rec.split(case["minibatch"]), 1):
        p = w.clone().requires_grad_(True)
        logp = torch.log_softmax(_logits(p, r, centre, scale), 1)
        wt = r[:, 7].double()
        pick = logp.gather(1, r[:, 11].contiguous().view(torch.int32).long()[:, None])[:, 0]
        (-(wt * pick).sum() / wt.sum()).backward()
        g = p.grad
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        w = w - 1e-3 * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
    return w
