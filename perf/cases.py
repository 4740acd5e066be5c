"""Performance cases: the work that users of this framework have it do.

A case is a dict of plain values.  ``listed`` names the ones that are followed
from change to change, ``draw`` gives others of the same ranges, ``prepare``
makes what a program holds before its call (inputs from a seed, resident
scenes, fitted buffers, captured graphs), ``run`` is one pass through the
public entry points and returns every output, and ``work`` is what the pass
cannot do without.

Every output is a whole number or a record whose bytes the reference fixes
(certificates, pair keys, candidate records, feature rows, statistics), so two
versions of the framework agree byte for byte or one of them is wrong.  Two
things are left out of the returned values because no caller can rely on them:
the order of an undecided queue (its entries are the undecided certificates,
which are returned) and the number of speculative any-hit evaluations (it
depends on the device's timing).
"""
from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "p2c-ccd_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from p2cccd_b200 import certify, dense_groups, proxy, records, scenes, workloads  # noqa: E402
from p2cccd_b200.batch import BatchPipeline  # noqa: E402
from p2cccd_b200.scene import ScenePipeline  # noqa: E402
from p2cccd_b200.serve import Request, ServeEngine  # noqa: E402

DEVICE = "cuda:0"


def listed() -> list[dict]:
    return [
        # a handful of queries, as an interactive tool or a solver's inner loop asks: launch latency
        {"name": "certify_96", "kind": "certify", "n_vf": 64, "n_ee": 32, "eps_time": 1e-6, "t0": 0.0, "t1": 1.0},
        # the plain exact-CCD batch of the benchmark: 10k vertex-face and 10k edge-edge queries
        {"name": "certify_20k", "kind": "certify", "n_vf": 10000, "n_ee": 10000, "eps_time": 1e-6, "t0": 0.0,
         "t1": 1.0},
        # host-owned records in and certificates out, the reference's own batch call, default tolerances
        {"name": "host_ee_30k", "kind": "host", "family": 2, "n": 30011, "eps_time": 1e-4},
        # the smallest serving mesh, stepped in a frame loop from a captured graph
        {"name": "scene_10k", "kind": "scene", "shape": "spheres", "objects": 2, "lon": 56, "rings": 45,
         "narrow": "certify", "thickness": 0.0, "self": False, "graph": True},
        # the default benchmark scene: two spheres of 40,960 triangles, captured
        {"name": "scene_82k", "kind": "scene", "shape": "spheres", "objects": 2, "lon": 160, "rings": 128,
         "narrow": "certify", "thickness": 0.0, "self": False, "graph": True},
        # many bodies in one large scene, proposed and replayed per body pair, not captured
        {"name": "bodies_27x20k", "kind": "scene", "shape": "spheres", "objects": 27, "lon": 112, "rings": 91,
         "narrow": "anyhit", "thickness": 0.0, "self": False, "graph": False},
        # a mid-size cloth whose every candidate is certified, self-contact included
        {"name": "cloth_60k_self", "kind": "scene", "shape": "cloth", "n": 159, "lon": 71, "rings": 70,
         "narrow": "certify", "thickness": 0.0, "self": True, "graph": False},
        # the dense-contact stress: 512 x 512 cloth cells on a 100k-triangle sphere, self pairs, scheduled any-hit
        {"name": "cloth_624k", "kind": "scene", "shape": "cloth", "n": 513, "lon": 250, "rings": 200,
         "narrow": "anyhit", "thickness": 0.0, "self": True, "graph": False},
        # independent scenes of uneven size certified together in one captured step
        {"name": "batch_64", "kind": "batch", "scenes": 64, "tri_min": 1000, "tri_max": 200000, "graph": True},
        # proxy scene: build, candidates and the learned scheduler's feature rows
        {"name": "proxy_51k", "kind": "proxy", "bodies": 32, "patches": 200, "segments": 2, "slabs": 4},
        # candidate-group early stop over a million rows
        {"name": "groups_1m", "kind": "groups", "rows": 1000000, "max_group": 256, "preserve": False},
        # a burst of requests of mixed meshes through the continuous-batching server
        {"name": "serve_24", "kind": "serve", "requests": 24, "tri_min": 10000, "tri_max": 300000,
         "narrow": "anyhit"},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sphere_shape(triangles: float) -> tuple[int, int]:
    """Longitudes and rings of a UV sphere of about that many triangles."""
    rings = max(3, int(round(math.sqrt(triangles / 2.5))))
    return max(4, int(round(triangles / 2.0 / rings))), rings


def draw(rng) -> dict:
    kind = rng.choice(["certify", "certify", "host", "spheres", "spheres", "spheres", "cloth", "cloth", "batch",
                       "proxy", "groups", "serve"])
    if kind == "certify":
        t0, t1 = rng.choice([(0.0, 1.0), (0.0, 1.0), (0.25, 0.5), (0.1, 0.7)])
        n_vf, n_ee = _log(rng, 1, 100000), _log(rng, 1, 100000)
        if rng.random() < 0.3:  # one family alone
            n_vf, n_ee = rng.choice([(n_vf, 0), (0, n_ee)])
        return {"kind": "certify", "n_vf": n_vf, "n_ee": n_ee, "eps_time": rng.choice([1e-6, 1e-4]), "t0": t0,
                "t1": t1}
    if kind == "host":
        return {"kind": "host", "family": rng.choice([1, 2]), "n": _log(rng, 1, 100000),
                "eps_time": rng.choice([1e-6, 1e-4])}
    if kind in ("spheres", "cloth"):
        c = {"kind": "scene", "shape": kind, "narrow": rng.choice(["certify", "certify", "anyhit"]),
             "thickness": rng.choice([0.0, 0.0, 1e-4]), "graph": rng.random() < 0.5}
        if kind == "spheres":
            k = rng.choice([2, 2, 2, 5, 12, 27])
            lon, rings = _sphere_shape(_log(rng, max(1000, 200 * k), 500000) / k)
            own = rng.random() < 0.2 and lon * rings * k < 20000
            return {**c, "objects": k, "lon": lon, "rings": rings, "self": own}
        n = _log(rng, 20, 460)
        lon, rings = _sphere_shape(0.4 * (n - 1) ** 2 + 40)
        return {**c, "n": n, "lon": lon, "rings": rings, "self": rng.random() < 0.7}
    if kind == "batch":
        lo = _log(rng, 1000, 5000)
        return {"kind": "batch", "scenes": _log(rng, 3, 80), "tri_min": lo, "tri_max": lo * rng.randint(2, 25),
                "graph": rng.random() < 0.7}
    if kind == "proxy":
        return {"kind": "proxy", "bodies": rng.randint(3, 40), "patches": _log(rng, 10, 300),
                "segments": rng.randint(1, 3), "slabs": rng.randint(1, 5)}
    if kind == "groups":
        return {"kind": "groups", "rows": _log(rng, 200, 900000), "max_group": _log(rng, 4, 400),
                "preserve": rng.random() < 0.3}
    lo = _log(rng, 5000, 20000)
    return {"kind": "serve", "requests": rng.randint(2, 24), "tri_min": lo, "tri_max": lo * rng.randint(2, 12),
            "narrow": rng.choice(["anyhit", "certify"])}


# -- scenes -----------------------------------------------------------------


def _edges(faces: np.ndarray, nv: int) -> np.ndarray:
    """Unique undirected edges (min, max) in lexicographic order."""
    a, b = faces.astype(np.int64), np.roll(faces, -1, axis=1).astype(np.int64)
    key = np.unique((np.minimum(a, b) * nv + np.maximum(a, b)).ravel())
    return np.stack([key // nv, key % nv], 1).astype(np.int32)


@functools.lru_cache(maxsize=256)
def _sphere(lon: int, rings: int):
    v, f = scenes.uv_sphere(lon, rings)
    return v, f, _edges(f, len(v))


@functools.lru_cache(maxsize=16)
def _cloth_mesh(n: int):
    idx = np.arange(n * n).reshape(n, n)
    a, b, c, d = idx[:-1, :-1].ravel(), idx[:-1, 1:].ravel(), idx[1:, :-1].ravel(), idx[1:, 1:].ravel()
    f = np.concatenate([np.stack([a, b, c], 1), np.stack([b, d, c], 1)]).astype(np.int32)
    xs = np.linspace(-1.5, 1.5, n)
    x, y = np.meshgrid(xs, xs, indexing="xy")
    return x.ravel(), y.ravel(), f, _edges(f, n * n)


def _turn(g: np.random.Generator, most: float) -> np.ndarray:
    """A rotation by up to ``most`` radians about a random axis."""
    k = g.normal(size=3)
    k /= np.linalg.norm(k)
    w = g.uniform(0.0, most)
    c = np.array([[0.0, -k[2], k[1]], [k[2], 0.0, -k[0]], [-k[1], k[0], 0.0]])
    return np.eye(3) + np.sin(w) * c + (1.0 - np.cos(w)) * (c @ c)


def _spheres(k: int, lon: int, rings: int, seed: int, jitter: float = 1e-3) -> dict:
    """k unit spheres on a cubic lattice, 0.05 apart at t0, drawn together by
    0.1 per step, so that lattice neighbours meet at mid-step.  Each keeps its
    own orientation within 0.05 radians; the seed turns it and moves every vertex."""
    g, turns = workloads.rng(seed), workloads.rng(7)
    v, f, e = _sphere(lon, rings)
    side = math.ceil(k ** (1 / 3) - 1e-9)
    objs = []
    for i in range(k):
        at = np.array([i % side, i // side % side, i // side ** 2], float)
        w = v @ (_turn(turns, math.pi) @ _turn(g, 0.05)).T
        objs.append((w + 2.05 * at + g.normal(0.0, jitter, v.shape), w + 1.95 * at + g.normal(0.0, jitter, v.shape),
                     f, e))
    return scenes.combine(objs)


def _cloth(n: int, lon: int, rings: int, seed: int, gap: float = 1e-4, drop: float = 0.02,
           jitter: float = 1e-5) -> dict:
    """An n x n cloth sheet draping onto a unit sphere over the step."""
    g = workloads.rng(seed)
    x, y, f, e = _cloth_mesh(n)
    v, sf, se = _sphere(lon, rings)
    r2 = x ** 2 + y ** 2
    z0 = np.full_like(x, 1.0 + gap)
    z1 = np.where(r2 < 1.0, np.sqrt(np.clip(1.0 - r2, 0.0, None)) + gap * 0.5,
                  1.0 + gap - drop - 0.5 * (np.sqrt(r2) - 1.0))
    z1 = np.minimum(z1, z0 - drop * 0.25)
    j = lambda w: w + g.normal(0.0, jitter, w.shape)  # noqa: E731
    return scenes.combine([(j(np.stack([x, y, z0], -1)), j(np.stack([x, y, z1], -1)), f, e), (j(v), j(v), sf, se)])


def _scene(c: dict, seed: int) -> dict:
    if c["shape"] == "spheres":
        return _spheres(c["objects"], c["lon"], c["rings"], seed)
    return _cloth(c["n"], c["lon"], c["rings"], seed)


def _batch_sizes(c: dict) -> list[float]:
    """Triangles per scene, spread evenly over their logarithm, in mixed order."""
    n = c["scenes"]
    step = next(s for s in range(max(1, int(0.6 * n)), n + 1) if math.gcd(s, n) == 1)
    return [c["tri_min"] * (c["tri_max"] / c["tri_min"]) ** (((i * step) % n + 0.5) / n) for i in range(n)]


def _pool(c: dict) -> list[tuple[str, float]]:
    """The server's registered meshes: kinds and triangle counts."""
    r = c["tri_max"] / c["tri_min"]
    return [(("spheres", "spheres", "cloth")[i % 3], c["tri_min"] * r ** (i / 4)) for i in range(5)]


def _pool_scene(kind: str, tris: float, seed: int) -> dict:
    if kind == "spheres":
        return _spheres(2, *_sphere_shape(tris / 2), seed)
    return _cloth(int(round(math.sqrt(tris * 5 / 12))) + 1, *_sphere_shape(tris / 6), seed)


# -- the interface ------------------------------------------------------------


def _config(c: dict) -> certify.CertConfig:
    return certify.CertConfig(c.get("eps_time", 1e-6), 1e-6, 32)


def prepare(case: dict, seed: int) -> dict:
    c, kind = case, case["kind"]
    s = {"case": c, "config": _config(c)}
    if kind in ("certify", "host"):
        fam = {1: (c.get("n"), 1), 2: (1, c.get("n"))}.get(c.get("family"), (c.get("n_vf"), c.get("n_ee")))
        w = workloads.plain_queries(workloads.PlainSpec(n_vf=fam[0], n_ee=fam[1], seed=seed))
        if kind == "host":
            s["records"] = w["vf" if c["family"] == 1 else "ee"]
        else:
            s["vf"] = certify.records_to_device(w["vf"], DEVICE)
            s["ee"] = certify.records_to_device(w["ee"], DEVICE)
            s["ws"] = certify.Workspace(torch.device(DEVICE))
    elif kind in ("scene", "batch"):
        # the first frame (the same for every seed) sizes the pair buffers; the seed's frame comes after it
        if kind == "scene":
            first, sc = _scene(c, 0), _scene(c, seed)
            p = ScenePipeline(first, DEVICE, thickness=c["thickness"], exclude_self=not c["self"],
                              config=s["config"], narrow=c["narrow"])
            frames = sc["v_t0"], sc["v_t1"]
        else:
            first, sc = ([_spheres(2, *_sphere_shape(t / 2), k * 1000 + i) for i, t in enumerate(_batch_sizes(c))]
                         for k in (0, seed))
            p = BatchPipeline(first, DEVICE, config=s["config"])
            frames = np.zeros(p.v_off[-1]), np.zeros(p.v_off[-1])
            for i, one in enumerate(sc):
                for f, k in zip(frames, ("v_t0", "v_t1")):
                    f[p.v_off[i]:p.v_off[i] + one[k].size] = one[k].ravel()
        p.step_checked()
        p.fit_capacities(margin=1.4, slack=1024)
        s["frame"] = tuple(torch.from_numpy(f).to(DEVICE) for f in frames)
        p.update_positions(*s["frame"])
        p.step_checked()
        for t in (p.vf_pairs, p.ee_pairs, p.vf_results, p.ee_results):
            t.zero_()  # slots past the counts are never written
        s["pipe"] = p
        if c["graph"]:
            p.capture()
    elif kind == "proxy":
        spread = 2.0 * (c["bodies"] / 64.0) ** (1.0 / 3.0)  # constant body density
        inp = scenes.proxy_build_input(c["bodies"], c["patches"], c["segments"], c["slabs"], seed=5, spread=spread)
        first = proxy.ProxyCandidates(proxy.ProxySceneBuild(inp, DEVICE).run_checked(), DEVICE)
        hits = len(first.run_checked()[0])  # the bodies' motion sizes the buffers; the seed places their patches
        g = workloads.rng(seed)
        for o in inp["objects"]:
            n = len(o["patch_id"])
            at = g.normal(size=(n, 3))
            o["local_center"] = at / np.linalg.norm(at, axis=1, keepdims=True) * np.linalg.norm(o["local_center"][0])
            o["radius"] = g.uniform(0.02, 0.08, n)
        b = proxy.ProxySceneBuild(inp, DEVICE)
        k = proxy.ProxyCandidates(b.run_checked(), DEVICE, raw_capacity=int(1.4 * hits) + 4096)
        k.run_checked()
        k.run()
        k.feature_rows_async()
        for t in (k.raw, k.cand, k.rows):
            t.zero_()
        s["build"], s["candidates"] = b, k
    elif kind == "groups":
        rows = workloads.dense_group_rows(c["rows"], seed=seed, max_group=c["max_group"])
        s["rows"] = dense_groups.upload(dense_groups.parse_arrays(rows, rows), DEVICE)
        s["bits"] = max(1, int(rows["query_id"].max()).bit_length())
        s["runner"] = dense_groups.DenseGroupEarlyStop(c["rows"], DEVICE)
    else:
        e = ServeEngine(DEVICE, config=s["config"], narrow=c["narrow"], memory_budget=6 << 30)
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory()  # noqa: E731
        frames = []
        for i, (shape, tris) in enumerate(_pool(c)):
            sc = _pool_scene(shape, tris, seed + 1000 * i)
            e.register_mesh(str(i), sc, exclude_self=shape != "cloth")
            frames.append((pin(sc["v_t0"]), pin(sc["v_t1"])))
        s["server"] = e
        # smaller meshes ask more often than larger ones
        order = [(0, 1, 0, 2, 1, 3, 0, 4)[i % 8] for i in range(c["requests"])]
        s["asks"] = [(str(m), *frames[m], seed * 64 + i) for i, m in enumerate(order)]
        e.run(_requests(s))  # every mesh's candidate state is resident before serving counts
    return s


def _requests(s: dict) -> list[Request]:
    return [Request(rid=i, mesh=m, v_t0=a, v_t1=b, arrival_s=0.0, seed=k,
                    keep_results=s["case"]["narrow"] == "anyhit") for i, (m, a, b, k) in enumerate(s["asks"])]


def run(state: dict):
    s, c, kind = state, state["case"], state["case"]["kind"]
    if kind == "certify":
        if c["n_vf"] and c["n_ee"]:
            return certify.certify_batch2(s["vf"], s["ee"], c["t0"], c["t1"], s["config"], workspace=s["ws"])
        recs, fam = (s["vf"], records.FAMILY_POINT_TRIANGLE) if c["n_vf"] else (s["ee"], records.FAMILY_EDGE_EDGE)
        return certify.certify_batch(recs, fam, c["t0"], c["t1"], s["config"], workspace=s["ws"])
    if kind == "host":
        out = certify.certify_batch_host(s["records"], 0.0, 1.0, s["config"])
        return out.view(np.uint8).reshape(-1, 72)
    if kind in ("scene", "batch"):
        p = s["pipe"]
        p.update_positions(*s["frame"])
        p.replay() if c["graph"] else p.step()
        if kind == "batch":
            return [p.counts[:, :3], p.vf_pairs, p.ee_pairs, p.vf_results, p.ee_results, p.summaries]
        out = [p.counts[:3], p.vf_pairs, p.ee_pairs]
        if c["narrow"] == "certify":
            return out + [p.vf_results, p.ee_results, p.summary]
        for a in (p.anyhit_vf, p.anyhit_ee):
            word = a.summary.view(torch.int64)
            out += [a.evaluated, a.hit, a.group_detected, a.group_proposal_calls, a.group_fallback_calls, word[:7],
                    word[8:]]
        return out
    if kind == "proxy":
        s["build"].run()
        k = s["candidates"]
        k.run()
        density, rows, error = k.feature_rows_async()
        return [[t.view(torch.uint8) for t in s["build"].out.values()], k.counts[:3], k.raw, k.cand, density, rows,
                error]
    if kind == "groups":
        s["runner"].run(s["rows"], c["rows"], preserve=c["preserve"], query_bits=s["bits"])
        return s["runner"].stats
    out = []
    for r in sorted(s["server"].run(_requests(s)), key=lambda r: r.rid):
        if c["narrow"] == "anyhit":
            flat = [v for f in ("vf", "ee") for k, v in r.anyhit[f].items() if k != "speculative"]
            out.append(np.concatenate([[r.queries], flat, *r.groups]).astype(np.int64))
        else:
            q = r.summary["query"]
            flat = [v for k, v in r.summary.items() if k != "query"]
            out.append(np.array([r.queries, *flat, q["status"], q["witness_index"],
                                 np.float64(q["toi_upper"]).view(np.int64)], np.int64))
    return np.stack(out)


def exact(case: dict, seed: int):
    """No output is a computed number with a tolerance: all are compared as
    whole numbers and record bytes."""
    return None


# FP64 operations of one certificate that separates at its root: three
# distance samples of about 130 operations, four motion norms, one radius.
_CERT_FLOPS = 3 * 130 + 36 + 10


def _scene_work(shape: str, tris: float, objects: int, own: bool, certificates: bool) -> tuple[float, float]:
    """Bytes and operations of one scene step: vertices of both frames,
    faces and edges read, pairs written (and their certificates).  Closed
    meshes and sheets have about 1/2 vertex and 3/2 edges per triangle;
    candidates per triangle are those of the contact patches the generators
    make (a sphere pair's share falls with the mesh's resolution)."""
    verts, edges = 0.5 * tris, 1.5 * tris
    if shape == "spheres":
        contacts = max(1, 3 * (objects - round(objects ** (2 / 3))))
        pairs = contacts * 0.05 * tris / objects * 2
    else:
        pairs = 5.0 * tris
    if own:
        pairs += (5.0 if shape == "cloth" else 20.0) * tris
    size = 48 * verts + 12 * tris + 8 * edges + 8 * pairs + (72 if certificates else 1) * pairs
    return size, pairs * _CERT_FLOPS


def work(case: dict) -> dict:
    c, kind = case, case["kind"]
    if kind in ("certify", "host"):
        n = c["n"] if kind == "host" else c["n_vf"] + c["n_ee"]
        return {"bytes": (240 + 72) * n, "flops": _CERT_FLOPS * n}
    if kind == "scene":
        sphere = 2 * c["lon"] * c["rings"]
        k = c.get("objects", 2)
        tris = k * sphere if c["shape"] == "spheres" else sphere + 2 * (c["n"] - 1) ** 2
        b, f = _scene_work(c["shape"], tris, k, c["self"], c["narrow"] == "certify")
    elif kind == "batch":
        parts = [_scene_work("spheres", t, 2, False, True) for t in _batch_sizes(c)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "proxy":
        n = c["bodies"] * c["patches"] * c["segments"] * c["slabs"]
        hits = 2.2 * n
        b, f = n * (36 + 185) + hits * (64 + 80 + 256), n * 200.0 + hits * 60
    elif kind == "groups":
        b, f = c["rows"] * (8 + 8 + 4 + 64 + 32 + 12) + 200, c["rows"] * 30.0
    else:
        pool = _pool(c)
        b = f = 0.0
        for i in range(c["requests"]):
            shape, t = pool[(0, 1, 0, 2, 1, 3, 0, 4)[i % 8]]
            x, y = _scene_work(shape, t, 2, shape == "cloth", c["narrow"] == "certify")
            b, f = b + x, f + y
    return {"bytes": b, "flops": f}
