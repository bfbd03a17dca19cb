"""The work that users of the engine have it do, as cases to be timed and compared.

A case is one pass of a user's program through the public entry points: a tick of a resident
layout (Engine.enqueue), a frame of an interactive one (upload, tick, readback), a tick of the
simulation object, a tick of a batch of graphs, or a sort in the caller's own device memory.
Sizes are those of the engine's own configurations (1,000 to 4,000,000 nodes, graphs of 100 to
20,000 nodes in a batch) and of the odd and ragged layouts in between.

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  what the program has in hand before a pass
  run(state)           one pass, and its outputs
  work(case)           the bytes and operations a pass cannot do without
  exact(case, seed)    the first pass's outputs in 64 bits, by plain torch
"""
import asyncio
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "d3-force-3d-webgpu_gb300"))

from forcegpu import (Engine, forceCenter, forceCollide, forceLink, forceManyBody,  # noqa: E402
                      forceSimulationGPU)
from forcegpu._lib import SORT_NOALLOC_MAX_PAIRS, desc_from_gpu, radix_sort_noalloc  # noqa: E402
from forcegpu.batch import Batch, GraphSpec  # noqa: E402
from forcegpu.graphs import link_defaults, phyllotaxis  # noqa: E402

ALPHA_DECAY = 1 - 0.001 ** (1 / 300)  # d3's default schedule
ALPHA = 0.1        # a layout that has cooled from 1, or one reheated by a drag
KEEP = 0.6         # 1 - velocityDecay, d3's default
MAX_NODES = 4_000_000


def layout(name, kind, n, ndim, **options):
    """A single layout's case. Options: theta (None: no charge), mixed (charges of both signs),
    dmax (distanceMax, None: no limit), links (per node), collide (iterations), center, radial,
    xy (forceX and forceY), pins (every 10th node fixed)."""
    case = {"kind": kind, "n": n, "ndim": ndim, "theta": 0.9, "mixed": False, "dmax": None,
            "links": 1.5, "collide": 0, "center": True, "radial": False, "xy": False, "pins": False}
    case.update(options)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the small layout of an ordinary web page, resident: launches and latency count
        layout("tick_1k_3d", "tick", 1000, 3),
        # the same size through the simulation object, the drop-in API: nodes as Python dicts
        layout("sim_1k_3d", "sim", 1000, 3),
        # a 2D graph drawn with collision by pairs and forceX / forceY in place of the centre
        layout("tick_5k_2d_collide", "tick", 5003, 2, collide=1, center=False, xy=True),
        # one frame of an interactive layout: positions up, a tick, positions and velocities back
        layout("frame_20k_3d", "frame", 20_000, 3),
        # the exact sum over all pairs (theta 0), as used to check accuracy
        layout("exact_20k_3d", "tick", 20_000, 3, theta=0.0),
        # every force at once: link, charge, grid collide, radial, centre, and pinned nodes
        layout("tick_100k_3d_full", "tick", 100_000, 3, collide=1, radial=True, pins=True),
        # a served 2D job at the top of its size range: dense links and collision
        layout("tick_200k_2d_collide", "tick", 200_003, 2, links=3.0, collide=1),
        # charges of both signs and a cut-off distance, an odd size
        layout("tick_300k_3d_mixed", "tick", 300_007, 3, mixed=True, dmax=400.0),
        # the headline layout
        layout("tick_1m_3d", "tick", 1_000_000, 3),
        # the largest layout: 1.2 GB of state and tree
        layout("tick_4m_3d", "tick", MAX_NODES, 3),
        # many uneven graphs advanced together, the state read back for their owners
        {"name": "batch_256_3d", "kind": "batch", "graphs": 256, "smallest": 100, "largest": 20_000,
         "ndim": 3, "collide": 0},
        # the key sort in a caller's own device memory, at the largest size it takes
        {"name": "sort_262k", "kind": "sort", "n": SORT_NOALLOC_MAX_PAIRS, "lo_bit": 0},
    ]


def limit(case):
    return math.inf if case["dmax"] is None else case["dmax"]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tick"] * 8 + ["frame"] * 2 + ["batch"] * 2 + ["sim", "exact", "sort"])
    if kind == "sort":
        return {"kind": "sort", "n": log_uniform(rng, 1000, SORT_NOALLOC_MAX_PAIRS),
                "lo_bit": rng.choice([0, 1, 16, 33])}
    if kind == "batch":
        return {"kind": "batch", "graphs": log_uniform(rng, 8, 256), "smallest": 100,
                "largest": log_uniform(rng, 2000, 20_000), "ndim": rng.choice([2, 3]),
                "collide": rng.choice([0, 0, 1])}
    ndim = rng.choice([2, 3, 3])
    if kind == "sim":
        return layout(None, "sim", log_uniform(rng, 300, 1500), ndim, collide=rng.choice([0, 1]))
    if kind == "exact":
        return layout(None, "tick", log_uniform(rng, 1000, 20_000), ndim, theta=0.0)
    n = log_uniform(rng, 1000, 1_500_000 if kind == "tick" else 1_000_000)
    collide = rng.choice([0, 0, 1, 1, 2])
    center = rng.choice([True, True, False])
    return layout(None, kind, n, ndim, theta=rng.choice([0.9, 0.9, 0.9, 0.7, 0.5]),
                  mixed=rng.choice([False, False, True]), dmax=rng.choice([None, None, 300.0]),
                  links=rng.choice([1.0, 1.5, 1.5, 2.0, 3.0]), collide=collide, center=center,
                  radial=rng.choice([False, False, True]), xy=not center,
                  pins=rng.choice([False, False, True]))


# ---------------------------------------------------------------- inputs

def graph(n, ndim, per_node, rng):
    """Start positions (a layout a little way from d3's phyllotaxis start) and links (a random
    tree and random pairs, the reference benchmark's shape)."""
    xyz = np.zeros((n, 4), np.float32)
    xyz[:, :ndim] = phyllotaxis(n, ndim)[:, :ndim] + rng.normal(0.0, 4.0, (n, ndim))
    tree = np.arange(1, n)
    src = np.concatenate([tree, rng.integers(0, n, int(n * (per_node - 1)))]).astype(np.int32)
    dst = np.concatenate([(rng.random(n - 1) * tree).astype(np.int64),
                          rng.integers(0, n, len(src) - (n - 1))]).astype(np.int32)
    keep = src != dst
    return xyz, src[keep], dst[keep]


def inputs(case, seed):
    """The arrays of a layout: what its program has loaded or computed itself."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    xyz, src, dst = graph(n, case["ndim"], case["links"], rng)
    bias, strength = link_defaults(n, src, dst)
    charge = np.full(n, -30.0, np.float32)
    if case["mixed"]:
        charge[::4] = 20.0
    radii = rng.uniform(1, 5, n).astype(np.float32)
    mask = np.zeros(n, np.uint32)
    if case["pins"]:
        mask[::10] = (1 << case["ndim"]) - 1
    return {"xyz": xyz, "src": src, "dst": dst, "bias": bias.astype(np.float32),
            "strength": strength.astype(np.float32), "charge": charge, "radii": radii, "mask": mask}


def forces(case, a):
    """The layout's forces as the engine's descriptors, in application order."""
    n = case["n"]
    out = [{"type": "link", "version": 1, "source": a["src"], "target": a["dst"], "iterations": 1,
            "strengths": a["strength"], "distances": np.full(len(a["src"]), 30.0), "bias": a["bias"]}]
    out.append({"type": "manyBody", "version": 1, "strengths": a["charge"], "distanceMin2": 1.0,
                "distanceMax2": limit(case) ** 2, "theta2": case["theta"] ** 2})
    if case["collide"]:
        out.append({"type": "collide", "version": 1, "radii": a["radii"], "strength": 1.0,
                    "iterations": case["collide"]})
    if case["radial"]:
        out.append({"type": "radial", "version": 1, "radiuses": np.full(n, 200.0),
                    "strengths": np.full(n, 0.05), "x": 0.0, "y": 0.0, "z": 0.0})
    if case["xy"]:
        for axis in (0, 1):
            out.append({"type": "position", "version": 1, "axis": axis, "targets": np.zeros(n),
                        "strengths": np.full(n, 0.1)})
    if case["center"]:
        out.append({"type": "center", "version": 0, "x": 0.0, "y": 0.0, "z": 0.0, "strength": 1.0})
    return out


def batch_specs(case, seed):
    """Graphs of uneven sizes (the case's own), log-uniform between the smallest and the largest."""
    spread = np.random.default_rng(case["graphs"]).uniform(size=case["graphs"])
    sizes = (case["smallest"] * (case["largest"] / case["smallest"]) ** spread).astype(int)
    rng = np.random.default_rng(seed)
    specs = []
    for n in sizes:
        xyz, src, dst = graph(int(n), case["ndim"], 1.5, rng)
        radii = rng.uniform(1, 5, n).astype(np.float32) if case["collide"] else None
        specs.append(GraphSpec(xyz=xyz[:, :case["ndim"]], source=src, target=dst, alpha=ALPHA,
                               radii=radii, collide_iterations=max(1, case["collide"])))
    return specs


def sort_pairs(case, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(0, 1 << 63, case["n"], dtype=np.int64), np.arange(case["n"], dtype=np.int32)


class DeviceArray:
    """n float4 records of `owner` at a device address, for torch.as_tensor (whose tensor keeps
    this object, and so the owner, alive)."""

    def __init__(self, owner, address, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n, 4), "typestr": "<f4", "data": (address, False),
                                         "version": 2}


def pinned(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True).numpy()


# ---------------------------------------------------------------- passes

def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        keys, vals = sort_pairs(case, seed)
        keys, vals = torch.from_numpy(keys).cuda(), torch.from_numpy(vals).cuda()
        return {"kind": kind, "n": case["n"], "lo_bit": case["lo_bit"], "keys": keys, "vals": vals,
                "keys_out": torch.empty_like(keys), "vals_out": torch.empty_like(vals)}
    if kind == "batch":
        batch = Batch()
        batch.set_graphs(batch_specs(case, seed), ndim=case["ndim"], seed=12345)
        n = int(batch.sizes.sum())
        return {"kind": kind, "batch": batch, "pos": pinned((n, 4)), "vel": pinned((n, 4))}
    a = inputs(case, seed)
    n, ndim = case["n"], case["ndim"]
    if kind == "sim":
        axes = "xyz"[:ndim]
        nodes = [dict(zip(axes, map(float, p))) for p in a["xyz"]]
        sim = forceSimulationGPU(nodes, ndim).stop()
        sim.force("link", forceLink([{"source": int(s), "target": int(t)}
                                     for s, t in zip(a["src"], a["dst"])]))
        sim.force("charge", forceManyBody())
        if case["collide"]:
            radii = a["radii"]
            sim.force("collide", forceCollide(lambda d, i, all_nodes: float(radii[i])))
        sim.force("center", forceCenter()).alpha(ALPHA)
        return {"kind": kind, "sim": sim, "nodes": nodes, "axes": axes}
    engine = Engine()
    engine.set_nodes(a["xyz"], ndim, fix4=a["xyz"], mask=a["mask"])
    engine.set_forces([desc_from_gpu(g, k + 1, n) for k, g in enumerate(forces(case, a))])
    engine.set_seed(12345)
    state = {"kind": kind, "engine": engine, "n": n, "alpha": ALPHA, "views": {}}
    if kind == "frame":
        state.update(up=pinned((n, ndim)), pos=pinned((n, ndim)), vel=pinned((n, ndim)))
        state["up"][:] = a["xyz"][:, :ndim]
    return state


def next_alpha(state):
    state["alpha"] += (0.0 - state["alpha"]) * ALPHA_DECAY
    return state["alpha"]


def view(state, address):
    """The device records at `address` as a tensor (made once per buffer, as a renderer maps it)."""
    if address not in state["views"]:
        state["views"][address] = torch.as_tensor(
            DeviceArray(state["engine"], address, state["n"]), device="cuda")
    return state["views"][address]


def run(state):
    kind = state["kind"]
    if kind == "sort":
        radix_sort_noalloc(state["keys"].data_ptr(), state["vals"].data_ptr(), state["n"],
                           state["lo_bit"], state["keys_out"].data_ptr(),
                           state["vals_out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"keys": state["keys_out"], "vals": state["vals_out"]}
    if kind == "batch":
        batch = state["batch"].run(1)
        batch._check(batch.L.fl_batch_sync(batch.h, state["pos"].ctypes.data, state["vel"].ctypes.data))
        return {"pos": state["pos"], "vel": state["vel"]}
    if kind == "sim":
        asyncio.run(state["sim"].tickAsync(1))
        axes, nodes = state["axes"], state["nodes"]
        return {"pos": np.array([[d[k] for k in axes] for d in nodes], np.float32),
                "vel": np.array([[d["v" + k] for k in axes] for d in nodes], np.float32)}
    engine = state["engine"]
    if kind == "frame":
        engine.update_positions_packed_async(0, state["up"])
        engine.enqueue([next_alpha(state)], KEEP)
        engine.sync_packed(state["pos"], state["vel"])
        return {"pos": state["pos"], "vel": state["vel"]}
    engine.enqueue([next_alpha(state)], KEEP)
    at = engine.buffers()
    return {"pos": view(state, at["positions"]), "vel": view(state, at["velocities"])}


def layout_work(n, ndim, theta, links, collide):
    """State read and written (positions and velocities, 16 bytes a record), pins and charges
    read, each link read once (both ends, distance, strength, bias); a point's interactions grow
    with log n and with the solid angle that theta leaves (or are all n), 20 operations each."""
    size = n * (64 + 8) + n * links * 20 + (4 * n if collide else 0)
    per = n if theta == 0 else min(n, (7 if ndim == 2 else 16) * math.log2(n) * (0.9 / theta) ** ndim)
    return {"bytes": size, "flops": n * (20 * per + 30 * links + 40)}


def work(case):
    if case["kind"] == "sort":
        return {"bytes": 24 * case["n"], "flops": 0}
    if case["kind"] == "batch":
        lo, hi = case["smallest"], case["largest"]
        mean = (hi - lo) / math.log(hi / lo)
        one = layout_work(mean, case["ndim"], 0.9, 1.5, case["collide"])
        return {k: v * case["graphs"] for k, v in one.items()}
    return layout_work(case["n"], case["ndim"], case["theta"], case["links"], case["collide"])


# ---------------------------------------------------------------- the same in 64 bits

class Tick64:
    """One tick of d3's forces on the GPU in float64: link and collide against one snapshot, the
    Barnes-Hut sum over d3's tree (or over all pairs), radial, x / y, centre, integration."""

    def __init__(self, xyz, ndim, alpha):
        self.p = torch.tensor(xyz[:, :ndim], dtype=torch.float64, device="cuda")
        self.v = torch.zeros_like(self.p)
        self.ndim, self.alpha = ndim, alpha

    def link(self, src, dst, distance, strength, bias):
        s, t, distance, strength, bias = (torch.as_tensor(np.asarray(x), device="cuda")
                                          for x in (src, dst, distance, strength, bias))
        s, t = s.long(), t.long()
        at = self.p + self.v
        d = at[t] - at[s]
        length = d.norm(dim=1)
        push = d * ((length - distance) / length * self.alpha * strength)[:, None]
        self.v.index_add_(0, t, -push * bias.double()[:, None])
        self.v.index_add_(0, s, push * (1 - bias.double())[:, None])

    def charge(self, strength, theta, dmax, dmin=1.0):
        strength = torch.as_tensor(strength, device="cuda").double()
        self.dmin2, self.dmax2 = dmin * dmin, dmax * dmax
        if theta == 0:
            self._pairs(strength)
        else:
            self._tree(strength, theta * theta)

    def _weight(self, d, value):
        l = (d * d).sum(-1)
        near = l < self.dmin2
        w = value * self.alpha / torch.where(near, (self.dmin2 * l).sqrt(), l)
        return torch.where((l < self.dmax2) & (l > 0), w, torch.zeros_like(w)), l

    def _pairs(self, strength):
        for a in range(0, len(self.p), 1024):
            d = self.p[None] - self.p[a:a + 1024, None]
            w, _ = self._weight(d, strength[None].expand(d.shape[:2]))
            self.v[a:a + 1024] += (d * w[..., None]).sum(1)

    def _tree(self, strength, theta2):
        n, nd, p = len(self.p), self.ndim, self.p
        levels = 21 if nd == 3 else 24
        origin, size = p.min(0).values.floor(), 1.0
        while not bool((p.max(0).values < origin + size).all()):
            size *= 2
        cell = ((p - origin) * (2.0 ** levels / size)).floor().long()
        key = torch.zeros(n, dtype=torch.long, device="cuda")
        for b in range(levels):
            for k in range(nd):
                key |= ((cell[:, k] >> b) & 1) << (b * nd + k)
        key, order = key.sort()
        c = math.sqrt(4 / 2 ** nd)
        # the occupied cells of every level, deepest first: points, value, centroid, children
        value, center = strength[order], p[order]
        count = torch.ones(n, dtype=torch.long, device="cuda")
        tree = [{"value": value, "center": center, "count": count, "first": None, "kids": None}]
        prefix = key
        for depth in range(levels, -1, -1):
            prefix = key if depth == levels else prefix >> nd
            prefix, inverse, kids = torch.unique_consecutive(prefix, return_inverse=True, return_counts=True)
            m = len(prefix)
            zeros = torch.zeros(m, dtype=torch.float64, device="cuda")
            below, weight = tree[-1], tree[-1]["value"].abs()
            total = zeros.clone().index_add_(0, inverse, below["value"])
            mass = zeros.clone().index_add_(0, inverse, weight)
            moment = torch.zeros(m, nd, dtype=torch.float64, device="cuda")
            moment.index_add_(0, inverse, weight[:, None] * below["center"])
            points = torch.zeros(m, dtype=torch.long, device="cuda").index_add_(0, inverse, below["count"])
            first = kids.cumsum(0) - kids
            alone = points == 1
            tree.append({"value": torch.where(alone, total, c * total), "count": points, "kids": kids,
                         "center": torch.where(alone[:, None], below["center"][first],
                                               moment / mass.clamp_min(1e-300)[:, None]),
                         "first": first})
        tree.reverse()
        chunk = 1 << 17
        sums = torch.zeros_like(p)
        for a in range(0, n, chunk):
            who = torch.arange(a, min(n, a + chunk), device="cuda")
            at = torch.zeros_like(who)
            for depth, level in enumerate(tree):
                val = level["value"][at]
                d = level["center"][at] - p[order[who]]
                w, l = self._weight(d, val)
                single = level["count"][at] == 1
                is_open = ~single & (val != 0) & ((size / 2.0 ** depth) ** 2 / theta2 >= l)
                w = torch.where(is_open, torch.zeros_like(w), w)
                sums.index_add_(0, who, d * w[:, None])
                if depth == len(tree) - 1:
                    break
                kids = level["kids"][at[is_open]]
                begin = level["first"][at[is_open]]
                who = who[is_open].repeat_interleave(kids)
                step = torch.arange(len(who), device="cuda") - (kids.cumsum(0) - kids).repeat_interleave(kids)
                at = begin.repeat_interleave(kids) + step
        self.v[order] += sums

    def collide(self, radii):
        r = torch.as_tensor(radii, device="cuda").double()
        at = self.p + self.v
        cell = (at / (2 * r.max())).floor().long()
        cell = cell - cell.min(0).values + 1
        spans = cell.max(0).values + 2

        def index(x):
            k = x[:, 0]
            for j in range(1, self.ndim):
                k = k * spans[j] + x[:, j]
            return k

        key, order = index(cell).sort()
        push = torch.zeros_like(at)
        for offset in np.ndindex(*(3,) * self.ndim):
            near = index(cell + torch.tensor(offset, device="cuda") - 1)
            lo, hi = torch.searchsorted(key, near), torch.searchsorted(key, near, right=True)
            i = torch.arange(len(at), device="cuda").repeat_interleave(hi - lo)
            skip = ((hi - lo).cumsum(0) - (hi - lo)).repeat_interleave(hi - lo)
            j = order[lo.repeat_interleave(hi - lo) + torch.arange(len(i), device="cuda") - skip]
            d, reach = at[i] - at[j], r[i] + r[j]
            length = d.norm(dim=1)
            hit = (length < reach) & (i != j)
            i, j, d, length, reach = i[hit], j[hit], d[hit], length[hit], reach[hit]
            share = r[j] ** 2 / (r[i] ** 2 + r[j] ** 2)
            push.index_add_(0, i, d * ((reach - length) / length * share)[:, None])
        self.v += push

    def radial(self, radius, strength):
        d = torch.full((len(self.p), 3), 1e-6, dtype=torch.float64, device="cuda")
        d[:, :self.ndim] = torch.where(self.p == 0, torch.full_like(self.p, 1e-6), self.p)
        r = d.norm(dim=1, keepdim=True)
        self.v += d[:, :self.ndim] * ((radius - r) * strength * self.alpha / r)

    def toward_axes(self, strength):
        self.v[:, :2] -= self.p[:, :2] * (strength * self.alpha)

    def outputs(self, center, mask=None, width=None):
        fixed = self.p.clone()
        if center:
            self.p -= self.p.mean(0)
        self.v *= KEEP
        self.p += self.v
        if mask is not None:
            pin = torch.as_tensor(mask.astype(np.int64), device="cuda")
            for k in range(self.ndim):
                held = (pin >> k) & 1 == 1
                self.p[held, k], self.v[held, k] = fixed[held, k], 0.0
        pad = (0, (width or self.ndim) - self.ndim)
        return {"pos": torch.nn.functional.pad(self.p, pad), "vel": torch.nn.functional.pad(self.v, pad)}


def exact(case, seed):
    kind, ndim = case["kind"], case["ndim"] if "ndim" in case else 0
    alpha = ALPHA - ALPHA * ALPHA_DECAY
    if kind == "sort":
        return None  # whole numbers
    if kind == "batch":
        parts = []
        for s in batch_specs(case, seed):
            n = len(s.xyz)
            bias, strength = link_defaults(n, s.source, s.target)
            t = Tick64(s.xyz, ndim, alpha)
            t.link(s.source, s.target, np.full(len(s.source), 30.0), strength, bias)
            t.charge(np.full(n, -30.0), 0.9, math.inf)
            if case["collide"]:
                for _ in range(case["collide"]):
                    t.collide(s.radii)
            parts.append(t.outputs(True, width=4))
        return {k: torch.cat([x[k] for x in parts]) for k in ("pos", "vel")}
    a = inputs(case, seed)
    t = Tick64(a["xyz"], ndim, alpha)
    t.link(a["src"], a["dst"], np.full(len(a["src"]), 30.0), a["strength"], a["bias"])
    t.charge(a["charge"], case["theta"], limit(case))
    for _ in range(case["collide"]):
        t.collide(a["radii"])
    if case["radial"]:
        t.radial(200.0, 0.05)
    if case["xy"]:
        t.toward_axes(0.1)
    return t.outputs(case["center"], a["mask"], 4 if kind == "tick" else ndim)
