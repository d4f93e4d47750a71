"""Performance cases of the derivation engine: what a program that uses it has it do.

Five kinds of call, over the sizes of this repository's scenes, tests and benchmark:

* "scene"    derive a batch of axioms into instanced terminals (Engine.execute), optionally with the LBVH over them
             (Engine.lbvh).  The emission order of a derivation is free, so the instances are handed on in an order of
             their own: by derivation path, or in the leaf order of the LBVH.
* "placing"  the two-phase scene of Collider / IfCollides: trees placed among buildings and billboards.
* "fit"      one gradient evaluation of the facade fit: autograd.derive_transforms, PathTarget.sse, backward.
* "step"     the differentiable step: derivation with the tape, LBVH over the device-side count, adjoint of
             L = |M|^2 / 2 read from the terminal records in place; captured in a CUDA graph or called directly.
* "records"  the LBVH over instance records that the program holds already (imported, or derived earlier), in any order.

Triangle meshes (pga_generate_meshes) are left out: the order of a mesh's faces is free and has no cheap canonical form.

Every kind takes its inputs from the seed alone.  exact() derives the terminals (and, by automatic differentiation, the
gradients) in 64 bits with plain torch from the dispatch table, and the boxes of a record set's LBVH.  The number of
terminals of a case is the same for every seed.
"""
import math

import numpy as np
import torch

from operatorgraph_gb300 import autograd, scenes
from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300.engine import Engine

DEVICE = "cuda"
SPONGE_THRESHOLDS = {1: 0.5, 2: 0.15, 3: 0.05, 4: 0.015, 5: 0.005}
MIXED_TERMINALS = 2330  # per axiom of the mixed batch, on average
TREE_TERMINALS = 3281
BUILDING_TERMINALS = 1430
FACADE_TERMINALS = 384


def listed():
    return [
        # One lot edited in a modelling tool: the smallest call, launch and level latency.
        {"name": "building", "kind": "scene", "scene": "city", "n": 1, "order": "path"},
        # The reference's own demo scene, one axiom, nine narrow levels, then its tree.
        {"name": "sponge_d3", "kind": "scene", "scene": "sponge", "n": 1, "depth": 3, "order": "leaf"},
        # A quarter of a city, streamed in as the camera moves.
        {"name": "city_61", "kind": "scene", "scene": "city", "n": 61, "order": "leaf"},
        # The headline city and the hierarchy over its instances.
        {"name": "city_4096", "kind": "scene", "scene": "city", "n": 4096, "order": "leaf"},
        # Trees with turned branches: the general-frame kernels.
        {"name": "forest_509", "kind": "scene", "scene": "forest", "n": 509, "order": "leaf"},
        # Vegetation placed around buildings: two phases with the colliders' tree between them.
        {"name": "placing_16384", "kind": "placing", "buildings": 1024, "trees": 16384, "boards": 1024},
        # The facade fit through torch.autograd, one optimiser step's gradients.
        {"name": "fit_250", "kind": "fit", "n": 250},
        # The benchmark's facades as a differentiable step, replayed as one graph.
        {"name": "facades_1024", "kind": "step", "scene": "facades", "n": 1024, "graph": True},
        # The mixed batch (sponges, buildings, random grammars), gradients to the axiom sizes.
        {"name": "mixed_1500", "kind": "step", "scene": "mixed", "n": 1500, "graph": False},
        # The large one: the mixed batch with parameter blocks, gradients to every parameter and size.
        {"name": "mixed_blocks_8192", "kind": "step", "scene": "mixed_blocks", "n": 8192, "graph": True},
        # A hierarchy over a small set of imported instances.
        {"name": "records_20011", "kind": "records", "n": 20011},
        # And over a large one.
        {"name": "records_3000017", "kind": "records", "n": 3000017},
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["scene", "scene", "scene", "placing", "fit", "step", "step", "records"])
    if kind == "scene":
        scene = rng.choice(["city", "city", "sponge", "forest"])
        case = {"kind": kind, "scene": scene}
        if scene == "sponge":
            case["depth"] = rng.choice([1, 2, 3, 4])
            case["n"] = _spread(rng, 1, {1: 4000, 2: 2000, 3: 300, 4: 20}[case["depth"]])
        else:
            case["n"] = _spread(rng, 1, 4096 if scene == "city" else 2048)
        small = case["n"] * {"city": BUILDING_TERMINALS, "forest": TREE_TERMINALS,
                             "sponge": 20 ** case.get("depth", 0)}[scene] < 100000
        case["order"] = rng.choice(["path", "leaf"]) if small else "leaf"
        return case
    if kind == "placing":
        n = _spread(rng, 64, 65536)
        return {"kind": kind, "buildings": max(2, n // rng.randint(8, 24)), "trees": n, "boards": max(2, n // 16)}
    if kind == "fit":
        return {"kind": kind, "n": _spread(rng, 1, 2048)}
    if kind == "step":
        scene = rng.choice(["facades", "mixed", "mixed_blocks"])
        return {"kind": kind, "scene": scene, "n": _spread(rng, 16, 4096), "graph": rng.choice([True, False])}
    return {"kind": kind, "n": _spread(rng, 100, 4000000)}


# ---------------------------------------------------------------- inputs

def _same_steps(rng, v, extent, least=0.0):
    """Other lengths that a Repeat of `extent` cuts into as many pieces as v, the last one on the same side of `least`."""
    whole, part = np.floor(v / extent), v / extent - np.floor(v / extent)
    edge = least / extent
    low = rng.uniform(0.1, 0.9, v.shape) * edge
    high = edge + rng.uniform(0.1, 0.9, v.shape) * (1.0 - edge)
    return (extent * (whole + np.where(part < edge, low, high))).astype(np.float32)


def _rebuilt(rng, ax, which):
    """The buildings `which` of a batch with other footprints, heights and places, floor and tile counts kept (the
    number of terminals is that of the scene, whatever the seed)."""
    for k in (0, 1):
        ax["size"][which, k] = _same_steps(rng, ax["size"][which, k].astype(np.float64), 2.5, 1.2)
    ax["custom"][which] = _same_steps(rng, ax["custom"][which].astype(np.float64), 3.0)
    ax["position"][which, :2] += rng.uniform(-4.0, 4.0, (int(which.sum()), 2)).astype(np.float32)


def _batch(case, seed):
    """The batch of a scene: dispatch table, axioms and parameter blocks.  Seeds change the continuous inputs."""
    scene, n = case["scene"], case["n"]
    rng = np.random.default_rng(seed)
    if scene == "city":
        b = scenes.city(n)
        _rebuilt(rng, b["axioms"], np.ones(n, bool))
        return b
    if scene == "sponge":
        b = scenes.menger(SPONGE_THRESHOLDS[case["depth"]], n)
        b["axioms"]["position"] += rng.uniform(-0.1, 0.1, (n, 3)).astype(np.float32)
        b["axioms"]["size"] = rng.uniform(0.95, 1.05, (n, 3)).astype(np.float32)
        return b
    if scene == "forest":
        b = scenes.forest(n, seed=seed)
        b["axioms"]["size"] *= rng.uniform(0.96, 1.04, (n, 3)).astype(np.float32)
        return b
    if scene == "facades":
        b = scenes.facades(n, seed=seed)
        b["axioms"]["size"] = rng.uniform(0.8, 1.25, (n, 3)).astype(np.float32)
        return b
    b = scenes.mixed(n, blocks=scene == "mixed_blocks")
    ax = b["axioms"]
    building = ax["shape"] == G.SHAPE_QUAD
    ax["position"] += rng.uniform(-0.2, 0.2, (n, 3)).astype(np.float32)
    _rebuilt(rng, ax, building)
    if b["blocks"] is not None:
        blocks = b["blocks"].reshape(n, scenes.MIXED_STRIDE)
        blocks[building, 2:] *= rng.uniform(0.8, 1.25, (int(building.sum()), 2)).astype(np.float32)
        blocks[~building] *= rng.uniform(0.98, 1.02, (int((~building).sum()), scenes.MIXED_STRIDE)).astype(np.float32)
    return b


def _placing(case, seed):
    """The collision scene moved as a whole, by steps that keep every distance (and so every placement) as it is."""
    b = scenes.collisions(case["buildings"], case["trees"], case["boards"])
    rng = np.random.default_rng(seed)
    ax = b["axioms"]
    ax["position"] = np.round(ax["position"] * 64.0) / 64.0 + rng.integers(-2000, 2000, 3) / 64.0
    ax["custom"] = rng.uniform(0.0, 1.0, len(ax)).astype(np.float32)
    return b


def _expected(case):
    """Terminals of a case, about (work is counted from it, and the first capacity sized)."""
    if case["kind"] == "placing":
        return int(1.1 * case["trees"]) + 6 * case["buildings"]
    if case["kind"] == "records":
        return case["n"]
    if case["kind"] == "fit":
        return FACADE_TERMINALS * case["n"]
    per = {"city": BUILDING_TERMINALS, "forest": TREE_TERMINALS, "facades": FACADE_TERMINALS,
           "mixed": MIXED_TERMINALS, "mixed_blocks": MIXED_TERMINALS}
    return case["n"] * (20 ** case["depth"] if case["scene"] == "sponge" else per[case["scene"]])


def _records_input(n, seed):
    """Instance records as an importer fills them: boxes and quads of furniture-to-house size, turned about z, in
    clusters (settlements) over a 4 km square, each with a random id in the path field."""
    g = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def uniform(lo, hi, *shape):
        return torch.rand(*shape, generator=g, device=DEVICE) * (hi - lo) + lo

    clusters = max(1, n // 2000)
    home = uniform(0.0, 4000.0, clusters, 2)
    which = torch.randint(0, clusters, (n,), generator=g, device=DEVICE)
    t = torch.empty(n, 3, device=DEVICE)
    t[:, :2] = home[which] + 60.0 * torch.randn(n, 2, generator=g, device=DEVICE)
    t[:, 2] = uniform(0.0, 40.0, n)
    t.clamp_(0.0, 4000.0)
    size = torch.exp(uniform(math.log(0.3), math.log(12.0), n, 3))
    turn = uniform(0.0, 2.0 * math.pi, n)
    rec = torch.zeros(n, 16, device=DEVICE)
    c, s = torch.cos(turn), torch.sin(turn)
    rec[:, 0], rec[:, 1] = c * size[:, 0], -s * size[:, 1]
    rec[:, 4], rec[:, 5] = s * size[:, 0], c * size[:, 1]
    rec[:, 10] = size[:, 2]
    rec[:, 3], rec[:, 7], rec[:, 11] = t[:, 0], t[:, 1], t[:, 2]
    quad = torch.randint(0, 4, (n,), generator=g, device=DEVICE) == 0
    rec.view(torch.int32)[:, 12] = torch.where(quad, -(1 << 31) + 1, 1).to(torch.int32)
    rec.view(torch.int64)[:, 7] = torch.randint(0, 1 << 62, (n,), generator=g, device=DEVICE) * 2 - (1 << 62)
    return rec.view(torch.uint8)


RECORD_BOUNDS = (-1.0, -1.0, -1.0, 4001.0, 4001.0, 41.0)


def _bounds(out, n):
    """The box of the terminal centres, a little widened, as a program keeps it for its scene."""
    c = out[:n].view(torch.float32).view(n, 16)[:, [3, 7, 11]]
    lo, hi = c.min(dim=0).values.cpu().numpy(), c.max(dim=0).values.cpu().numpy()
    pad = 0.01 * (hi - lo) + 0.01
    return tuple(float(v) for v in lo - pad) + tuple(float(v) for v in hi + pad)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "records":
        n = case["n"]
        eng = Engine(scenes.menger_table(0.5), node_capacity=1 << 12, max_terminals=n)
        return {"case": case, "engine": eng, "records": _records_input(n, seed), "n": n, "bounds": RECORD_BOUNDS}
    if kind == "placing":
        b = _placing(case, seed)
        cap = case["trees"] + 6 * case["buildings"] + 2 * case["boards"] + 1024
        eng = Engine(b["entries"], node_capacity=cap, max_terminals=cap)
        return {"case": case, "engine": eng, "axioms": autograd.axioms_tensor(b["axioms"]), "capacity": cap}
    if kind == "fit":
        return _prepare_fit(case, seed)
    b = _batch(case, seed)
    step = kind == "step"
    cap = int(1.35 * _expected(case)) + 20000
    eng = Engine(b["entries"], node_capacity=cap + (1 << 18), max_terminals=cap, block_stride=b["block_stride"],
                 record_tape=step, group_axioms=case["scene"].startswith("mixed"))
    blocks = None if b["blocks"] is None else torch.from_numpy(b["blocks"]).to(DEVICE)
    state = {"case": case, "engine": eng, "axioms": autograd.axioms_tensor(b["axioms"]), "blocks": blocks,
             "n_axioms": len(b["axioms"])}
    # A first derivation gives the count and the extent of the scene, which size the buffers and the tree's grid.
    out, n, _ = eng.execute(state["axioms"], blocks=blocks, capacity=cap)
    state["bounds"] = _bounds(out, n)
    state["capacity"] = min(cap, n + n // 50 + 64)
    del out
    if step:
        state["out"] = torch.empty((state["capacity"], 64), dtype=torch.uint8, device=DEVICE)
        state["count"] = torch.zeros(1, dtype=torch.int64, device=DEVICE)
        state["leaves"] = n  # the axioms and parameters stay: so does the count
        state["g_sizes"] = torch.empty((state["n_axioms"], 3), device=DEVICE)
        state["g_blocks"] = None if blocks is None else torch.empty_like(blocks)
        if case["graph"]:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                _step(state)  # the first call on an engine fixes its launch shapes
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            state["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state["graph"]):
                state["result"] = _step(state)
    return state


def _prepare_fit(case, seed):
    n = case["n"]
    b = scenes.facades(n, seed=seed)
    cap = FACADE_TERMINALS * n + 1024
    eng = Engine(b["entries"], node_capacity=max(1 << 14, 512 * n), max_terminals=cap,
                 block_stride=b["block_stride"], record_tape=True)
    axioms = autograd.axioms_tensor(b["axioms"])
    sizes = torch.ones((n, 3), device=DEVICE)
    goal = torch.from_numpy(scenes.facade_target_params(b["blocks"], seed=seed + 1)).to(DEVICE)
    with torch.no_grad():
        M, paths = autograd.derive_transforms(eng, axioms, goal, sizes, cap)
    return {"case": case, "engine": eng, "axioms": axioms, "capacity": cap, "target": autograd.PathTarget(M, paths),
            "params": torch.from_numpy(b["blocks"]).to(DEVICE).requires_grad_(), "sizes": sizes.requires_grad_()}


# ---------------------------------------------------------------- one pass

def _fields(out, order):
    """The fields of the instance records out[order] (64 bytes each, moved as four 16-byte words, a thread to a word)."""
    n = order.shape[0]
    rec = out.view(torch.complex128)[order[:, None], torch.arange(4, device=out.device)].view(torch.float32)
    w = rec.view(torch.int32)
    return {"m": rec[:, :12], "rule": w[:, 12], "custom": rec[:, 13], "path": rec.view(torch.int64).view(n, 8)[:, 7]}


def _by_path(out, n):
    return _fields(out, torch.argsort(out.view(torch.int64)[:n, 7]))


def _tree(bv, n):
    return {"nodes": bv["nodes"][: n - 1], "parents": bv["leafParents"][:n], "boxes": bv["aabbs"][: n - 1],
            "keys": bv["keys"][:n]}


def _step(state):
    eng = state["engine"]
    out, blocks = state["out"], state["blocks"]
    eng.derive_raw(state["axioms"].data_ptr(), state["n_axioms"], None if blocks is None else blocks.data_ptr(),
                   out.data_ptr(), state["capacity"], state["count"].data_ptr())
    bv = eng.lbvh(out, state["capacity"], state["bounds"], count=state["count"])
    eng.adjoint_raw(out.data_ptr(), None if blocks is None else state["g_blocks"].data_ptr(),
                    0 if blocks is None else state["n_axioms"], state["g_sizes"].data_ptr(), grad_stride=16)
    n = state["leaves"]
    res = _tree(bv, n)
    res["instances"] = _fields(out, bv["leafTerminal"][:n])
    res["g_sizes"] = state["g_sizes"]
    if blocks is not None:
        res["g_blocks"] = state["g_blocks"]
    return res


def run(state):
    case, eng = state["case"], state["engine"]
    kind = case["kind"]
    if kind == "step":
        if "graph" not in state:
            return _step(state)
        state["graph"].replay()
        return state["result"]
    if kind == "fit":
        params, sizes = state["params"], state["sizes"]
        params.grad = sizes.grad = None
        M, paths = autograd.derive_transforms(eng, state["axioms"], params, sizes, state["capacity"])
        loss = state["target"].sse(M, paths)
        loss.backward()
        return {"loss": loss.detach(), "g_params": params.grad, "g_sizes": sizes.grad}
    if kind == "records":
        bv = eng.lbvh(state["records"], state["n"], state["bounds"])
        return {**_tree(bv, state["n"]), "leaf": bv["leafTerminal"]}
    out, n, _ = eng.execute(state["axioms"], blocks=state.get("blocks"), capacity=state["capacity"])
    if case.get("order", "path") == "path":
        return _by_path(out, n)
    bv = eng.lbvh(out, n, state["bounds"])
    return {**_tree(bv, n), "instances": _fields(out, bv["leafTerminal"])}


def work(case):
    """Inputs read once (axioms of 48 bytes, parameter blocks, records of 64 bytes), outputs written once (records; tree
    nodes, parents, boxes, keys and leaf order: 52 bytes a leaf; gradients).  Operations: about 60 a terminal (split,
    frame, hash), 60 a leaf (box, code, merge), 100 a terminal of the adjoint."""
    kind, t = case["kind"], _expected(case)
    tree = kind in ("step", "records") or case.get("order") == "leaf"
    axioms = {"placing": case.get("buildings", 0) + case.get("trees", 0) + case.get("boards", 0),
              "records": 0}.get(kind, case.get("n", 0))
    floats = {"facades": 16, "mixed_blocks": scenes.MIXED_STRIDE}.get(case.get("scene"), 16 if kind == "fit" else 0)
    nbytes = 48 * axioms + 4 * floats * axioms
    if kind == "fit":
        # the transforms are matched with the target's centres and extents (24 bytes each)
        nbytes += 24 * t + (4 * floats + 12) * axioms
    else:
        nbytes += 64 * t + (52 * t if tree else 0)
    if kind == "step":
        nbytes += (4 * floats + 12) * axioms
    flops = (0 if kind == "records" else 60 * t) + (60 * t if tree else 0) + (100 * t if kind in ("fit", "step") else 0)
    return {"bytes": int(nbytes), "flops": int(flops)}


# ---------------------------------------------------------------- the same in 64 bits

_MASK32 = 0xFFFFFFFF


def _shr(z, k):
    return (z >> k) & ((1 << (64 - k)) - 1)


def _signed(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def _mix64(z):
    z = (z ^ _shr(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _child_path(path, ordinal, entry):
    if not torch.is_tensor(ordinal):
        ordinal = torch.full_like(path, ordinal)
    return _mix64(path ^ ((ordinal << 32) | (int(entry) & _MASK32)))


class _Shapes:
    """A batch of shapes at one table entry: translation, size, rotation, path, axiom."""

    def __init__(self, t, s, R, path, axiom):
        self.t, self.s, self.R, self.path, self.axiom = t, s, R, path, axiom

    def pick(self, index):
        return _Shapes(self.t[index], self.s[index], self.R[index], self.path[index], self.axiom[index])

    def but(self, **kw):
        return _Shapes(**{**self.__dict__, **kw})

    def moved(self, axis, o):
        return self.t + self.R[:, :, axis] * o[:, None]

    def sized(self, axis, v):
        return torch.stack([v if k == axis else self.s[:, k] for k in range(3)], dim=1)

    def turned(self, *columns):
        """Columns of the rotation rearranged: (source, sign) for each of the three."""
        return torch.stack([self.R[:, :, c] * sg for c, sg in columns], dim=2)

    @staticmethod
    def joined(parts):
        if len(parts) == 1:
            return parts[0]
        return _Shapes(*(torch.cat([getattr(p, k) for p in parts]) for k in ("t", "s", "R", "path", "axiom")))


class _Table:
    """Derives a batch from its dispatch table in 64 bits, entry by entry, level by level."""

    FACES = [  # axis, sign, rotation columns, size components, successor, ordinal
        (2, -1, ((0, -1), (1, 1), (2, -1)), (0, 1), 2, 2), (2, 1, ((0, 1), (1, 1), (2, 1)), (0, 1), 2, 3),
        (0, -1, ((2, 1), (1, 1), (0, -1)), (2, 1), 2, 4), (0, 1, ((2, -1), (1, 1), (0, 1)), (2, 1), 2, 5),
        (1, -1, ((0, 1), (2, 1), (1, -1)), (0, 2), 1, 1), (1, 1, ((0, 1), (2, -1), (1, 1)), (0, 2), 0, 0)]

    def __init__(self, entries, axioms, blocks, stride):
        self.rules = []
        for e in entries:
            p = G.DEFAULT_PROCS[int(e["operatorCode"])]
            params = [(int(q["type"]), q["value"].copy()) for q in e["parameters"][: int(e["numParameters"])]]
            succ = [int(q["entryIndex"]) for q in e["successors"][: int(e["numSuccessors"])]]
            self.rules.append((int(p["op"]), int(p["numChildren"]), int(p["shape"]), params, succ))
        self.custom = torch.from_numpy(axioms["custom"].astype(np.float64)).to(DEVICE)
        self.block = torch.from_numpy(axioms["block"].astype(np.int64)).to(DEVICE)
        self.blocks, self.stride = blocks, stride
        self.axioms = axioms

    def param(self, p, x):
        kind, v = p
        if kind == G.PT_SCALAR:
            return torch.full((len(x.path),), float(v[0]), dtype=torch.float64, device=DEVICE)
        if kind == G.PT_BLOCK:
            return self.blocks.view(-1, self.stride)[self.block[x.axiom], int(v[0])]
        if kind == G.PT_SHAPE_ATTR:
            return self.attribute(int(v[0]), x)
        assert kind == G.PT_EXP
        stack = []
        for word in v[1 : 1 + int(v[0])].view(np.uint32):
            op, value = int(word) >> 30, float(np.uint32((int(word) << 2) & _MASK32).view(np.float32))
            if op == G.ORT_SCALAR:
                stack.append(torch.full((len(x.path),), value, dtype=torch.float64, device=DEVICE))
            elif op == G.ORT_SHAPE_ATTR:
                stack.append(self.attribute(int(round(value)), x))
            else:
                b, a = stack.pop(), stack.pop()
                stack.append([a + b, a - b, a / b, a * b][int(round(value))])
        return stack[-1]

    def attribute(self, k, x):
        return self.custom[x.axiom] if k == 16 else x.s[:, k - 12]

    def derive(self, sizes):
        """Terminals as (M, axiom, path), unordered; `sizes` (numAxioms x 3) may ask for its gradient."""
        n = len(self.axioms)
        at = torch.from_numpy(self.axioms["position"].astype(np.float64)).to(DEVICE)
        ids = torch.arange(n, device=DEVICE)
        eye = torch.eye(3, dtype=torch.float64, device=DEVICE).expand(n, 3, 3)
        whole = _Shapes(at, sizes, eye, _mix64(ids + _signed(0x9E3779B97F4A7C15)), ids)
        entry = self.axioms["entry"]
        todo = {int(e): [whole.pick(torch.from_numpy(np.nonzero(entry == e)[0]).to(DEVICE))] for e in np.unique(entry)}
        self.done = []
        while todo:
            self.next = {}
            for e in sorted(todo):
                self.expand(e, _Shapes.joined(todo[e]))
            todo = self.next
        return [torch.cat(part) for part in zip(*self.done)]

    def to(self, entry, x, ordinal=None):
        if ordinal is not None:
            x = x.but(path=_child_path(x.path, ordinal, entry))
        if len(x.path):
            self.next.setdefault(entry, []).append(x)

    def expand(self, e, x):
        op, pairs, shape, params, succ = self.rules[e]
        value = [self.param(p, x) for p in params] if op not in (G.OP_GENERATE, G.OP_ROTATE) else []
        axis = int(params[0][1][0]) if params and params[0][0] == G.PT_SCALAR else 0
        if op == G.OP_GENERATE:
            M = torch.cat([x.R * x.s[:, None, :], x.t[:, :, None]], dim=2).reshape(-1, 12)
            self.done.append((M, x.axiom, x.path))
        elif op == G.OP_IF_SIZE_LESS:
            less = x.s[:, axis] < value[1]
            self.to(succ[0], x.pick(less), 0)
            self.to(succ[1], x.pick(~less), 1)
        elif op == G.OP_EXTRUDE:
            s = torch.stack([x.s[:, 0], value[1], x.s[:, 1]], dim=1)
            self.to(succ[0], x.but(s=s, R=x.turned((0, 1), (2, 1), (1, -1))), 0)
        elif op == G.OP_TRANSLATE:
            self.to(succ[0], x.but(t=x.t + (x.R * torch.stack(value, dim=1)[:, None, :]).sum(dim=2)))
        elif op == G.OP_SCALE:
            s = [torch.where(v < 0, -v * x.s[:, k], v) for k, v in enumerate(value)]
            self.to(succ[0], x.but(s=torch.stack(s, dim=1)))
        elif op == G.OP_ROTATE:
            self.to(succ[0], x.but(R=x.R @ _rotation([float(p[1][0]) for p in params])))
        elif op == G.OP_REPLICATE:
            for c, nxt in enumerate(succ):
                self.to(nxt, x, c)
        elif op in (G.OP_SUBDIVIDE, G.OP_SUBDIVIDE_STATIC):
            f = value[1 : 1 + pairs] if op == G.OP_SUBDIVIDE_STATIC else value[1:]
            total = x.s[:, axis]
            fixed, shares = sum(v.clamp(min=0) for v in f), sum((-v).clamp(min=0) for v in f)
            scale = torch.where(shares > 0, (total - fixed) / shares.clamp(min=1e-300), torch.zeros_like(total))
            offset = -0.5 * total
            for c, v in enumerate(f):
                size = torch.where(v < 0, -v * scale, v)
                self.to(succ[c], x.but(s=x.sized(axis, size), t=x.moved(axis, offset + 0.5 * size)), c)
                offset = offset + size
        elif op == G.OP_REPEAT:
            self.repeat(x, axis, value[1], int(params[2][1][0]), succ[0])
        elif op == G.OP_COMPONENT_SPLIT:
            for k, sign, columns, (u, v), which, ordinal in self.FACES:
                s = torch.stack([x.s[:, u], x.s[:, v], torch.ones_like(x.s[:, 0])], dim=1)
                y = x.but(t=x.moved(k, 0.5 * sign * x.s[:, k]), s=s, R=x.turned(*columns))
                self.to(succ[which], y, ordinal)
        else:
            assert op == G.OP_DISCARD

    def repeat(self, x, axis, extent, mode, nxt):
        total = x.s[:, axis]
        extent = torch.where(extent < 0, -extent * total, extent)
        if mode == G.ADJUST_TO_FILL:
            reps = torch.floor(total.detach() / extent.detach())
            first = middle = last = total / reps.clamp(min=1)
        else:
            reps = torch.ceil(total.detach() / extent.detach())
            rest = total - (reps - 1) * extent
            first, middle, last = (rest, extent, extent) if mode == G.ANCHOR_TO_START else (extent, extent, rest)
        reps = reps.clamp(min=1).to(torch.int64)
        who = torch.repeat_interleave(torch.arange(len(reps), device=DEVICE), reps)
        c = torch.arange(len(who), device=DEVICE) - (torch.cumsum(reps, 0) - reps)[who]
        first, middle, last, total = first[who], middle[who], last[who], total[who]
        isfirst, islast = c == 0, (c > 0) & (c + 1 == reps[who])
        size = torch.where(isfirst, first, torch.where(islast, last, middle))
        before = torch.where(isfirst, torch.zeros_like(first), first + (c - 1).clamp(min=0) * middle)
        y = x.pick(who)
        y = y.but(t=y.moved(axis, before + 0.5 * size - 0.5 * total), s=y.sized(axis, size))
        self.to(nxt, y, c + 1)


def _rotation(degrees):
    (sa, sb, sg), (ca, cb, cg) = (np.sin(np.radians(degrees)), np.cos(np.radians(degrees)))
    return torch.tensor([[cb * cg, cg * sa * sb - ca * sg, ca * cg * sb + sa * sg],
                         [cb * sg, ca * cg + sa * sb * sg, -cg * sa + ca * sb * sg],
                         [-sb, cb * sa, ca * cb]], dtype=torch.float64, device=DEVICE)


def _record_boxes(rec, bounds):
    """Boxes of the radix tree's internal nodes over records, in 64 bits.  The tree is the one of the Morton codes of the
    centres (30 bits) and, for equal codes, of the positions in (code, path) order."""
    n = rec.shape[0]
    f = rec.view(torch.float32).view(n, 16)
    code = torch.zeros(n, dtype=torch.int64, device=DEVICE)
    for k in range(3):
        lo = torch.tensor(bounds[k], dtype=torch.float32, device=DEVICE)
        hi = torch.tensor(bounds[3 + k], dtype=torch.float32, device=DEVICE)
        cell = ((f[:, 4 * k + 3] - lo) / (hi - lo) * 1023.0).to(torch.int64)
        for bit in range(10):
            code |= ((cell >> bit) & 1) << (3 * bit + k)
    path = rec.view(torch.int64).view(n, 8)[:, 7]
    order = torch.argsort(path ^ (-1 << 63))  # as unsigned numbers
    order = order[torch.argsort(code[order], stable=True)]
    code = (code[order] << 32) | torch.arange(n, device=DEVICE)
    m = f[order].double()
    half = 0.5 * torch.stack([m[:, 0:3].abs(), m[:, 4:7].abs(), m[:, 8:11].abs()], dim=1)
    quad = rec.view(torch.int32).view(n, 16)[order, 12] < 0
    half[quad, :, 2] = 0.0
    half, t = half.sum(dim=2), m[:, [3, 7, 11]]
    low, high = t - half, t + half

    i = torch.arange(n - 1, device=DEVICE)

    def common(j):
        """Leading bits that the codes at i and j share, -1 outside."""
        inside = (j >= 0) & (j < n)
        diff = code[i] ^ code[j.clamp(0, n - 1)]
        top = torch.zeros_like(diff)
        for s in (32, 16, 8, 4, 2, 1):
            more = (diff >> s) > 0
            top, diff = torch.where(more, top + s, top), torch.where(more, diff >> s, diff)
        return torch.where(inside, 63 - top, torch.full_like(top, -1))

    after, before = common(i + 1), common(i - 1)
    d = torch.where(after >= before, 1, -1)
    least = torch.minimum(after, before)
    length = torch.zeros_like(i)
    step = 1 << int(math.ceil(math.log2(n)))
    while step:
        further = common(i + (length + step) * d) > least
        length = torch.where(further, length + step, length)
        step >>= 1
    start, count = torch.where(d > 0, i, i - length), length + 1
    boxes = torch.empty(n - 1, 6, dtype=torch.float64, device=DEVICE)
    level = torch.floor(torch.log2(count.double())).to(torch.int64)
    width, k = 1, 0
    while width <= n:  # low[p], high[p] cover the leaves [p, p + width)
        here = torch.nonzero(level == k).flatten()
        a, b = start[here], start[here] + count[here] - width
        boxes[here] = torch.cat([torch.minimum(low[a], low[b]), torch.maximum(high[a], high[b])], dim=1)
        if n - width < width:
            break
        low, high = torch.minimum(low[:-width], low[width:]), torch.maximum(high[:-width], high[width:])
        width, k = 2 * width, k + 1
    return boxes


def exact(case, seed):
    kind = case["kind"]
    if kind == "records":
        boxes = _record_boxes(_records_input(case["n"], seed), RECORD_BOUNDS)
        return {"nodes": None, "parents": None, "boxes": boxes, "keys": None, "leaf": None}
    if kind == "placing":
        return None  # overlap tests between phases
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "scene" and case["order"] == "leaf":
        return None  # the order of the leaves hangs on the last bit of a centre
    if _expected(case) > 4000000:
        return None
    b = _batch(case, seed)
    blocks = None if b["blocks"] is None else torch.from_numpy(b["blocks"].astype(np.float64)).to(DEVICE)
    sizes = torch.from_numpy(b["axioms"]["size"].astype(np.float64)).to(DEVICE)
    if kind == "scene":
        M, axiom, path = _Table(b["entries"], b["axioms"], blocks, b["block_stride"]).derive(sizes)
        order = torch.argsort(path)
        custom = torch.from_numpy(b["axioms"]["custom"].astype(np.float64)).to(DEVICE)[axiom]
        return {"m": M[order], "rule": None, "custom": custom[order], "path": None}
    sizes.requires_grad_()
    if blocks is not None:
        blocks.requires_grad_()
    M = _Table(b["entries"], b["axioms"], blocks, b["block_stride"]).derive(sizes)[0]
    (0.5 * M.square().sum()).backward()
    res = {"nodes": None, "parents": None, "boxes": None, "keys": None, "instances": None, "g_sizes": sizes.grad}
    if blocks is not None:
        res["g_blocks"] = blocks.grad
    return res


def _exact_fit(case, seed):
    b = scenes.facades(case["n"], seed=seed)
    goal = scenes.facade_target_params(b["blocks"], seed=seed + 1)

    def look(blocks, sizes):
        M, _, path = _Table(b["entries"], b["axioms"], blocks, b["block_stride"]).derive(sizes)
        M = M[torch.argsort(path)]
        R = M.view(-1, 3, 4)[:, :, :3]
        return torch.cat([M[:, [3, 7, 11]], R.square().sum(dim=1).sqrt()], dim=1)

    sizes = torch.ones((case["n"], 3), dtype=torch.float64, device=DEVICE, requires_grad=True)
    params = torch.from_numpy(b["blocks"].astype(np.float64)).to(DEVICE).requires_grad_()
    with torch.no_grad():
        want = look(torch.from_numpy(goal.astype(np.float64)).to(DEVICE), sizes)
    loss = (look(params, sizes) - want).square().sum()
    loss.backward()
    return {"loss": loss.detach(), "g_params": params.grad, "g_sizes": sizes.grad}
