"""The work that users of this engine have it do, as a list of sized cases.

Four kinds of programs call the package:

- "ticks": a d3 simulation driven through the facade. The program sets the
  node table's positions, asks for some ticks (`Simulation.tick`) and reads
  x, y, vx, vy. Exact mode and the three forms of fast mode, with the forces
  that the reference's own scenarios combine.
- "batch": many small layouts ticked together (`batch.Batch`), each tick read
  back as float32 arrays.
- "kick": the batched many-body force alone (`Batch.kick`), as a host that
  integrates by itself uses it.
- "train": the learned form's network trained on the GPU (`learned.train`).

`exact` restates the passes that have a value independent of the order of
their operations (the fast forms' forces as direct sums and Jacobi passes,
the network's training) in float64. Exact mode's results are defined by d3's
tree and visit order and have no such value.
"""

import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("d3-force-wasm_b200")
batches = importlib.import_module("d3-force-wasm_b200.batch")
learned = importlib.import_module("d3-force-wasm_b200.learned")

ALPHA_DECAY = 1 - 0.001 ** (1 / 300)
DECAY = 0.6

# every option of a "ticks" case and its default
TICKS = {"kind": "ticks", "n": 1000, "ticks": 1, "mode": "exact", "form": "plain", "order": 8,
         "layout": "spiral", "links": "uniform", "radius": 0.0, "collide_iterations": 1,
         "link_iterations": 1, "center": True, "axes": False, "radial": False, "theta": 0.9,
         "distance_max": 0.0, "coincident": 0.0, "near": 0.0, "pinned": 0.0}


def ticks_case(name, **kw):
    return dict(TICKS, name=name, **kw)


def listed():
    return [
        # an interactive graph of a few dozen nodes, one frame per tick: pure latency
        ticks_case("exact_77_frame", n=77, layout="uniform"),
        # a static layout of 1,000 nodes: the whole 300-tick schedule in one call
        ticks_case("exact_1k_schedule", n=1000, ticks=300),
        # an odd-sized graph with every exact force and option in use
        ticks_case("exact_5003_options", n=5003, ticks=10, layout="mixture", radius=4.0,
                   collide_iterations=2, link_iterations=2, axes=True, radial=True, theta=0.7,
                   distance_max=800.0, pinned=0.01),
        # exact mode at scale, with coincident, nearly coincident and pinned nodes
        ticks_case("exact_50k_collide", n=50000, ticks=20, radius=5.0, coincident=0.01, near=0.01,
                   pinned=0.005),
        # a medium graph in the reference's fast mode, frame by frame, with its collide
        ticks_case("fast_6k_frame", n=6001, mode="fast", layout="mixture", radius=3.0),
        # the reference's FMM at a million nodes
        ticks_case("fast_1m_plain", n=1000000, ticks=4, mode="fast", layout="uniform"),
        # the tensor-core form at a million nodes, a run of ticks between two reads
        ticks_case("fast_1m_tensor", n=1000000, ticks=3, mode="fast", form="bf16x3",
                   layout="uniform"),
        # the tensor-core form on a clustered graph of odd size, many-body and links
        ticks_case("fast_41k_tensor", n=41003, ticks=2, mode="fast", form="bf16x3",
                   layout="mixture", links="blocks", center=False),
        # the learned form (its sampled check and its fallback) on clusters
        ticks_case("learned_200k", n=200003, ticks=2, mode="fast", form="learned",
                   layout="mixture", links="blocks"),
        # a dashboard of small layouts with positions of their own, frame by frame
        {"kind": "batch", "name": "batch_40_frame", "graphs": 40, "nmin": 64, "nmax": 2048,
         "layout": "mixture", "ticks": 1, "threads": 512, "per_sm": 1, "leaf": 16},
        # thousands of graphs of uneven sizes, about six million nodes
        {"kind": "batch", "name": "batch_2048", "graphs": 2048, "nmin": 64, "nmax": 16384,
         "layout": "spiral", "ticks": 1, "threads": 1024, "per_sm": 1, "leaf": 16},
        # the network's training: forward, backward and Adam
        {"kind": "train", "name": "train_200", "samples": 100000, "steps": 200, "batch": 8192,
         "rate": 2e-3},
    ]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["exact", "exact", "exact", "plain", "tensor", "tensor", "learned", "batch",
                       "batch", "kick", "train"])
    if kind == "exact":
        n = log_uniform(rng, 40, 50000)
        case = dict(TICKS, n=n, ticks=rng.randint(1, max(1, min(100, 400000 // n))),
                    layout=rng.choice(["spiral", "uniform", "mixture"]),
                    links=rng.choice(["uniform", "blocks"]),
                    radius=rng.choice([0.0, 0.0, round(rng.uniform(2, 6), 2)]),
                    collide_iterations=rng.choice([1, 1, 2]), link_iterations=rng.choice([1, 1, 2]),
                    center=rng.random() < 0.8, axes=rng.random() < 0.3, radial=rng.random() < 0.15,
                    theta=rng.choice([0.9, 0.9, 0.7]),
                    distance_max=rng.choice([0.0, 0.0, 600.0]),
                    coincident=rng.choice([0.0, 0.01]), pinned=rng.choice([0.0, 0.005]))
        return case
    if kind in ("plain", "tensor", "learned"):
        n = log_uniform(rng, 2000, 700000 if kind != "learned" else 250000)
        return dict(TICKS, n=n, ticks=rng.randint(1, 2 if n > 100000 or kind != "plain" else 4),
                    mode="fast",
                    form={"plain": "plain", "tensor": "bf16x3", "learned": "learned"}[kind],
                    layout=rng.choice(["uniform", "mixture"]),
                    links=rng.choice(["uniform", "blocks"]),
                    radius=rng.choice([0.0, 3.0]) if kind == "plain" else 0.0,
                    center=rng.random() < 0.7,
                    distance_max=rng.choice([0.0, 0.0, 900.0]) if kind == "plain" else 0.0)
    if kind == "train":
        return {"kind": "train", "samples": log_uniform(rng, 9000, 150000),
                "steps": rng.randint(20, 200), "batch": rng.choice([1000, 4096, 8192]),
                "rate": 2e-3}
    nmax = log_uniform(rng, 256, 16384)
    return {"kind": kind, "graphs": log_uniform(rng, 1, min(1500, 3000000 // nmax)), "nmin": 64,
            "nmax": nmax, "layout": "mixture" if kind == "kick" else rng.choice(["spiral", "mixture"]),
            "ticks": rng.randint(1, 2), "threads": rng.choice([256, 512, 1024]),
            "per_sm": 1, "leaf": rng.choice([8, 16, 32])}


# ---- inputs -------------------------------------------------------------------------------------


def layout(kind, n, rng):
    """Start positions: d3's phyllotaxis, uniform or a mixture of Gaussian
    clusters at its density (one node per 100 square units)."""
    if kind == "spiral":
        i = np.arange(n, dtype=np.float64)
        r, a = 10 * np.sqrt(0.5 + i), i * (math.pi * (3 - math.sqrt(5)))
        return r * np.cos(a), r * np.sin(a)
    side = 10 * math.sqrt(n)
    if kind == "uniform":
        return rng.random(n) * side, rng.random(n) * side
    k = 16
    label = rng.integers(0, k, n)
    sigma = side * (0.02 + 0.06 * rng.random(k))
    return ((rng.random(k) * side)[label] + sigma[label] * rng.standard_normal(n),
            (rng.random(k) * side)[label] + sigma[label] * rng.standard_normal(n))


def positions(case, rng):
    """A simulation's start, with some nodes on or next to others."""
    n = case["n"]
    x, y = layout(case["layout"], n, rng)
    for share, scale in ((case["coincident"], 0.0), (case["near"], 1e-12)):
        k = int(share * n)
        if k:
            i, j = rng.choice(n, k, replace=False), rng.integers(0, n, k)
            x[i] = x[j] + scale * (rng.random(k) - 0.5)
            y[i] = y[j] + scale * (rng.random(k) - 0.5)
    return x, y


def links(case, rng):
    """m = 2n links: uniform endpoints, or mostly within 16 index blocks."""
    n, m = case["n"], 2 * case["n"]
    src = rng.integers(0, n, m)
    if case["links"] == "uniform":
        tgt = (src + 1 + rng.integers(0, n - 1, m)) % n
    else:
        size = max(2, n // 16)
        start = np.minimum(src // size * size, n - size)
        tgt = np.where(rng.random(m) < 0.8, start + rng.integers(0, size, m), rng.integers(0, n, m))
        tgt = np.where(tgt == src, (tgt + 1) % n, tgt)
    return src, tgt


def ticks_inputs(case, seed):
    rng = np.random.default_rng([seed, 11])
    x, y = positions(case, rng)
    src, tgt = links(case, rng)
    pin = rng.choice(case["n"], int(case["pinned"] * case["n"]), replace=False)
    return x, y, src, tgt, pin


def batch_inputs(case, seed):
    """[(n, src, tgt)] and [(x, y)]: sizes log-uniform in [nmin, nmax] in no
    order, m = 2n links; half the graphs uniform, half mostly within 8
    communities."""
    rng = np.random.default_rng([seed, 12])
    span, graphs, starts = math.log(case["nmax"] / case["nmin"]), [], []
    for g in range(case["graphs"]):
        n = int(round(case["nmin"] * math.exp(span * ((g * 0.6180339887498949 + 0.5) % 1.0))))
        src = rng.integers(0, n, 2 * n)
        tgt = rng.integers(0, n, 2 * n)
        if g % 2:
            inside = (src % 8) + 8 * rng.integers(0, n // 8, 2 * n)
            tgt = np.where(rng.random(2 * n) < 0.74, inside, tgt)
        tgt = np.where(tgt == src, (tgt + 1) % n, tgt)
        graphs.append((n, src.astype(np.uint32), tgt.astype(np.uint32)))
        starts.append(layout(case["layout"], n, rng))
    return graphs, starts


def train_inputs(case, seed):
    """Leaf rows as the order-4 pass gives them: scaled coefficients of
    falling size, level / 16, count / 32, a small mean offset; the targets a
    smooth function of them plus noise."""
    rng = np.random.default_rng([seed, 13])
    n = case["samples"]
    x = np.empty((n, 12), np.float32)
    x[:, :8] = rng.standard_normal((n, 8)) * np.repeat(0.5 ** np.arange(4), 2)
    x[:, 8] = rng.integers(5, 10, n) / 16
    x[:, 9] = rng.integers(1, 33, n) / 32
    x[:, 10:] = 0.2 * rng.standard_normal((n, 2))
    w = rng.standard_normal((12, 2))
    y = np.tanh(x @ w) + 0.3 * rng.standard_normal((n, 2))
    return x, y.astype(np.float32)


# ---- the programs -------------------------------------------------------------------------------


class Result(dict):
    """Arrays by name, and the program whose memory they view."""

    def __init__(self, owner, **arrays):
        super().__init__(arrays)
        self.owner = owner


class Ticks:
    """A simulation and the arrays that the program sets before each run."""

    def __init__(self, case, seed):
        x, y, src, tgt, pin = ticks_inputs(case, seed)
        n = case["n"]
        self.case, self.x, self.y = case, x, y
        self.nodes = pkg.Nodes(n, x=x, y=y, vx=np.zeros(n), vy=np.zeros(n))
        self.nodes.fx[pin], self.nodes.fy[pin] = x[pin], y[pin]
        self.sim = sim = pkg.forceSimulation(self.nodes)
        charge = pkg.forceManyBody().theta(case["theta"])
        if case["distance_max"]:
            charge.distanceMax(case["distance_max"])
        sim.force("charge", charge)
        sim.force("link", pkg.forceLink(src, tgt).iterations(case["link_iterations"]))
        if case["radius"]:
            sim.force("collide",
                      pkg.forceCollide(case["radius"]).iterations(case["collide_iterations"]))
        if case["axes"]:
            sim.force("x", pkg.forceX(3.0))
            sim.force("y", pkg.forceY(-5.0))
        if case["radial"]:
            sim.force("radial", pkg.forceRadial(4.0 * math.sqrt(n)))
        if case["center"]:
            sim.force("center", pkg.forceCenter())
        if case["mode"] == "fast":
            sim.precision("fast", order=case["order"], opening=1.5, form=case["form"])
            if case["form"] == "learned":
                sim.learned(learned.init_params(seed))

    def run(self):
        nodes = self.nodes
        torch.from_numpy(nodes.x).copy_(torch.from_numpy(self.x))
        torch.from_numpy(nodes.y).copy_(torch.from_numpy(self.y))
        torch.from_numpy(nodes.vx).zero_()
        torch.from_numpy(nodes.vy).zero_()
        self.sim.alpha(1.0).tick(self.case["ticks"])
        out = Result(self, x=nodes.x, y=nodes.y, vx=nodes.vx, vy=nodes.vy)
        if self.case["form"] != "plain":
            # the FP32 forms' programs draw from float32 buffers
            out = {k: torch.from_numpy(v).to(torch.float32) for k, v in out.items()}
        return out

    def __del__(self):
        if hasattr(self, "sim"):
            self.sim.close()


class Graphs:
    """A batch of layouts with its launch shape."""

    def __init__(self, case, seed):
        self.case = case
        self.batch = batches.Batch(pkg.cuda_core(), *batch_inputs(case, seed))
        self.batch.set_shape(case["threads"], case["per_sm"], case["leaf"])

    def run(self):
        if self.case["kind"] == "kick":
            return {"kick": self.batch.kick()[0]}
        self.batch.run(self.case["ticks"])
        return dict(zip(("x", "y", "vx", "vy"), self.batch.read()))

    def __del__(self):
        if hasattr(self, "batch"):
            self.batch.close()


class Training:
    """The samples of a training run."""

    def __init__(self, case, seed):
        self.case = case
        self.x, self.y = train_inputs(case, seed)

    def run(self):
        c = self.case
        params, losses = learned.train(pkg.cuda_core(), self.x, self.y, steps=c["steps"],
                                       batch=c["batch"], lr=c["rate"])
        return {"params": params, "losses": losses}


def prepare(case, seed):
    kind = case["kind"]
    return (Ticks if kind == "ticks" else Training if kind == "train" else Graphs)(case, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without --------------------------------------------------------------


def work(case):
    if case["kind"] == "train":
        per = 12 * 64 + 64 * 64 + 64 * 2
        seen = case["steps"] * min(case["batch"], case["samples"])
        # the samples once, the parameters in and out; forward 2, backward 4 flops per weight
        return {"bytes": 56 * min(case["samples"], seen) + 8 * (per + 130), "flops": 6.0 * per * seen}
    if case["kind"] != "ticks":
        sizes = [64 * (case["nmax"] / 64) ** ((g + 0.5) / case["graphs"])
                 for g in range(case["graphs"])]
        n = sum(sizes)
        if case["kind"] == "kick":
            return {"bytes": 16 * n, "flops": 1500 * n}
        # x, y, vx, vy in and out, the 2n links' endpoints and parameters; per node and tick the
        # expansions (about 1,000 flops), 13 leaves of 8 points (12 flops a pair), links, collide
        return {"bytes": (32 + 2 * 12) * n, "flops": 2500.0 * n * case["ticks"]}
    n, t = case["n"], case["ticks"]
    data = n * (48 + 32) + 2 * n * (8 + 24)  # node state up and down, the links
    if case["mode"] == "exact":
        # Barnes-Hut: about 16 log2(n) interactions of 10 flops; 4 links a node of 15 flops
        per = 160 * math.log2(n) + 60 * case["link_iterations"]
        if case["radius"]:
            per += 200 * case["collide_iterations"]
    else:
        # FMM of order 8: about 250 near pairs of 10 flops and 1,000 flops of expansions
        per = 3500 + 60 * case["link_iterations"] + (200 if case["radius"] else 0)
    return {"bytes": float(data), "flops": float(per * n * t)}


# ---- the same in float64 ------------------------------------------------------------------------


def direct(x, y, strength, dmax2=math.inf):
    """sum_j strength (r_j - r_i) / l with d3's clamp below distanceMin 1."""
    kx, ky = torch.zeros_like(x), torch.zeros_like(y)
    rows = max(1, min(len(x), (1 << 25) // len(x)))
    for a in range(0, len(x), rows):
        dx, dy = x[None, :] - x[a:a + rows, None], y[None, :] - y[a:a + rows, None]
        l = dx * dx + dy * dy
        out = (l == 0) | (l >= dmax2)
        l = torch.where(l < 1, torch.sqrt(l), l)
        w = strength / l.masked_fill_(out, math.inf)
        kx[a:a + rows], ky[a:a + rows] = (dx * w).sum(1), (dy * w).sum(1)
    return kx, ky


def jacobi_links(x, y, vx, vy, src, tgt, alpha, distance=30.0):
    """Each node's own side of its links, from the snapshot x + v."""
    n = len(x)
    px, py = x + vx, y + vy
    degree = torch.bincount(src, minlength=n) + torch.bincount(tgt, minlength=n)
    ds, dt = degree[src].double(), degree[tgt].double()
    strength, bias = 1 / torch.minimum(ds, dt), ds / (ds + dt)
    dx, dy = px[tgt] - px[src], py[tgt] - py[src]
    l = torch.sqrt(dx * dx + dy * dy)
    f = (l - distance) / l * alpha * strength
    vx = vx.index_add(0, tgt, -dx * f * bias).index_add(0, src, dx * f * (1 - bias))
    vy = vy.index_add(0, tgt, -dy * f * bias).index_add(0, src, dy * f * (1 - bias))
    return vx, vy


def jacobi_collide(x, y, vx, vy, radius):
    """Equal radii: each node takes half of each overlap, from x + v."""
    px, py = x + vx, y + vy
    ox, oy = torch.zeros_like(x), torch.zeros_like(y)
    rows = max(1, min(len(x), (1 << 25) // len(x)))
    for a in range(0, len(x), rows):
        dx, dy = px[a:a + rows, None] - px[None, :], py[a:a + rows, None] - py[None, :]
        l = torch.sqrt(dx * dx + dy * dy)
        push = torch.where((l < 2 * radius) & (l > 0), (2 * radius - l) / l * 0.5, 0.0)
        ox[a:a + rows], oy[a:a + rows] = (dx * push).sum(1), (dy * push).sum(1)
    return vx + ox, vy + oy


def fast_ticks(x, y, src, tgt, ticks, radius, link_iterations=1, collide_iterations=1,
               center=False, dmax2=math.inf):
    """Ticks of a fast-mode simulation from rest, all on `x`'s device."""
    vx, vy, alpha = torch.zeros_like(x), torch.zeros_like(y), 1.0
    for _ in range(ticks):
        alpha += (0 - alpha) * ALPHA_DECAY
        kx, ky = direct(x, y, -30.0 * alpha, dmax2)
        vx, vy = vx + kx, vy + ky
        for _ in range(link_iterations):
            vx, vy = jacobi_links(x, y, vx, vy, src, tgt, alpha)
        for _ in range(collide_iterations if radius else 0):
            vx, vy = jacobi_collide(x, y, vx, vy, radius)
        if center:
            x, y = x - x.mean(), y - y.mean()
        vx, vy = vx * DECAY, vy * DECAY
        x, y = x + vx, y + vy
    return x, y, vx, vy


def on_device(*arrays):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return [torch.from_numpy(np.asarray(a)).to(dev, torch.int64 if np.asarray(a).dtype.kind in "iu"
                                               else torch.float64) for a in arrays]


def exact_batch(case, seed):
    parts = []
    for (n, src, tgt), (x, y) in zip(*batch_inputs(case, seed)):
        x, y, src, tgt = on_device(x.astype(np.float32), y.astype(np.float32), src, tgt)
        if case["kind"] == "kick":
            parts.append((torch.stack(direct(x, y, -30.0 * (1 - ALPHA_DECAY)), 1),))
        else:
            parts.append(fast_ticks(x, y, src, tgt, case["ticks"], 3.0))
    whole = [torch.cat(p) for p in zip(*parts)]
    if case["kind"] == "kick":
        return {"kick": whole[0]}
    return dict(zip(("x", "y", "vx", "vy"), whole))


def exact_train(case, seed):
    """Adam on the network in float64, from learned.train's own start."""
    x, y = train_inputs(case, seed)
    perm = np.random.default_rng(0).permutation(len(x))  # learned.train's shuffle
    start = np.random.default_rng(0)
    w = []
    for fan_in, fan_out in ((12, 64), (64, 64), (64, 2)):  # He-scaled float32 weights, zero biases
        flat = (start.standard_normal(fan_in * fan_out) * np.sqrt(2.0 / fan_in)).astype(np.float32)
        w += [flat.reshape(fan_out, fan_in), np.zeros(fan_out, np.float32)]
    x, y = on_device(x[perm], y[perm])
    w = [p.requires_grad_() for p in on_device(*w)]
    adam = torch.optim.Adam(w, lr=case["rate"], betas=(0.9, 0.999), eps=1e-8)
    n, size, at, losses = len(x), min(case["batch"], len(x)), 0, []
    for _ in range(case["steps"]):
        if at + size > n:
            at = 0
        h, t = x[at:at + size], y[at:at + size]
        at += size
        for k in (0, 2):
            h = torch.nn.functional.gelu(h @ w[k].T + w[k + 1])
        loss = ((h @ w[4].T + w[5] - t) ** 2).sum(1).mean()
        adam.zero_grad()
        loss.backward()
        adam.step()
        losses.append(float(loss))
    return {"params": torch.cat([p.detach().reshape(-1) for p in w]),
            "losses": torch.tensor(losses, dtype=torch.float64)}


def exact(case, seed):
    if case["kind"] == "train":
        return exact_train(case, seed)
    if case["kind"] in ("batch", "kick"):
        return exact_batch(case, seed)
    if case["mode"] == "exact":
        return None  # d3's tree, visit order and serial loops define the value
    if float(case["n"]) ** 2 * case["ticks"] > 2e11:
        return None  # the direct sum takes too long
    x, y, src, tgt, _ = ticks_inputs(case, seed)
    x, y, src, tgt = on_device(x, y, src, tgt)
    dmax2 = case["distance_max"] ** 2 if case["distance_max"] else math.inf
    return dict(zip(("x", "y", "vx", "vy"),
                    fast_ticks(x, y, src, tgt, case["ticks"], case["radius"],
                               case["link_iterations"], case["collide_iterations"], case["center"],
                               dmax2)))
