"""The work this library is measured on: what a program that uses it calls, over the sizes it calls it with.

Four kinds of call, each through the Python face of the C ABI:

  build     LBVH build of a triangle mesh that is already in device memory (a rebuild per mesh or per frame)
  optimize  LBVH build followed by Bittner13 iterations on a kept workspace, plain or with a learned scorer
  trace     closest hits: a camera image, a frame with one diffuse bounce, or a batch of given rays
  batch     many meshes of uneven size built, optimised and traced by one captured graph
  log       logging of (feature row, realised gain) pairs from a plain optimizer run
  train     training of the reinsertion scorer on logged pairs

The scenes are the seeded synthetic ones of the benchmark configurations, drawn here on the device so that
they are quick to make: uniform triangle soups, a Gaussian mixture over a ground grid, and a Gaussian mixture
with rotated, tessellated boxes.
"""
import math

import numpy as np
import torch

from bvhtest_gb300 import api, learned

CAMERAS = {
    # the small scene's pinhole in front of the unit cube, and the large scene's from above the ground
    "uniform": dict(pos=(0.5, 0.5, -1.5), lookAt=(0.5, 0.5, 0.0), up=(0.0, 1.0, 0.0), fov=60.0),
    "mixture": dict(pos=(5.0, 7.0, 5.0), lookAt=(5.0, 0.0, 5.0), up=(0.0, 0.0, 1.0), fov=60.0),
    "boxes": dict(pos=(5.0, 16.0, 5.0), lookAt=(5.0, 0.0, 5.0), up=(0.0, 0.0, 1.0), fov=60.0),
}


def listed():
    return [
        # The smallest rebuild: a prop of a thousand triangles, where launches and latency are everything.
        {"name": "build_small", "kind": "build", "scene": "uniform", "n": 1000, "bits": 30, "topology": "refCompat"},
        # The large single scene of the benchmark, 21 bits per axis.
        {"name": "build_large", "kind": "build", "scene": "mixture", "n": 4194304, "bits": 63, "topology": "karras"},
        # The combined stress scene, the largest build: half boxes, half mixture.
        {"name": "build_stress", "kind": "build", "scene": "boxes", "n": 33554432, "bits": 63, "topology": "karras"},
        # The small configuration: build and ten plain iterations at 1% (41 items per chunk: latency of short chunks).
        {"name": "optimize_small", "kind": "optimize", "scene": "uniform", "n": 65536, "bits": 30,
         "topology": "refCompat", "iterations": 10, "learned": False},
        # The large scene with the plain inefficiency measure, the reference's own method.
        {"name": "optimize_large", "kind": "optimize", "scene": "mixture", "n": 4194304, "bits": 63,
         "topology": "karras", "iterations": 4, "learned": False},
        # The headline: the large scene with the learned scorer alternating with plain iterations.
        {"name": "optimize_learned", "kind": "optimize", "scene": "mixture", "n": 4194304, "bits": 63,
         "topology": "karras", "iterations": 5, "learned": True},
        # The small configuration's picture, straight on the node array (the tracer command's path).
        {"name": "trace_preview", "kind": "image", "scene": "uniform", "n": 65536, "bits": 30, "topology": "refCompat",
         "iterations": 10, "width": 512, "height": 512, "prepared": False, "bounce": False},
        # One frame of the large scene: records of the tree, primary rays and one diffuse bounce per hit.
        {"name": "trace_frame", "kind": "image", "scene": "mixture", "n": 4194304, "bits": 63, "topology": "karras",
         "iterations": 2, "width": 1920, "height": 1080, "prepared": True, "bounce": True},
        # The largest batch of incoherent rays of the stress test on its prepared tree.
        {"name": "trace_rays", "kind": "rays", "scene": "boxes", "n": 33554432, "bits": 63, "topology": "karras",
         "iterations": 0, "rays": 4194304},
        # 256 meshes of log-uniform size through the whole pipeline: build, iterations, random rays.
        {"name": "batch_meshes", "kind": "batch", "meshes": 256, "lo": 1024, "hi": 524288, "iterations": 8,
         "rays_per_mesh": 65536},
        # One training scene of the scorer: rows and realised gains of every inner node, every fourth iteration.
        {"name": "log_pairs", "kind": "log", "scene": "uniform", "n": 65536, "bits": 30, "topology": "refCompat",
         "iterations": 8, "every": 4},
        # Steps of the scorer's training at its batch size (the configuration runs 20,000 of them).
        {"name": "train_scorer", "kind": "train", "rows": 1048576, "batch": 8192, "steps": 400},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "build", "optimize", "optimize", "image", "rays", "batch", "log", "train"])
    if kind == "train":
        return {"kind": "train", "rows": _log_uniform(rng, 20000, 2000000), "batch": _log_uniform(rng, 500, 8192),
                "steps": rng.randint(50, 400)}
    if kind == "batch":
        lo = _log_uniform(rng, 500, 3000)
        return {"kind": "batch", "meshes": _log_uniform(rng, 4, 256), "lo": lo, "hi": lo * rng.randint(4, 100),
                "iterations": rng.randint(1, 8), "rays_per_mesh": _log_uniform(rng, 1000, 65536)}
    scene = rng.choice(["uniform", "mixture", "boxes"])
    bits, topology = rng.choice([(30, "refCompat"), (30, "karras"), (63, "refCompat"), (63, "karras")])
    base = {"scene": scene, "bits": bits, "topology": topology}
    if kind == "build":
        return {"kind": kind, **base, "n": _log_uniform(rng, 500, 33554432)}
    if kind == "optimize":
        return {"kind": kind, **base, "n": _log_uniform(rng, 8000, 4194304), "iterations": rng.randint(1, 6),
                "learned": rng.random() < 0.4}
    if kind == "log":
        return {"kind": kind, **base, "n": _log_uniform(rng, 8000, 80000), "iterations": rng.randint(2, 9),
                "every": rng.choice([2, 4, 8])}
    if kind == "rays":
        return {"kind": kind, **base, "n": _log_uniform(rng, 10000, 33554432), "iterations": rng.randint(0, 2),
                "rays": _log_uniform(rng, 2000, 4194304)}
    return {"kind": kind, **base, "n": _log_uniform(rng, 10000, 4194304), "iterations": rng.randint(0, 4),
            "width": rng.randint(100, 1920), "height": rng.randint(100, 1080), "prepared": rng.random() < 0.7,
            "bounce": rng.random() < 0.5}


# ---- scenes ---------------------------------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device="cuda")


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device="cuda")


def _mixture(g, n, clusters):
    means = _rand(g, clusters, 3) * 10.0
    sigma = torch.exp(math.log(0.05) + _rand(g, clusters) * math.log(0.8 / 0.05))
    comp = torch.randint(0, clusters, (n,), generator=g, device="cuda")
    centre = means[comp] + _randn(g, n, 3) * sigma[comp, None]
    return centre[:, None, :] + 0.01 * _randn(g, n, 3, 3)


def _ground(cells):
    t = torch.linspace(0.0, 10.0, cells + 1, dtype=torch.float64, device="cuda").float()
    x0, z0 = torch.meshgrid(t[:-1], t[:-1], indexing="ij")
    x1, z1 = torch.meshgrid(t[1:], t[1:], indexing="ij")
    x0, z0, x1, z1 = (a.reshape(-1) for a in (x0, z0, x1, z1))
    y = torch.zeros_like(x0)

    def tri(*corners):
        return torch.stack([torch.stack([x, y, z], 1) for x, z in corners], 1)

    return torch.cat([tri((x0, z0), (x1, z0), (x1, z1)), tri((x0, z0), (x1, z1), (x0, z1))])


def _boxes(g, boxes, cells):
    t = torch.linspace(-1.0, 1.0, cells + 1, device="cuda")
    u0, v0 = (a.reshape(-1) for a in torch.meshgrid(t[:-1], t[:-1], indexing="ij"))
    u1, v1 = (a.reshape(-1) for a in torch.meshgrid(t[1:], t[1:], indexing="ij"))
    parts = []
    for axis in range(3):
        others = [k for k in range(3) if k != axis]
        for side in (-1.0, 1.0):
            for corners in (((u0, v0), (u1, v0), (u1, v1)), ((u0, v0), (u1, v1), (u0, v1))):
                tri = torch.empty((u0.shape[0], 3, 3), device="cuda")
                for c, (u, v) in enumerate(corners):
                    tri[:, c, axis] = side
                    tri[:, c, others[0]] = u
                    tri[:, c, others[1]] = v
                parts.append(tri)
    cube = torch.cat(parts)
    q = _randn(g, boxes, 4)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    rot = torch.stack([
        torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)], -1),
        torch.stack([2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)], -1),
        torch.stack([2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1)], 1)
    half = 0.1 + 0.5 * _rand(g, boxes, 3)
    centre = 10.0 * _rand(g, boxes, 3)
    local = (cube[None] * half[:, None, None, :]).reshape(boxes, -1, 3)
    # sums of three products written out: no matrix library decides their order
    out = torch.stack([sum(local[:, :, k] * rot[:, None, j, k] for k in range(3)) for j in range(3)], -1)
    return (out + centre[:, None, :]).reshape(-1, 3, 3)


def _mesh(scene, n, seed):
    """A triangle soup (vertices [3n, 3] float32, faces [n, 3] int32) of about the scene's make-up: exactly n faces."""
    g = _generator(seed)
    if scene == "uniform":
        tri = _rand(g, n, 1, 3) + 0.004 * _randn(g, n, 3, 3)
    elif scene == "mixture":  # a quarter ground grid, the rest a mixture of 64 clusters
        ground = _ground(max(1, int(math.sqrt(n / 8.0))))
        tri = torch.cat([_mixture(g, n - ground.shape[0], 64), ground])
    else:  # half boxes (512 of them where there is room), half a mixture of 256 clusters
        count = max(1, min(512, n // 200))
        cells = max(1, int(math.sqrt(n / (24.0 * count))))
        boxes = _boxes(g, count, cells)
        tri = torch.cat([_mixture(g, n - boxes.shape[0], 256), boxes])
    faces = torch.arange(3 * n, dtype=torch.int32, device="cuda").reshape(n, 3)
    return tri.reshape(-1, 3).contiguous(), faces


def _rays(vert, n, seed):
    """Origins uniform in the mesh's box, directions uniform on the sphere."""
    g = _generator(seed + 7919)
    lo, hi = vert.amin(0), vert.amax(0)
    org = lo + _rand(g, n, 3) * (hi - lo)
    d = _randn(g, n, 3)
    return org, d / d.norm(dim=1, keepdim=True)


def _scorer(seed):
    """A scorer trained for a moment on one small scene of the mixture's make-up."""
    n = 32768
    v, f = _mesh("mixture", n, seed + 104729)
    nodes = api.LBVH(n, 63, "karras").build(v, f)
    data = learned.log_pairs([nodes], iterations=3, every=2, seed=seed)
    return learned.train(data, steps=300, seed=seed)[0]


def _training_rows(case, seed):
    """Rows like the logged ones: 14 features of the rows' ranges and ten zeros, BF16; targets in the log scale
    of the realised gains."""
    g = _generator(seed)
    m = case["rows"]
    x = torch.zeros((m, 24), device="cuda")
    x[:, 0] = -12.0 + 4.0 * _randn(g, m)
    x[:, 1:4] = 0.2 + 0.8 * _rand(g, m, 3)
    x[:, 4] = 0.5 + _rand(g, m)
    x[:, 5:7] = 12.0 * _rand(g, m, 2) ** 2
    x[:, 7] = -14.0 + 4.0 * _randn(g, m)
    x[:, 8:10] = 1.0 + 2.0 * _randn(g, m, 2)
    x[:, 10:14] = _rand(g, m, 4)
    t = torch.sin(x[:, 0] * 0.5) + 2.0 * x[:, 3] * x[:, 10] - 0.2 * x[:, 8] + 0.5 * _randn(g, m)
    return x.to(torch.bfloat16), t


# ---- the cases ------------------------------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, t = _training_rows(case, seed)
        return {"case": case, "seed": seed, "data": learned.TrainingSet(x, t)}
    if kind == "batch":
        # the log-uniform sizes at their quantiles (so that every seed has the same total), in the seed's order
        q = (np.arange(case["meshes"]) + 0.5) / case["meshes"]
        counts = np.exp(math.log(case["lo"]) + q * math.log(case["hi"] / case["lo"])).astype(np.int64)
        counts = np.random.default_rng(seed).permutation(counts)
        dev = _generator(seed)
        mesh = torch.repeat_interleave(torch.arange(case["meshes"], device="cuda"), torch.from_numpy(counts).cuda())
        total = int(counts.sum())
        # per mesh 1 to 16 clusters in the unit cube, sigma log-uniform in [0.005, 0.08]
        clusters = torch.randint(1, 17, (case["meshes"],), generator=dev, device="cuda")
        comp = (_rand(dev, total) * clusters[mesh]).long().clamp_(max=15)
        comp = torch.minimum(comp, clusters[mesh] - 1) + 16 * mesh
        means = _rand(dev, 16 * case["meshes"], 3)
        sigma = torch.exp(math.log(0.005) + _rand(dev, 16 * case["meshes"]) * math.log(0.08 / 0.005))
        centre = means[comp] + _randn(dev, total, 3) * sigma[comp, None]
        vert = (centre[:, None, :] + 0.004 * _randn(dev, total, 3, 3)).reshape(-1, 3).contiguous()
        faces = torch.arange(3 * total, dtype=torch.int32, device="cuda").reshape(total, 3)
        batch = api.Batch(counts.astype(np.uint32))
        hits = torch.empty(case["meshes"] * case["rays_per_mesh"], dtype=torch.int64, device="cuda")
        return {"case": case, "seed": seed, "vert": vert, "faces": faces, "batch": batch,
                "nodes": batch.empty_nodes(), "hits": hits}
    vert, faces = _mesh(case["scene"], case["n"], seed)
    builder = api.LBVH(case["n"], case["bits"], case["topology"])
    state = {"case": case, "seed": seed, "vert": vert, "faces": faces, "builder": builder}
    if kind == "build":
        return state
    state["nodes"] = nodes = builder.build(vert, faces)
    if kind == "log":
        return state
    if kind == "optimize":
        state["opt"] = opt = api.Bittner13GPU(nodes)
        if case["learned"]:
            opt.set_scorer(_scorer(seed))  # alternating with plain iterations
        return state
    if case["iterations"]:
        opt = api.Bittner13GPU(nodes)
        opt.run(case["iterations"])
        torch.cuda.synchronize()
        opt.close()
    del state["builder"]
    builder.close()
    if kind == "rays":
        state["org"], state["dir"] = _rays(vert, case["rays"], seed)
        state["tracer"] = api.Tracer(nodes.shape[0]).update(nodes)
        return state
    state["camera"] = dict(CAMERAS[case["scene"]], width=case["width"], height=case["height"])
    if case["prepared"]:
        state["tracer"] = api.Tracer(nodes.shape[0])
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "build":
        return state["builder"].build(state["vert"], state["faces"])
    if kind == "optimize":
        nodes, opt = state["nodes"], state["opt"]
        state["builder"].build(state["vert"], state["faces"], nodes)
        opt.iteration = 0
        opt.run(case["iterations"])
        return nodes
    if kind == "image":
        nodes, vert, faces, camera = state["nodes"], state["vert"], state["faces"], state["camera"]
        if not case["prepared"]:
            img, hits = api.trace_image(nodes, vert, faces, camera)
            if not case["bounce"]:
                return img, hits
            return img, hits, api.trace_bounce(nodes, vert, faces, camera, hits, seed=state["seed"])[0]
        tracer = state["tracer"].update(nodes)
        img, hits = tracer.trace_image(vert, faces, camera)
        if not case["bounce"]:
            return img, hits
        return img, hits, tracer.trace_bounce(vert, faces, camera, hits, seed=state["seed"])[0]
    if kind == "rays":
        return state["tracer"].trace_rays(state["vert"], state["faces"], state["org"], state["dir"])
    if kind == "batch":
        state["batch"].run(state["vert"], state["faces"], state["nodes"], case["iterations"], case["rays_per_mesh"],
                           state["hits"], seed=state["seed"])
        return state["nodes"], state["hits"]
    if kind == "log":
        state["builder"].build(state["vert"], state["faces"], state["nodes"])
        data = learned.log_pairs([state["nodes"]], iterations=case["iterations"], every=case["every"])
        return data.x, data.t, state["nodes"]
    scorer, history, _ = learned.train(state["data"], steps=case["steps"], batch=case["batch"], seed=state["seed"])
    return scorer.params(), history


# ---- what a pass cannot do without ----------------------------------------------------------------------------


def _build_work(n):
    # faces and vertices read once, every node written once
    return 48 * n + 48 * (2 * n - 1)


def _optimize_work(n, iterations):
    # Per iteration every inner node's area and its children's decide the selection (12 bytes each); each of the 1%
    # reinserted nodes walks at least two root-to-leaf paths of node boxes and rewrites about ten nodes.
    items = 0.02 * n
    depth = math.log2(max(n, 2))
    return iterations * (12 * n + items * (2 * depth * 48 + 10 * 48))


def _ray_work(rays, n, io):
    # the ray and its hit, and of the tree and the triangles at most once what one path per ray needs
    depth = math.log2(max(n, 2))
    return rays * io + min(48 * (2 * n - 1) + 48 * n, rays * (depth * 48 + 48)), rays * depth * 2 * 25


def work(case):
    kind = case["kind"]
    if kind == "build":
        return {"bytes": _build_work(case["n"]), "flops": 0}
    if kind == "optimize":
        return {"bytes": _build_work(case["n"]) + _optimize_work(case["n"], case["iterations"]), "flops": 0}
    if kind == "image":
        pixels = case["width"] * case["height"]
        nbytes, flops = _ray_work(pixels, case["n"], 12)
        if case["bounce"]:
            more, moreflops = _ray_work(pixels, case["n"], 16)
            nbytes, flops = nbytes + more, flops + moreflops
        return {"bytes": nbytes, "flops": flops}
    if kind == "rays":
        nbytes, flops = _ray_work(case["rays"], case["n"], 32)
        return {"bytes": nbytes, "flops": flops}
    if kind == "batch":
        # the mean of the log-uniform counts
        n = case["meshes"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        nbytes, flops = _ray_work(case["meshes"] * case["rays_per_mesh"], n, 8)
        return {"bytes": nbytes + _build_work(n) + _optimize_work(n, case["iterations"]), "flops": flops}
    if kind == "log":
        # an optimizer run, and per logged node two searches, its row and its target
        logs = -(-case["iterations"] // case["every"])
        per = 2 * math.log2(case["n"]) * 48 + 52
        return {"bytes": _build_work(case["n"]) + _optimize_work(case["n"], case["iterations"]) + logs * case["n"] * per,
                "flops": 0}
    # forward and backward of 24 -> 64 -> 64 -> 1: three products per layer but the first's input gradient
    per_row = 2 * (24 * 64 * 2 + 64 * 64 * 3 + 64 * 3)
    rows = case["batch"] * case["steps"]
    return {"bytes": rows * 52 + case["steps"] * 5825 * 4 * 6, "flops": rows * per_row}


# ---- the computed numbers in 64 bits ----------------------------------------------------------------------------


def _mix(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def exact(case, seed):
    """Only training has outputs that are computed numbers with a value of their own: trees, hits and pixels are whole
    numbers and bytes, and logged rows and gains belong to the tree that the optimizer made."""
    if case["kind"] != "train":
        return None
    x, t = _training_rows(case, seed)
    x, t = x.double(), t.double()

    def bf(v):  # weights, inputs and activations of this network are BF16 numbers
        return v.float().to(torch.bfloat16).double()

    # the scorer's documented start: SplitMix64 of its seed (0), uniform in +-sqrt(6 / fan-in), the last layer a tenth
    with np.errstate(over="ignore"):
        i = np.arange(1, 24 * 64 + 64 * 64 + 64 + 1, dtype=np.uint64)
        u = (_mix(i * np.uint64(0x9E3779B97F4A7C15)) >> np.uint64(40)).astype(np.float64) / 2.0**24 * 2.0 - 1.0
    p = [torch.from_numpy(a.astype(np.float32)).double().cuda() for a in (
        u[: 24 * 64].reshape(64, 24) * math.sqrt(6 / 24), np.zeros(64),
        u[24 * 64: 24 * 64 + 64 * 64].reshape(64, 64) * math.sqrt(6 / 64), np.zeros(64),
        u[-64:] * math.sqrt(6 / 64) * 0.1, np.zeros(1))]
    m, v = [torch.zeros_like(a) for a in p], [torch.zeros_like(a) for a in p]
    c = math.sqrt(2 / math.pi)

    def gelu(z):
        return 0.5 * z * (1 + torch.tanh(c * (z + 0.044715 * z**3)))

    def slope(z):
        th = torch.tanh(c * (z + 0.044715 * z**3))
        return 0.5 * (1 + th) + 0.5 * z * (1 - th * th) * c * (1 + 3 * 0.044715 * z * z)

    history = []
    for step in range(1, case["steps"] + 1):
        with np.errstate(over="ignore"):  # the batch: SplitMix64 of (seed, step, position), modulo the rows
            k = np.uint64(step) * np.uint64(case["batch"]) + np.arange(1, case["batch"] + 1, dtype=np.uint64)
            row = _mix(np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * k) % np.uint64(case["rows"])
        row = torch.from_numpy(row.astype(np.int64)).cuda()
        a0, y0 = x[row], t[row]
        w1, b1, w2, b2, w3, b3 = (bf(a) for a in p)
        z1 = a0 @ w1.T + b1
        a1 = bf(gelu(z1))
        z2 = a1 @ w2.T + b2
        a2 = bf(gelu(z2))
        diff = a2 @ w3 + b3 - y0
        history.append((diff * diff).mean())
        dy = 2 * diff / case["batch"]
        d2 = dy[:, None] * w3 * slope(z2)
        d1 = (d2 @ w2) * slope(z1)
        grads = [d1.T @ a0, d1.sum(0), d2.T @ a1, d2.sum(0), a2.T @ dy, dy.sum().reshape(1)]
        for k, g in enumerate(grads):
            m[k] = 0.9 * m[k] + 0.1 * g
            v[k] = 0.999 * v[k] + 0.001 * g * g
            if k % 2 == 0:  # decoupled decay on weights only
                p[k] = p[k] - 1e-3 * 1e-4 * p[k]
            p[k] = p[k] - 1e-3 * (m[k] / (1 - 0.9**step)) / (torch.sqrt(v[k] / (1 - 0.999**step)) + 1e-8)
    return torch.cat([a.reshape(-1) for a in p]), torch.stack(history)
