"""The work this framework is timed on: microenvironment steps of single meshes from the smallest to
the headline size, a population that moves every step, a batch of uneven meshes, and the learned
surrogate's prediction and gradients.

A case is a dict of plain values.  ``prepare`` builds what a program holds before the call, ``run``
is one pass through the public entry points, ``exact`` restates the pass in float64 torch.
"""

import math

import numpy as np
import torch

from parabiofvm_b200 import Batch, Solver

VOXEL = 20  # um, the edge of a voxel in every workload

_stream = None


def stream():
    """One stream for all of a program's solvers: passes follow one another in the order of the calls."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


class _View:
    """A solver's resident buffer, for torch.as_tensor; the tensor keeps the solver, and so the buffer, alive."""

    def __init__(self, solver, pointer, count):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (pointer, False), "version": 3,
                                         "strides": None}


def listed():
    return [
        # the smallest mesh a model is built and debugged on, stepped one call at a time: launches and latency
        step("step-20x1", 20, 20, 20, S=1, agents=100, steps=1),
        # the CPU-runnable configuration: 50 cubed, four substrates, ten steps (one rebinning) a call
        step("step-50x4", 50, 50, 50, S=4, agents=5000, steps=10),
        # a tissue slice: a 2-D mesh with three substrates
        step("step-2d-400x300x3", 400, 300, 1, S=3, agents=2000, steps=10),
        # sizes that divide nothing, five substrates, a vessel's worth of interior Dirichlet voxels
        step("step-97x61x83x5", 97, 61, 83, S=5, agents=3000, steps=10, interior=0.01),
        # the mesh the surrogate is trained for, with clustered agents
        step("step-128x4", 128, 128, 128, S=4, agents=200_000, steps=10, clustered=True, boundary=False),
        # the reference driver's shape: 250 cubed, four substrates, two million agents, 5 minutes a step
        step("step-250x4", 250, 250, 250, S=4, agents=2_000_000, steps=10, dt=5.0, boundary=False),
        # the headline configuration
        step("step-320x16", 320, 320, 320, S=16, agents=1_000_000, steps=10, clustered=True, interior=0.01),
        # a long vessel: lines of more than 512 voxels
        step("step-640x160x128x4", 640, 160, 128, S=4, agents=50_000, steps=10),
        # a model whose agents move: positions in, one step with rebinning, internalized amounts out
        step("move-100x4", 100, 100, 100, S=4, agents=50_000, steps=1, clustered=True, moving=True),
        # a parameter sweep: uneven meshes stepped together
        {"name": "batch-32", "kind": "batch", "meshes": 32, "edge_min": 24, "edge_max": 96, "S_max": 8,
         "agents_max": 20_000, "steps": 10},
        # the learned surrogate: one macro-step of 16 steps, and one training batch's gradients
        {"name": "infer-128x4", "kind": "infer", "X": 128, "Y": 128, "Z": 128, "S": 4, "batch": 1, "agents": 100_000},
        {"name": "gradients-128x4", "kind": "gradients", "X": 128, "Y": 128, "Z": 128, "S": 4, "batch": 2,
         "agents": 100_000},
    ]


def step(name, X, Y, Z, S, agents, steps, dt=0.01, clustered=False, boundary=True, interior=0.0, moving=False):
    c = {"kind": "step", "X": X, "Y": Y, "Z": Z, "S": S, "agents": agents, "steps": steps, "dt": dt,
         "clustered": clustered, "boundary": boundary, "interior": interior, "moving": moving}
    return dict(c, name=name) if name else c


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["slice", "long", "moving", "moving", "batch", "infer", "gradients"])
    if kind == "batch":
        lo = rng.randint(16, 48)
        return {"kind": "batch", "meshes": rng.randint(4, 32), "edge_min": lo, "edge_max": lo + rng.randint(0, 48),
                "S_max": rng.randint(1, 8), "agents_max": _log_int(rng, 100, 20_000), "steps": rng.choice([1, 10])}
    if kind in ("infer", "gradients"):
        c = {"kind": kind, "X": rng.choice([128, 128, 130, 160, 192, 256]), "Y": _log_int(rng, 24, 128),
             "Z": _log_int(rng, 24, 128), "S": rng.randint(1, 10), "batch": rng.randint(1, 2),
             "agents": _log_int(rng, 1000, 100_000)}
        return c
    dt = rng.choice([0.01, 0.01, 0.1, 5.0])
    more = {"dt": dt, "clustered": rng.random() < 0.5, "boundary": rng.random() < 0.6,
            "interior": rng.choice([0.0, 0.0, 0.01])}
    if kind == "slice":
        X, Y = _log_int(rng, 20, 1000), _log_int(rng, 20, 1000)
        return step(None, X, Y, 1, S=rng.randint(1, 8), agents=_log_int(rng, 50, max(100, X * Y // 20)), steps=10, **more)
    if kind == "long":
        n = [_log_int(rng, 520, 1024), _log_int(rng, 16, 128), _log_int(rng, 16, 128)]
        rng.shuffle(n)
        return step(None, *n, S=rng.randint(1, 8), agents=_log_int(rng, 1000, 100_000), steps=10, **more)
    if kind == "moving":
        n = [_log_int(rng, 16, 160) for _ in range(3)]
        S = rng.randint(1, 8)
        return step(None, *n, S=S, agents=_log_int(rng, 50, 100_000), steps=1, moving=True, **more)
    e = _log_int(rng, 12, 250)
    n = [max(5, min(320, int(e * rng.uniform(0.7, 1.4)))) for _ in range(3)]
    S = rng.choice([1, 2, 3, 4, 5, 6, 8, 12, 16])
    V = n[0] * n[1] * n[2]
    agents = _log_int(rng, 20, min(1_000_000, max(100, V // 10)))
    return step(None, *n, S=S, agents=agents, steps=rng.choice([1, 10]), **more)


# ------------------------------------------------------------------------------------------------
# inputs, from the seed alone


def _generator(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed))
    return g


def _positions(g, n, dims, agents, clustered, device="cuda"):
    """Agent positions inside the mesh: uniform, or in 32 Gaussian clusters of 200 um (less in small meshes)."""
    L = torch.tensor([float(v * VOXEL) for v in n[:dims]], device=device)
    if clustered:
        centres = torch.rand(32, dims, generator=g, device=device) * L
        k = torch.randint(0, 32, (agents,), generator=g, device=device)
        sigma = torch.clamp(L / 8, max=200.0)
        p = centres[k] + torch.randn(agents, dims, generator=g, device=device) * sigma
        inside = ((p >= 0) & (p < L)).all(dim=1, keepdim=True)
        p = torch.where(inside, p, torch.rand(agents, dims, generator=g, device=device) * L)
    else:
        p = torch.rand(agents, dims, generator=g, device=device) * L
    return torch.minimum(p, torch.nextafter(L, torch.zeros_like(L)))


def _mesh_inputs(c, seed):
    """A microenvironment: coefficients log-uniform in [1e3, 1e5] um^2/min, decay U(0.01, 1)/min, field
    U(0, 1), agents of volume 1000 with secretion U(0, 10), saturation and uptake U(0, 1), the value 1 of
    substrate 0 on the faces and U(0, 1) in the interior Dirichlet voxels.  With dt in minutes the
    agents' rates are per 0.01 / dt of that, so a step moves the same share of a voxel."""
    n = (c["X"], c["Y"], c["Z"])
    dims = 2 if n[2] == 1 else 3
    S, A = c["S"], c["agents"]
    V = n[0] * n[1] * n[2]
    g = _generator(seed)

    def u(*shape):
        return torch.rand(*shape, generator=g, device="cuda")

    d = {"n": n, "dims": dims, "S": S, "dt": float(np.float32(c["dt"]))}
    d["D"] = torch.exp(math.log(1e3) + (math.log(1e5) - math.log(1e3)) * u(S)).cpu().numpy()
    d["decay"] = (0.01 + 0.99 * u(S)).cpu().numpy()
    d["field"] = u(V, S)
    rate = 0.01 / c["dt"]
    d["agents"] = {"sec": 10 * rate * u(A, S), "sat": u(A, S), "upt": rate * u(A, S),
                   "nex": torch.zeros(A, S, device="cuda"), "int": torch.zeros(A, S, device="cuda"), "frac": u(A, S),
                   "vol": torch.full((A,), 1000.0, device="cuda"),
                   "pos": _positions(g, n, dims, A, c["clustered"])}
    if c.get("moving"):
        d["moved"] = _positions(g, n, dims, A, c["clustered"])
    d["boundary"] = bool(c["boundary"])
    d["interior"] = None
    inner = [max(v - 2, 0) for v in n[:dims]]
    k = int(round(c["interior"] * math.prod(inner)))
    if k:
        pick = torch.randperm(math.prod(inner), generator=g, device="cuda")[:k]
        at = []
        for v in inner:
            at.append(pick % v + 1)
            pick = pick // v
        d["interior"] = (torch.stack(at, dim=1).to(torch.int32), u(k, S))
    return d


def _solver(d):
    dims, n, S = d["dims"], d["n"], d["S"]
    s = Solver(dims, (0,) * 3, tuple(v * VOXEL for v in n[:dims]), (VOXEL,) * 3, d["D"], d["decay"], d["dt"],
               compute_internalized=True)
    s.set_stream(stream().cuda_stream)
    if d["boundary"]:
        vals, conds = np.zeros(S, np.float32), np.zeros(S, np.uint8)
        vals[0], conds[0] = 1.0, 1
        for axis in range(dims):
            s.set_boundary_dirichlet(axis, False, vals, conds)
            s.set_boundary_dirichlet(axis, True, vals, conds)
    if d["interior"] is not None:
        at, v = d["interior"]
        s.set_interior_dirichlet(at.cpu().numpy(), v.cpu().numpy(), np.ones(tuple(v.shape), np.uint8))
    torch.cuda.synchronize()
    s.store_densities_device(d["field"])
    a = {k: v.cpu().numpy() for k, v in d["agents"].items()}
    s.store_agents(a["sec"], a["sat"], a["upt"], a["nex"], a["int"], a["frac"], a["vol"], a["pos"])
    s.synchronize()
    return s


def _views(s):
    return {"densities": torch.as_tensor(_View(s, *s.device_densities()), device="cuda"),
            "gradients": torch.as_tensor(_View(s, *s.device_gradients()), device="cuda")}


def _batch_members(c, seed):
    """The meshes of a batch: cubes with U{edge_min..edge_max} voxels an edge, U{1..S_max} substrates and
    up to agents_max clustered agents.  Sizes do not depend on the inputs' seed."""
    r = np.random.default_rng(20261204)
    members = []
    for i in range(c["meshes"]):
        e, S = int(r.integers(c["edge_min"], c["edge_max"] + 1)), int(r.integers(1, c["S_max"] + 1))
        A = int(r.integers(min(100, c["agents_max"]), c["agents_max"] + 1))
        members.append((step(None, e, e, e, S=S, agents=A, steps=c["steps"], clustered=True), seed * 64 + i))
    return members


LAYERS, TAPS, WIDTH = 10, 27, 32
LAYER_PARAMETERS = TAPS * WIDTH * WIDTH + WIDTH


def _surrogate_inputs(c, seed):
    """Fields of 8 Gaussian bumps per substrate and the secretion terms of uniform agents, as the network
    is trained on; the target is the field after 16 steps of decay and light smoothing."""
    X, Y, Z, S, B = c["X"], c["Y"], c["Z"], c["S"], c["batch"]
    g = _generator(seed)

    def u(*shape):
        return torch.rand(*shape, generator=g, device="cuda")

    centre, width, height = u(3, B, S, 8), 4 + 12 * u(B, S, 8), u(B, S, 8)
    axes = []
    for d, n in enumerate((X, Y, Z)):
        i = torch.arange(n, device="cuda", dtype=torch.float32).view(-1, 1, 1, 1)
        axes.append(torch.exp(-0.5 * ((i - centre[d] * n) / width) ** 2))
    field = torch.einsum("xbsk,ybsk,zbsk,bsk->bzyxs", *axes, height).contiguous()
    sources, sinks = torch.zeros(B, Z * Y * X, S, device="cuda"), torch.zeros(B, Z * Y * X, S, device="cuda")
    A = c["agents"]
    for b in range(B):
        at = torch.randint(0, X * Y * Z, (A,), generator=g, device="cuda")
        sec, sat, upt = 10 * u(A, S), u(A, S), u(A, S)
        # one agent's terms in a voxel that several share: the last written, whatever the order of a sum
        first = torch.zeros(X * Y * Z, dtype=torch.int64, device="cuda").scatter_reduce_(
            0, at, torch.arange(A, device="cuda"), "amax")[at]
        sources[b, at] = (sec * sat * 0.01 / 8)[first]
        sinks[b, at] = ((upt + sec) * 0.01 / 8)[first]
    decay = 0.01 + 0.99 * u(S)
    near = torch.nn.functional.avg_pool3d(field.permute(0, 4, 1, 2, 3), 3, 1, 1, count_include_pad=False)
    target = ((0.5 * field + 0.5 * near.permute(0, 2, 3, 4, 1)) * torch.exp(-0.16 * decay)).contiguous()
    # He-uniform weights; the layers that end a residual block and the projection start small
    p = torch.zeros(LAYERS, LAYER_PARAMETERS, device="cuda")
    w = (2 * u(LAYERS, TAPS, WIDTH, WIDTH) - 1) * math.sqrt(6 / (TAPS * WIDTH))
    for layer in (2, 4, 6, 8, 9):
        w[layer] *= 0.3
    p[:, :TAPS * WIDTH * WIDTH] = w.reshape(LAYERS, -1)
    p[:, TAPS * WIDTH * WIDTH:] = 0.02 * (2 * u(LAYERS, WIDTH) - 1)
    return {"field": field.view(B, -1, S), "sources": sources, "sinks": sinks, "target": target.view(B, -1, S),
            "parameters": p.reshape(-1)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        solvers = [_solver(_mesh_inputs(c, k)) for c, k in _batch_members(case, seed)]
        return {"case": case, "solvers": solvers, "batch": Batch(solvers), "views": [_views(s) for s in solvers],
                "step": 0}
    if kind in ("infer", "gradients"):
        from parabiofvm_b200.surrogate import Surrogate

        d = _surrogate_inputs(case, seed)
        net = Surrogate((case["X"], case["Y"], case["Z"]), case["S"], max_batch=case["batch"], stream=stream())
        net.load(d.pop("parameters").cpu().numpy())
        torch.cuda.synchronize()
        return dict(d, case=case, net=net, prediction=torch.empty_like(d["field"]))
    d = _mesh_inputs(case, seed)
    s = _solver(d)
    state = {"case": case, "solver": s, "views": _views(s), "step": 0}
    if case["moving"]:
        state["positions"] = d["moved"].cpu().pin_memory().numpy()
        state["internalized"] = torch.empty(case["agents"] * case["S"], pin_memory=True).numpy()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "infer":
        state["net"].infer(state["field"], state["sources"], state["sinks"], state["prediction"])
        return state["prediction"]
    if kind == "gradients":
        net = state["net"]
        loss = net.gradients(state["field"], state["sources"], state["sinks"], state["target"], state["prediction"])
        return {"loss": loss, "prediction": state["prediction"], "gradients": net.load_gradients()}
    first, state["step"] = state["step"], state["step"] + case["steps"]
    if kind == "batch":
        state["batch"].run_steps(case["steps"], first)
        return state["views"]
    s = state["solver"]
    if not case["moving"]:
        s.run_steps(case["steps"], first)
        return state["views"]
    s.store_agent_positions_async(state["positions"])
    s.run_steps(1, 0)
    s.load_internalized_async(state["internalized"])
    return dict(state["views"], internalized=state["internalized"])


def work(case):
    kind = case["kind"]
    if kind in ("infer", "gradients"):
        V = case["X"] * case["Y"] * case["Z"] * case["batch"]
        conv = 2.0 * TAPS * WIDTH * WIDTH * V * LAYERS
        backward = kind == "gradients"
        return {"bytes": 4.0 * V * case["S"] * (5 if backward else 4), "flops": conv * (2.9 if backward else 1.0)}
    if kind == "batch":
        parts = [work(c) for c, _ in _batch_members(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    dims = 2 if case["Z"] == 1 else 3
    VS = case["X"] * case["Y"] * case["Z"] * case["S"]
    A, S = case["agents"], case["S"]
    # a step: the field read and written, the gradients written, the agents' terms and amounts
    step_bytes = VS * (8.0 + 4.0 * dims) + A * S * 20.0
    # a sweep: 3 operations forward and 2 back; the gradient 2 per axis; the update 10 per agent
    step_flops = VS * (5.0 * dims + 2.0 * dims) + A * S * 10.0
    return {"bytes": step_bytes * case["steps"], "flops": step_flops * case["steps"]}


# ------------------------------------------------------------------------------------------------
# the same passes in float64


def _along(u, axis, b, c):
    """Thomas solve of every line along dimension `axis` of u [Z][Y][X][S]; b [n][S] reciprocal pivots."""
    w = u.movedim(axis, 0).contiguous()
    n = w.shape[0]
    for i in range(1, n):
        w[i].addcmul_(w[i - 1], (c * b[i - 1]).expand_as(w[i]), value=-1)
    w[n - 1].mul_(b[n - 1])
    for i in range(n - 2, -1, -1):
        w[i].addcmul_(w[i + 1], c.expand_as(w[i]), value=-1).mul_(b[i])
    u.copy_(w.movedim(0, axis))


def _exact_steps(d, steps, moving=False):
    dims, S, n, dt = d["dims"], d["S"], d["n"], d["dt"]
    D = torch.tensor(d["D"], dtype=torch.float64, device="cuda")
    lam = torch.tensor(d["decay"], dtype=torch.float64, device="cuda")
    u = d.pop("field").double().view(n[2], n[1], n[0], S)
    flat = u.view(-1, S)
    tables = []
    for axis in range(dims):
        k = dt * D / (VOXEL * VOXEL)
        diag = [1 + lam * dt / dims + (1 if i in (0, n[axis] - 1) else 2) * k for i in range(n[axis])]
        b = [1 / diag[0]]
        for i in range(1, n[axis]):
            b.append(1 / (diag[i] - k * k * b[i - 1]))
        tables.append((torch.stack(b), -k))

    def overwrite():
        if d["boundary"]:
            for axis in range(dims):
                for end in (0, n[axis] - 1):
                    u.select(2 - axis, end)[..., 0] = 1.0
        if d["interior"] is not None:
            at, v = d["interior"]
            at = at.long()
            index = at[:, 0] + n[0] * (at[:, 1] + (n[1] * at[:, 2] if dims == 3 else 0))
            flat[index] = v.double()

    a = d["agents"]
    pos = (d["moved"] if moving else a["pos"]) / float(VOXEL)
    cell = pos.to(torch.int64)
    index = cell[:, 0] + n[0] * (cell[:, 1] + (n[1] * cell[:, 2] if dims == 3 else 0))
    volume = float(VOXEL ** 3)
    sec, sat, upt, nex, vol = (a[k].double() for k in ("sec", "sat", "upt", "nex", "vol"))
    share = dt * vol[:, None] / volume
    num, den, fac = sec * sat * share, (sec + upt) * share, nex * dt / volume
    voxels, slot = torch.unique(index, return_inverse=True)
    sums = [torch.zeros(len(voxels), S, dtype=torch.float64, device="cuda").index_add_(0, slot, t)
            for t in (num, den, fac)]
    inside = a["int"].double()
    for i in range(steps):
        for axis in range(dims):
            overwrite()
            _along(u, 2 - axis, *tables[axis])
        overwrite()
        if i == steps - 1:
            gradients = []
            for axis in range(dims):
                w = u.movedim(2 - axis, 0)
                m = n[axis]
                g = torch.empty_like(u)
                t = g.movedim(2 - axis, 0)
                t[1:m - 1] = (w[2:] - w[:m - 2]) / (2 * VOXEL)
                t[0] = (w[1] - w[0]) / VOXEL
                t[m - 1] = (w[m - 1] - w[m - 2]) / VOXEL
                gradients.append(g)
        at = flat[index]
        inside -= volume * ((num - den * at) / (1 + den) + fac)
        flat[voxels] = (flat[voxels] + sums[0]) / (1 + sums[1]) + sums[2]
    g = torch.stack([t.reshape(-1) for t in gradients], dim=0 if dims == 3 else 1).reshape(-1)
    out = {"densities": u.reshape(-1), "gradients": g}
    if moving:
        out["internalized"] = inside.reshape(-1)
    return out


def _taps():
    for t in range(TAPS):
        yield t, t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1


def _ranges(o, n):
    """Where out[v] reads in[v + o]: the slices of out and of in."""
    return slice(max(0, -o), n - max(0, o)), slice(max(0, o), n + min(0, o))


def _convolve(x, W, b=None):
    out = torch.zeros(*x.shape[:4], W.shape[1], dtype=x.dtype, device=x.device)
    for t, dz, dy, dx in _taps():
        (oz, iz), (oy, iy), (ox, ix) = _ranges(dz, x.shape[1]), _ranges(dy, x.shape[2]), _ranges(dx, x.shape[3])
        out[:, oz, oy, ox] += x[:, iz, iy, ix] @ W[t].T
    return out if b is None else out + b


def _weight_gradient(x, g):
    rows = []
    for t, dz, dy, dx in _taps():
        (oz, iz), (oy, iy), (ox, ix) = _ranges(dz, x.shape[1]), _ranges(dy, x.shape[2]), _ranges(dx, x.shape[3])
        rows.append(g[:, oz, oy, ox].reshape(-1, WIDTH).T @ x[:, iz, iy, ix].reshape(-1, WIDTH))
    return torch.cat([torch.stack(rows).reshape(-1), g.sum(dim=(0, 1, 2, 3))])


def _exact_surrogate(case, seed):
    d = _surrogate_inputs(case, seed)
    B, X, Y, Z, S = case["batch"], case["X"], case["Y"], case["Z"], case["S"]
    shape = (B, Z, Y, X, S)
    field = d["field"].double().view(shape)
    p = d["parameters"].double().view(LAYERS, LAYER_PARAMETERS)
    W = [(v[:-WIDTH].view(TAPS, WIDTH, WIDTH), v[-WIDTH:]) for v in p]
    x = torch.zeros(B, Z, Y, X, WIDTH, dtype=torch.float64, device="cuda")
    x[..., :S] = field
    x[..., S:2 * S] = 16 * d["sources"].double().view(shape)
    x[..., 2 * S:3 * S] = 16 * d["sinks"].double().view(shape)
    h, t = [_convolve(x, *W[0]).relu_()], []
    for k in range(4):
        t.append(_convolve(h[k], *W[2 * k + 1]).relu_())
        h.append(_convolve(t[k], *W[2 * k + 2]) + h[k])
    prediction = field + _convolve(h[4], *W[9])[..., :S]
    if case["kind"] == "infer":
        return prediction.reshape(B, -1, S)
    off = prediction - d["target"].double().view(shape)
    g = torch.zeros(B, Z, Y, X, WIDTH, dtype=torch.float64, device="cuda")
    g[..., :S] = 2 * off / off.numel()

    def back(y, w):
        return _convolve(y, w.flip(0).transpose(1, 2))

    grads = [None] * LAYERS
    grads[9] = _weight_gradient(h[4], g)
    g = back(g, W[9][0])
    for k in range(3, -1, -1):
        grads[2 * k + 2] = _weight_gradient(t[k], g)
        inner = back(g, W[2 * k + 2][0]) * (t[k] > 0)
        grads[2 * k + 1] = _weight_gradient(h[k], inner)
        g = g + back(inner, W[2 * k + 1][0])
    grads[0] = _weight_gradient(x, g * (h[0] > 0))
    return {"loss": float((off ** 2).mean()), "prediction": prediction.reshape(B, -1, S), "gradients": torch.cat(grads)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("infer", "gradients"):
        return _exact_surrogate(case, seed)
    if kind == "batch":
        return [_exact_steps(_mesh_inputs(c, k), case["steps"]) for c, k in _batch_members(case, seed)]
    return _exact_steps(_mesh_inputs(case, seed), case["steps"], case["moving"])
