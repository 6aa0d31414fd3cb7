"""Evaluation workloads of the dipole FMM, as its users run them.

A case names a geometry (`points`, `n`, `targets`, `order`, `depth`), how many
moment states one call carries, and the public entry point it goes through
(`entry`):

  device    DevicePlan.evaluate on CUDA tensors, stream-ordered
  host      DevicePlan.evaluate on pinned host arrays, copies included
  dropin    cdfmm.UniformFmm.evaluate: numpy moments in, numpy results out
  gradient  dipole_field under torch autograd: the field, dL/dmoments and
            dL/dtarget-positions of L = sum w . H
  batch     Batch.launch: independent single-state problems, one graph launch
  cuboid    DevicePlan.evaluate with uniformly magnetised cuboid sources

The inputs are synthetic: seeded points and moments of the distributions the
benchmark of this repository uses.
"""

import math
import os
import sys

import numpy as np
import torch

_PYTHON = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dip-fmm_b200", "python")
if _PYTHON not in sys.path:
    sys.path.insert(0, _PYTHON)

import cdfmm  # noqa: E402
import cdfmm_b200  # noqa: E402

DEFAULTS = {"entry": "device", "points": "uniform", "n": 4096, "targets": 0, "order": 6, "depth": 3, "states": 1,
            "output": "field", "dtype": "float32", "problems": 1}

# Direct sums in FP64 up to this many (target, source) pairs take a few
# seconds on the card; larger cases have no 64-bit answer here.
EXACT_PAIRS = 7.0e10
EXACT_CUBOID_PAIRS = 1.2e9


def _case(**kw):
    return {**DEFAULTS, **kw}


def listed():
    return [
        # A small system relaxed step by step through the drop-in class: the
        # reference's own first configuration, host arrays, latency.
        _case(name="dropin_4k", entry="dropin", n=4096, order=4, depth=3),
        # The smallest device-resident call: a few thousand dipoles of odd
        # count, a handful of states (an odd number), both outputs.
        _case(name="small_states", n=6007, order=5, depth=3, states=3, output="both"),
        # One state on the reference's large single-state configuration.
        _case(name="single_1m", n=1048576, order=6, depth=5, output="both"),
        # Field sampled on points other than the sources, FP64 moments.
        _case(name="probe_points", n=100003, targets=50021, order=6, depth=4, output="both", dtype="float64"),
        # The flagship: 64 states per call on the million-dipole geometry.
        _case(name="states_1m", n=1048576, order=6, depth=5, states=64, output="both"),
        # High order on a jittered lattice, 64 states.
        _case(name="lattice_p8", points="lattice", n=262144, order=8, depth=5, states=64),
        # A mid-size ensemble: 16 states, 32 dipoles per leaf.
        _case(name="states_131k", n=131072, order=6, depth=4, states=16),
        # States kept on the host (pinned): copies in and out are the call's.
        _case(name="host_262k", entry="host", n=262144, order=6, depth=4, states=32, output="both"),
        # Differentiable use, one state at high order: forward and both
        # gradients.
        _case(name="gradient_p8", entry="gradient", n=524288, order=8, depth=5),
        # Differentiable use with a batch of states (an inverse problem's
        # ensemble).
        _case(name="gradient_states", entry="gradient", n=131072, order=6, depth=4, states=16),
        # Many uneven clustered problems in one graph launch.
        _case(name="problems_48", entry="batch", points="clusters", n=524288, order=6, problems=48),
        # Cuboid cells filling a body (30^3 touching cells), a few states.
        _case(name="cuboid_cells", entry="cuboid", points="lattice", n=27000, order=6, depth=3, states=4),
    ]


def _depth_for(n, rng):
    """About 32 dipoles per leaf (the benchmark's choice), sometimes a level coarser or finer."""
    d = int(round(math.log(max(n, 64) / 32.0, 8))) + rng.choice([0, 0, 0, 0, -1, 1])
    return min(5, max(1, d))


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    top = work(_case(n=1048576, order=6, depth=5, states=64, output="both"))["flops"]
    while True:
        entry = rng.choice(["device"] * 6 + ["host"] * 2 + ["gradient"] * 2 + ["dropin", "batch", "cuboid"])
        c = _case(entry=entry, points=rng.choice(["uniform", "uniform", "lattice", "clusters"]),
                  n=_log_int(rng, 2000, 1048576), order=rng.randint(3, 9), states=_log_int(rng, 1, 100),
                  output=rng.choice(["field", "field", "both", "potential"]), dtype=rng.choice(["float32"] * 3 + ["float64"]))
        if entry == "device" and rng.random() < 0.3:
            c["targets"] = _log_int(rng, 1000, c["n"])
        if entry == "dropin":
            c.update(states=1, dtype="float64", n=_log_int(rng, 2000, 262144))
        if entry == "gradient":
            c.update(output="field", dtype="float32", points=rng.choice(["uniform", "clusters"]))
        if entry == "batch":
            c.update(problems=rng.randint(3, 24), states=1, output="field", dtype="float32",
                     points=rng.choice(["uniform", "clusters"]), n=_log_int(rng, 16384, 262144))
        if entry == "cuboid":
            c.update(points="lattice", n=_log_int(rng, 3000, 40000), states=_log_int(rng, 1, 8), output="field")
        if c["points"] == "lattice":
            c["n"] = int(round(c["n"] ** (1 / 3))) ** 3
        c["depth"] = _depth_for(c["n"], rng)
        # clustered points put tens of times more pairs into the near field
        if c["points"] == "clusters" and c["n"] * c["states"] > 2 ** 21:
            continue
        if c["n"] * c["states"] <= 2 ** 26 and work(c)["flops"] <= top:
            return c


# ------------------------------------------------------------------ inputs

def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)
    return g


def _points(kind, n, g):
    """(n, 3) FP64 positions on the GPU."""
    if kind == "uniform":
        return torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64)
    if kind == "lattice":
        side = int(round(n ** (1 / 3)))
        a = torch.arange(side, device="cuda", dtype=torch.float64)
        x = torch.stack(torch.meshgrid(a, a, a, indexing="ij"), dim=-1).reshape(-1, 3)
        jitter = torch.rand(x.shape, generator=g, device="cuda", dtype=torch.float64) * 0.2 - 0.1
        return (x + 0.5 + jitter) / side
    # 8 Gaussian clusters, points outside the unit cube drawn again
    centres = torch.from_numpy(np.random.RandomState(n % 65537).uniform(0.1, 0.9, (8, 3))).cuda()
    out = torch.empty((0, 3), device="cuda", dtype=torch.float64)
    while len(out) < n:
        c = centres[torch.randint(0, 8, (2 * n,), generator=g, device="cuda")]
        x = c + 0.05 * torch.randn(c.shape, generator=g, device="cuda", dtype=torch.float64)
        out = torch.cat([out, x[((x >= 0) & (x < 1)).all(dim=1)]])
    return out[:n].contiguous()


def _moments(case, k, n, g):
    """(k, n, 3): i.i.d. normal states on the lattice, unit directions times U[0.5, 1.5] otherwise."""
    m = torch.randn((k, n, 3), generator=g, device="cuda", dtype=torch.float32)
    if case["points"] != "lattice":
        m /= m.norm(dim=2, keepdim=True).clamp_min(1e-20)
        m *= torch.rand((k, n, 1), generator=g, device="cuda", dtype=torch.float32) + 0.5
    return m.double() if case["dtype"] == "float64" else m


def _problem_sizes(case):
    """Sizes of a batch: log-uniform in [8192, n], the same for every seed."""
    r = np.random.RandomState(1000 + case["problems"])
    u = r.uniform(math.log(8192), math.log(case["n"]), size=case["problems"])
    return [int(v) for v in np.round(np.exp(u))]


def _problem_depth(n):
    return max(1, int(round(math.log(n / 32.0, 8))))


def _inputs(case, seed):
    """Positions, targets and moments of a single-geometry case."""
    g = _generator(seed, case["n"] + 7 * case["states"] + 131 * case["order"])
    if case["entry"] == "cuboid":
        # cells on an exact lattice: touching cubes
        side = int(round(case["n"] ** (1 / 3)))
        a = torch.arange(side, device="cuda", dtype=torch.float64)
        x = ((torch.stack(torch.meshgrid(a, a, a, indexing="ij"), dim=-1).reshape(-1, 3) + 0.5) / side).contiguous()
    else:
        x = _points(case["points"], case["n"], g)
    t = _points(case["points"] if case["points"] != "lattice" else "uniform", case["targets"], g) if case["targets"] else None
    m = _moments(case, case["states"], len(x), g)
    return x, t, m, g


def _options(case):
    o = cdfmm.UniformFmmOptions()
    o.expansion_order = case["order"]
    o.tree.max_level = case["depth"]
    return o


def prepare(case, seed):
    case = {**DEFAULTS, **case}
    entry = case["entry"]
    if entry == "batch":
        items = []
        for i, n in enumerate(_problem_sizes(case)):
            g = _generator(seed, 17 * n + i)
            x = _points(case["points"], n, g)
            plan = cdfmm_b200.DevicePlan.from_points(x, case["order"], _problem_depth(n), max_states=1)
            items.append((plan, _moments(case, 1, n, g), torch.empty((1, n, 3), device="cuda"), None))
        return {"case": case, "batch": cdfmm_b200.Batch(items, output="field"), "items": items}
    x, t, m, g = _inputs(case, seed)
    k, n = m.shape[0], m.shape[1]
    if entry == "dropin":
        xh = x.cpu().numpy()
        o = _options(case)
        o.fixed_target_source_indices = list(range(len(xh)))  # no dipole acts on itself
        return {"case": case, "fmm": cdfmm.UniformFmm(xh, xh, o), "moments": m[0].cpu().numpy()}
    plan = cdfmm_b200.DevicePlan.from_points(x, case["order"], case["depth"], targets=t, max_states=k)
    nt = plan.n_targets
    state = {"case": case, "plan": plan}
    if entry == "gradient":
        state["moments"] = m.requires_grad_(True)
        state["positions"] = x.float().requires_grad_(True)
        state["weights"] = torch.randn((k, nt, 3), generator=g, device="cuda", dtype=torch.float32)
        return state
    if entry == "cuboid":
        plan.set_source_cuboids([1.0 / int(round(n ** (1 / 3)))] * 3)
    want_h, want_phi = case["output"] != "potential", case["output"] != "field"
    if entry == "host":
        state["moments"] = torch.empty(m.shape, dtype=m.dtype, pin_memory=True).copy_(m)
        where = {"pin_memory": True}
    else:
        state["moments"] = m
        where = {"device": "cuda"}
    state["field"] = torch.zeros((k, nt, 3), **where) if want_h else None
    state["potential"] = torch.zeros((k, nt), **where) if want_phi else None
    return state


# -------------------------------------------------------------------- pass

def run(state):
    case = state["case"]
    entry = case["entry"]
    if entry == "dropin":
        out = state["fmm"].evaluate(state["moments"], output=case["output"])
        keep = {"field": ("H",), "potential": ("phi",), "both": ("H", "phi")}[case["output"]]
        return {key: out[key] for key in keep}
    stream = torch.cuda.current_stream().cuda_stream
    if entry == "batch":
        state["batch"].launch(stream=stream, synchronize=False)
        return [item[2] for item in state["items"]]
    if entry == "gradient":
        H = cdfmm_b200.dipole_field(state["plan"], state["moments"], state["positions"])
        gm, gx = torch.autograd.grad(H, (state["moments"], state["positions"]), grad_outputs=state["weights"])
        return {"H": H.detach(), "moments": gm, "positions": gx}
    state["plan"].evaluate(state["moments"], output=case["output"], field=state["field"],
                           potential=state["potential"], stream=stream, synchronize=False)
    return {key: v for key, v in (("H", state["field"]), ("phi", state["potential"])) if v is not None}


# -------------------------------------------------------------------- work

def _near_pairs(case, n, nt, depth):
    """(target, source) pairs in touching leaves: exact in the mean for uniform points; for clusters, counted on a
    sample of points of the same density."""
    side = 1 << depth
    if case["points"] != "clusters":
        return nt * n * ((3 * side - 2) / side ** 2) ** 3
    r = np.random.RandomState(5)
    centres = np.random.RandomState(n % 65537).uniform(0.1, 0.9, (8, 3))
    s = min(n, 20000)
    x = np.clip(centres[r.randint(0, 8, s)] + 0.05 * r.normal(size=(s, 3)), 0.0, 1.0 - 1e-9)
    cell = (x * side).astype(np.int64)
    count = np.zeros((side + 2,) * 3)
    np.add.at(count, tuple((cell + 1).T), 1.0)
    near = sum(np.roll(count, (a, b, c), (0, 1, 2)) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1))
    return nt * n / s ** 2 * float((count * near).sum())


def _far_pairs(depth):
    """List-2 (target box, source box) pairs of a full octree, all levels."""
    total = 0
    for level in range(2, depth + 1):
        side = 1 << level
        inner = [sum(1 for s in range(side) if s // 2 in range(t // 2 - 1, t // 2 + 2)) for t in range(side)]
        near = [min(t + 1, side - 1) - max(t - 1, 0) + 1 for t in range(side)]
        total += sum(inner) ** 3 - sum(near) ** 3
    return total


def work(case):
    """Bytes: inputs and positions read once, outputs written once.  FLOPs: near pairs (13 + 20 per state, 2 more of
    each for the potential), the order-(p + 1)^2 translations, and per point and state the expansions' 4 n."""
    case = {**DEFAULTS, **case}
    p, k = case["order"], case["states"]
    n_coef, t_coef = (p + 1) * (p + 2) * (p + 3) // 6, (p + 1) ** 2
    sizes = [(n, n, _problem_depth(n)) for n in _problem_sizes(case)] if case["entry"] == "batch" else \
        [(case["n"], case["targets"] or case["n"], case["depth"])]
    bytes_, flops = 0.0, 0.0
    for n, nt, depth in sizes:
        pairs = _near_pairs(case, n, nt, depth)
        wide = 8 if case["dtype"] == "float64" else 4
        out = {"field": 3, "potential": 1, "both": 4}[case["output"]]
        b = 12 * (n + (nt if case["targets"] else 0)) + 3 * wide * n * k + 4 * out * nt * k
        per_pair = {"field": 13 + 18 * k, "potential": 11 + 6 * k, "both": 13 + 20 * k}[case["output"]]
        f = pairs * per_pair + 2.0 * t_coef * t_coef * k * _far_pairs(depth) + 4.0 * n_coef * k * (n + nt)
        if case["entry"] == "cuboid":
            b += 24 * pairs  # the stored pair tensors
            f = pairs * 18 * k + 2.0 * t_coef * t_coef * k * _far_pairs(depth) + 4.0 * n_coef * k * (n + nt)
        if case["entry"] == "gradient":
            # forward, transposed evaluation, and the position gradient's near and leaf parts
            b += 4 * (3 * nt * k + 3 * n * k + 3 * nt)
            f = 2 * f + pairs * (20 + 40 * k)
        bytes_ += b
        flops += f
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """Four times what two arithmetics of the same precision differ by: the split tensor-core near field and M2L
    against their FP32 forms gave up to 1.7e-6 (largest value 5.5e-5) on random points, and on lattices, whose
    fields cancel and whose potentials are small, up to 6.4e-6 (5e-5)."""
    return {"rel": 2.5e-5 if case.get("points") == "lattice" else 7e-6, "max": 2.2e-4}


# ------------------------------------------------- 64-bit direct summation

def _pair_geometry(x, t, i0, i1, self_excluded):
    """Differences and 1/r of targets [i0, i1) against every source."""
    d = [t[i0:i1, a, None] - x[None, :, a] for a in range(3)]
    r2 = d[0] * d[0]
    r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
    if self_excluded:
        i = torch.arange(i0, i1, device="cuda")
        r2[i - i0, i] = math.inf
    return d, r2.rsqrt_()


def _direct(x, t, m, self_excluded, want_h, want_phi):
    """H (k, nt, 3) and phi (k, nt) of the dipoles m (k, n, 3) in FP64."""
    k, n, nt = m.shape[0], len(x), len(t)
    mm = [m[:, :, a].T.contiguous() for a in range(3)]  # (n, k)
    H = torch.zeros((3, nt, k), dtype=torch.float64, device="cuda") if want_h else None
    phi = torch.zeros((nt, k), dtype=torch.float64, device="cuda") if want_phi else None
    step = max(1, min(nt, int(1.5e8) // max(n, 1)))
    for i0 in range(0, nt, step):
        i1 = min(nt, i0 + step)
        d, u = _pair_geometry(x, t, i0, i1, self_excluded)
        u3 = u * u * u
        if want_phi:
            for a in range(3):
                phi[i0:i1].addmm_(d[a] * u3, mm[a])
        if want_h:
            u5 = u.mul_(u).mul_(u3).mul_(3.0)
            for a in range(3):
                for b in range(a, 3):
                    T = d[a] * d[b]
                    T.mul_(u5)
                    if a == b:
                        T.sub_(u3)
                    H[a, i0:i1].addmm_(T, mm[b])
                    if a != b:
                        H[b, i0:i1].addmm_(T, mm[a])
        del d, u, u3
    c = 1.0 / (4.0 * math.pi)
    return (H.mul_(c).permute(2, 1, 0).contiguous() if want_h else None,
            phi.mul_(c).T.contiguous() if want_phi else None)


def _direct_position_gradient(x, m, w):
    """d/dx_i of sum_k w_ki . H_ki for targets == sources, in FP64: (n, 3)."""
    n = len(x)
    out = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    step = max(1, min(n, int(1.0e8) // n))
    for i0 in range(0, n, step):
        i1 = min(n, i0 + step)
        d, u = _pair_geometry(x, x, i0, i1, True)
        u2 = u * u
        u5 = u2 * u2 * u
        u7 = u5 * u2
        # S_ab = sum_k w_a m_b per pair
        S = lambda a, b: w[:, i0:i1, a].T @ m[:, :, b]  # noqa: E731
        full = torch.zeros_like(u)  # sum_ab r_a S_ab r_b
        trace = torch.zeros_like(u)
        side = [torch.zeros_like(u) for _ in range(3)]  # sum_a r_a (S_ad + S_da)
        for a in range(3):
            for b in range(3):
                s = S(a, b)
                if a == b:
                    trace += s
                side[b].addcmul_(d[a], s)
                side[a].addcmul_(d[b], s)
        for a in range(3):
            full.addcmul_(d[a], side[a], value=0.5)
        full.mul_(u7).mul_(-15.0)
        for a in range(3):
            v = side[a].addcmul_(trace, d[a]).mul_(u5).mul_(3.0).addcmul_(full, d[a])
            out[i0:i1, a] = v.sum(dim=1)
    return out / (4.0 * math.pi)


def _direct_cuboids(x, m, h):
    """H of uniformly magnetised cubes of side h (self pairs included): the closed form with surface charges."""
    n, k = len(x), m.shape[0]
    mm = [m[:, :, a].T.contiguous() for a in range(3)]
    H = torch.zeros((3, n, k), dtype=torch.float64, device="cuda")
    step = max(1, int(2e7) // n)
    for i0 in range(0, n, step):
        i1 = min(n, i0 + step)
        r = [x[i0:i1, a, None] - x[None, :, a] for a in range(3)]
        T = {}
        for sx in (-1, 1):
            for sy in (-1, 1):
                for sz in (-1, 1):
                    c = [r[0] - sx * h / 2, r[1] - sy * h / 2, r[2] - sz * h / 2]
                    R = torch.sqrt(c[0] ** 2 + c[1] ** 2 + c[2] ** 2)
                    s = float(sx * sy * sz)
                    for a in range(3):
                        b, e = (a + 1) % 3, (a + 2) % 3
                        v = torch.atan(c[b] * c[e] / (c[a] * R))
                        T[a, a] = T[a, a] + s * v if (a, a) in T else s * v
                        v = torch.asinh(c[e] / torch.sqrt(c[a] ** 2 + c[b] ** 2))
                        T[a, b] = T[a, b] - s * v if (a, b) in T else -s * v
        f = 1.0 / (4.0 * math.pi * h ** 3)
        for (a, b), v in T.items():
            v = torch.nan_to_num(v * f)
            H[a, i0:i1].addmm_(v, mm[b])
            if a != b:
                H[b, i0:i1].addmm_(v, mm[a])
    return H.permute(2, 1, 0).contiguous()


def exact(case, seed):
    """The quantity the FMM approximates: the direct sum over all pairs, in FP64.  The difference holds the truncation
    at the case's order beside the rounding."""
    case = {**DEFAULTS, **case}
    if case["entry"] == "batch":
        if sum(n * n for n in _problem_sizes(case)) > EXACT_PAIRS:
            return None
        out = []
        for i, n in enumerate(_problem_sizes(case)):
            g = _generator(seed, 17 * n + i)
            x = _points(case["points"], n, g)
            m = _moments(case, 1, n, g).double()
            out.append(_direct(x, x, m, True, True, False)[0])
        return out
    pairs = float(case["n"]) * (case["targets"] or case["n"])
    if pairs > (EXACT_CUBOID_PAIRS if case["entry"] == "cuboid" else EXACT_PAIRS):
        return None
    if case["entry"] == "gradient" and pairs > 2e10:
        return None
    x, t, m, g = _inputs(case, seed)
    m = m.double()
    if case["entry"] == "cuboid":
        return {"H": _direct_cuboids(x, m, 1.0 / int(round(len(x) ** (1 / 3))))}
    if case["entry"] == "gradient":
        w = torch.randn(m.shape, generator=g, device="cuda", dtype=torch.float32).double()
        return {"H": _direct(x, x, m, True, True, False)[0], "moments": _direct(x, x, w, True, True, False)[0],
                "positions": _direct_position_gradient(x, m, w)}
    want_h, want_phi = case["output"] != "potential", case["output"] != "field"
    H, phi = _direct(x, x if t is None else t, m, t is None, want_h, want_phi)
    out = {key: v for key, v in (("H", H), ("phi", phi)) if v is not None}
    if case["entry"] == "dropin":
        return {key: v[0].cpu().numpy() for key, v in out.items()}
    return out
