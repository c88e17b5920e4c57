"""Performance cases of the framework: one pass each of the calls that a user's
time loop makes, over the range of sizes that the library takes.

The workloads are those of this repository's benchmark, tests and
configurations: the Rossby-Haurwitz barotropic vorticity (BVE) step on the
unit sphere (Omega = 2 pi, dt = 0.005, eps = 1e-4), the balanced shallow-water
(SWE) flow, the Gaussian-vortex adjoint, the batched ensemble, the Poisson
solve and the plain direct sum.  Every field is synthetic and made from a seed.

exact() evaluates the same step in float64 with plain torch and the direct sum
(every velocity method approximates it), on a grid built here with numpy.
"""
import functools
import importlib
import math

import numpy as np
import torch

sb = importlib.import_module("spectral-bslpm_b200")

EPS, OMEGA, DT, SWE_DT, ADJ_DT = 1e-4, 2 * math.pi, 0.005, 0.002, 0.01
K4 = 1.0 / (4.0 * math.pi)


# ----------------------------------------------------------------- cases ----

def listed():
    return [
        # the smallest problem a user steps (set-up checks, teaching, unit tests): launches and latency
        dict(name="bve_fp64_small", kind="bve", method="spectral", precision="float64", levels=3, degree=3, theta=0.7,
             call="step", steps=1, tracers=0),
        # the library's default configuration (levels 5, degree 3, float64, theta 0.7) with a tracer, run between outputs
        dict(name="bve_fp64_default", kind="bve", method="spectral", precision="float64", levels=5, degree=3,
             theta=0.7, call="run", steps=10, tracers=1),
        # the reference's own method in float64 at the largest theta that meets the 1e-6 bar, 393,216 particles
        dict(name="bve_fp64_large", kind="bve", method="spectral", precision="float64", levels=7, degree=3, theta=0.45,
             call="run", steps=2, tracers=0),
        # host arrays in and out each step (the drop-in's route), mixed precision, an odd panel size (25 points)
        dict(name="bve_mixed_host_d4", kind="bve", method="spectral", precision="mixed", levels=6, degree=4, theta=0.5,
             call="host", steps=1, tracers=0),
        # the benchmark's headline: mixed-precision treecode, 393,216 particles
        dict(name="bve_tree_mixed_large", kind="bve", method="tree", precision="mixed", levels=7, degree=3, theta=0.7,
             proxy=8, leaf=256, call="run", steps=2, tracers=0),
        # the treecode in float64, 98,304 particles
        dict(name="bve_tree_fp64", kind="bve", method="tree", precision="float64", levels=6, degree=3, theta=0.7,
             proxy=8, leaf=256, call="run", steps=2, tracers=0),
        # the plain direct sum over scattered points (no grid), sizes that divide by nothing
        dict(name="direct_fp64_odd", kind="direct", precision="float64", targets=10007, sources=24577),
        # one step of the shallow-water driver in float64, degree 2 (9 points a panel), 55,296 particles
        dict(name="swe_fp64_d2", kind="swe", method="spectral", precision="float64", levels=6, degree=2, theta=0.7,
             call="step", steps=1, tracers=0),
        # the shallow-water driver's loop on the mixed-precision treecode, 98,304 particles
        dict(name="swe_tree_mixed", kind="swe", method="tree", precision="mixed", levels=6, degree=3, theta=0.7,
             proxy=8, leaf=256, call="run", steps=1, tracers=0),
        # one reverse step of the float64 treecode (the gradient of a rollout), 24,576 particles
        dict(name="adjoint_tree_fp64", kind="adjoint", method="tree", precision="float64", levels=5, degree=3,
             theta=0.7, proxy=8, leaf=256),
        # an uneven mixed-precision ensemble stepped together: 16 members of 24,576 particles
        dict(name="ensemble_mixed", kind="ensemble", precision="mixed", levels=5, degree=3, members=16, leaf=256,
             steps=1),
        # the Poisson solve of the inverse-Laplacian driver, 98,304 points
        dict(name="poisson_fp64", kind="poisson", levels=6, degree=3, theta=0.7),
    ]


def draw(rng):
    kind = rng.choice(["bve", "bve", "bve", "tree", "tree", "direct", "swe", "swetree", "adjoint", "ensemble",
                       "poisson"])
    theta = round(rng.uniform(0.45, 0.85), 3)
    precision = rng.choice(["float64", "float64", "mixed"])
    if kind == "direct":
        n = [int(math.exp(rng.uniform(math.log(500), math.log(24577)))) for _ in range(2)]
        return dict(kind="direct", precision=precision, targets=n[0], sources=n[1])
    if kind == "ensemble":
        return dict(kind="ensemble", precision="mixed", levels=rng.choice([4, 5]), degree=3,
                    members=rng.randint(2, 16), leaf=256, steps=1)
    if kind == "adjoint":
        method = rng.choice(["tree", "spectral", "direct"])
        c = dict(kind="adjoint", method=method, precision="float64", levels=rng.choice([3, 4, 5]), degree=3,
                 theta=min(theta, 0.7))
        return dict(c, proxy=rng.choice([6, 7, 8]), leaf=rng.choice([64, 256])) if method == "tree" else c
    degree = rng.choice([2, 3, 3, 4])
    top = {2: 6, 3: 6, 4: 5}[degree]
    if kind == "poisson":
        return dict(kind="poisson", levels=rng.randint(3, top), degree=degree, theta=theta)
    levels = rng.randint(4 if kind.endswith("tree") else 3, top)
    c = dict(kind="swe" if kind.startswith("swe") else "bve", method="tree" if kind.endswith("tree") else "spectral",
             precision=precision, levels=levels, degree=degree, theta=theta, tracers=rng.choice([0, 0, 1, 2]))
    if c["method"] == "tree":
        c.update(proxy=rng.randint(5, 9), leaf=rng.choice([64, 256]))
    if c["kind"] == "swe":
        return dict(c, call=rng.choice(["step", "run"]), steps=1)
    call = rng.choice(["step", "run", "host"])
    return dict(c, call=call, steps=rng.randint(2, 5) if call == "run" and levels < 6 else 1)


# ------------------------------------------------------------------ grid ----

@functools.lru_cache(maxsize=8)
def grid(levels, degree):
    """The leaf points of the cubed sphere, [leaf][q]: Chebyshev extrema of each
    panel, exact Clenshaw-Curtis weights times the panel's spherical area."""
    face, bits = np.arange(6), [np.zeros(6, int), np.zeros(6, int)]
    for _ in range(levels - 1):  # children (+,+), (-,+), (-,-), (+,-) in (xi, eta)
        face = np.repeat(face, 4)
        child = np.tile(np.arange(4), len(bits[0]))
        bits = [np.repeat(b, 4) * 2 + np.isin(child, up) for b, up in zip(bits, ((0, 3), (0, 1)))]
    n = 2 ** (levels - 1)
    lo = [math.pi / 4 * (2.0 * b / n - 1) for b in bits]
    hi = [math.pi / 4 * (2.0 * (b + 1) / n - 1) for b in bits]
    i = np.arange(degree + 1)
    node = np.cos(math.pi * i / degree)
    node[np.abs(node) < 1e-16] = 0
    cc = np.array([(1.0 if k in (0, degree) else 2.0) / degree *
                   (1 - sum((1.0 if 2 * j == degree else 2.0) * math.cos(2 * j * math.pi * k / degree) /
                            (4.0 * j * j - 1) for j in range(1, degree // 2 + 1))) for k in i])

    def point(xi, eta, f):
        X, Y = np.tan(xi), np.tan(eta)
        r = 1 / np.sqrt(1 + X * X + Y * Y)
        p = [(r, X * r, Y * r), (-X * r, r, Y * r), (-r, -X * r, Y * r), (X * r, -r, Y * r), (-Y * r, X * r, r),
             (Y * r, X * r, -r)]
        return np.stack([np.choose(f, [a[c] for a in p]) for c in range(3)])

    xi = 0.5 * (lo[0] + hi[0])[:, None] + 0.5 * (hi[0] - lo[0])[:, None] * node
    eta = 0.5 * (lo[1] + hi[1])[:, None] + 0.5 * (hi[1] - lo[1])[:, None] * node
    A, q = len(face), (degree + 1) ** 2
    XI, ETA = np.repeat(xi, degree + 1, 1), np.tile(eta, (1, degree + 1))
    x, y, z = point(XI, ETA, np.broadcast_to(face[:, None], (A, q)))
    c = [point(a, b, face) for a, b in ((hi[0], hi[1]), (hi[0], lo[1]), (lo[0], lo[1]), (lo[0], hi[1]))]

    def triangle(p, r, s):  # spherical excess of a triangle (L'Huilier)
        e = [np.arccos(1 - 0.5 * ((a - b) ** 2).sum(0)) for a, b in ((r, s), (s, p), (p, r))]
        h = sum(e) / 2
        return 4 * np.arctan(np.sqrt(np.tan(h / 2) * np.prod([np.tan((h - a) / 2) for a in e], axis=0)))

    area = (triangle(c[0], c[1], c[2]) + triangle(c[0], c[2], c[3]))[:, None] / 4 * np.outer(cc, cc).ravel()
    g = dict(x=x, y=y, z=z, area=area, lo=lo, hi=hi, face=face, node=node, XI=XI, ETA=ETA)
    return g


def particles(case):
    return 6 * 4 ** (case["levels"] - 1) * (case["degree"] + 1) ** 2


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@functools.lru_cache(maxsize=4)
def on_gpu(levels, degree):
    g = grid(levels, degree)
    return tuple(cuda(g[k]) for k in ("x", "y", "z", "area"))


def smooth(g, rng, amplitude):
    """A seeded smooth field: harmonics of degrees 1 to 3."""
    x, y, z = g["x"], g["y"], g["z"]
    terms = (x, y, z, x * y, y * z, z * x, x * x - y * y, x * y * z, z * (x * x - y * y), x * (x * x - 3 * y * y))
    return amplitude * sum(c * t for c, t in zip(rng.standard_normal(len(terms)), terms))


def rossby_haurwitz(g, seed):
    """RH4 (omega0 = K = 0.5) with a seeded perturbation, mean removed."""
    lat, lon = np.arcsin(np.clip(g["z"], -1, 1)), np.arctan2(g["y"], g["x"])
    v = np.sin(lat) - 0.5 * np.sin(lat) * np.cos(lat) ** 4 * 30 * np.cos(4 * lon)
    v = v + smooth(g, np.random.default_rng(seed), 0.05)
    return v - (v * g["area"]).sum() * K4


def tracers_of(g, count):
    return np.stack([np.exp(-((g["x"] - math.cos(k)) ** 2 + (g["y"] - math.sin(k)) ** 2 + g["z"] ** 2) / 0.2)
                     for k in range(count)], -1) if count else None


def vortex(g, seed):
    """The Gaussian vortex at 30 degrees north with a seeded smooth perturbation, and a smooth cotangent."""
    rng = np.random.default_rng(seed)
    c = math.cos(math.pi / 6), math.sin(math.pi / 6)
    v = np.exp(-((g["x"] - c[0]) ** 2 + g["y"] ** 2 + (g["z"] - c[1]) ** 2) / (2 * 0.15 ** 2)) + smooth(g, rng, 0.02)
    return v, g["area"] * (smooth(g, rng, 1.0) + 0.2 * rng.standard_normal(v.shape))


def balanced(g, seed):
    """Steady geostrophic flow (g/a = 1) with a seeded disturbance of vorticity, divergence and height."""
    rng, u0 = np.random.default_rng(seed), OMEGA / 12
    vors = 2 * u0 * g["z"] + smooth(g, rng, 0.02)
    divs = smooth(g, rng, 0.02)
    h = 2.94 - (OMEGA * u0 + 0.5 * u0 * u0) * g["z"] ** 2 + smooth(g, rng, 1e-3)
    mean = [(f * g["area"]).sum() * K4 for f in (vors, divs)]
    return vors - mean[0], divs - mean[1], h


def members_of(case, seed):
    rng = np.random.default_rng(2026 + case["members"])  # the members' methods are the plan's, not the inputs'
    theta = rng.uniform(0.5, 0.8, case["members"])
    degree = rng.choice([6, 8, 10], case["members"])
    g = grid(case["levels"], case["degree"])
    return theta, degree, np.stack([rossby_haurwitz(g, 1000 * seed + m) for m in range(case["members"])])


def scattered(case, seed):
    rng = np.random.default_rng(seed)

    def sphere(n):
        p = rng.standard_normal((3, n))
        return p / np.sqrt((p * p).sum(0))

    t, s = sphere(case["targets"]), sphere(case["sources"])
    return t, s, rng.standard_normal(case["sources"]) * 4 * math.pi / case["sources"]


# --------------------------------------------------------------- prepare ----

def config(case, **more):
    c = dict(levels=case["levels"], interp_degree=case["degree"], kernel_eps=EPS, omega=OMEGA, dt=DT,
             precision=sb.MIXED if case.get("precision") == "mixed" else sb.FP64, fmm_theta=case.get("theta", 0.7),
             tracer_count=case.get("tracers", 0), exact_cc=1)
    if case.get("method") == "tree":
        c.update(proxy_degree=case["proxy"], leaf_size=case["leaf"])
    if case.get("method") == "direct":
        c.update(velocity=sb.VEL_DIRECT)
    c.update(more)
    return sb.config_default(**c)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "direct":
        t, s, w = scattered(case, seed)
        return dict(case=case, args=[cuda(a) for a in (*t, *s, w)],
                    out=tuple(torch.zeros(case["targets"], dtype=torch.float64, device="cuda") for _ in range(3)))
    g = grid(case["levels"], case["degree"])
    xyza = on_gpu(case["levels"], case["degree"])
    vel = [torch.zeros_like(xyza[0]) for _ in range(3)]
    if kind == "bve":
        ctx = sb.Context(config(case))
        v0, tr = cuda(rossby_haurwitz(g, seed)), tracers_of(g, case["tracers"])
        tr = None if tr is None else cuda(tr)
        # the initial velocity (a driver's first output) also settles the launch shapes; the results of a mixed
        # treecode are then kept independent of that timing, as a program that has to reproduce its runs does
        ctx.bve_velocity(*xyza, v0, *vel)
        if case["method"] == "tree":
            ctx.set_near_mutual(False)
        st = dict(case=case, ctx=ctx, xyza=xyza, v0=v0, t0=tr, v=v0.clone(), vel=vel,
                  tr=None if tr is None else tr.clone())
        if case["call"] == "host":
            for k in ("v0", "t0", "v", "tr"):
                st[k] = None if st[k] is None else st[k].cpu().pin_memory()
            st["xyza"] = [t.cpu().pin_memory() for t in xyza]
            st["vel"] = [t.cpu().pin_memory() for t in vel]
        return st
    if kind == "swe":
        ctx = sb.Context(config(case, dt=SWE_DT, g_over_a=1.0))
        f0 = [cuda(a) for a in balanced(g, seed)]
        base = [torch.zeros_like(vel[0]) for _ in range(3)]
        ctx.swe_init(*xyza, *f0, *vel, *base)
        base = [torch.zeros_like(b) for b in base]  # a free run: no base tendencies
        tr = tracers_of(g, case["tracers"])
        tr = None if tr is None else cuda(tr)
        return dict(case=case, ctx=ctx, xyza=xyza, f0=f0, f=[a.clone() for a in f0], vel=vel, base=base, t0=tr,
                    tr=None if tr is None else tr.clone())
    if kind == "adjoint":
        ctx = sb.Context(config(case, dt=ADJ_DT))
        v, bar = vortex(g, seed)
        v = cuda(v)
        ctx.bve_velocity(*xyza, v, *vel)
        return dict(case=case, ctx=ctx, xyza=xyza, v=v, bar=cuda(bar), out=torch.zeros_like(v))
    if kind == "ensemble":
        theta, degree, v = members_of(case, seed)
        batch = sb.Batch(config(case, leaf_size=case["leaf"]), theta, degree)
        batch.set_cc_mode(sb.Batch.CC_SHARED)  # reproducible: the timing of the modes does not choose the rounding
        v0 = cuda(v)
        vel = torch.zeros((case["members"], 3) + tuple(v0.shape[1:]), dtype=torch.float64, device="cuda")
        batch.step(*xyza, v0.clone(), vel)
        return dict(case=case, batch=batch, xyza=xyza, v0=v0, v=v0.clone(), vel=vel)
    f = cuda(smooth(g, np.random.default_rng(seed), 1.0))
    return dict(case=case, ctx=sb.Context(config(case)), xyza=xyza, f=f, out=torch.zeros_like(f))


# ------------------------------------------------------------------- run ----

def run(s):
    """One pass; the time loops start again from the initial state each time."""
    case = s["case"]
    kind = case["kind"]
    if kind == "direct":
        return sb.direct_sum_bve(*s["args"], EPS, sb.MIXED if case["precision"] == "mixed" else sb.FP64, s["out"])
    if kind == "bve":
        s["v"].copy_(s["v0"])
        if s["tr"] is not None:
            s["tr"].copy_(s["t0"])
        args = (*s["xyza"], s["v"], *s["vel"], s["tr"])
        if case["call"] == "run":
            s["ctx"].bve_run(*args, nsteps=case["steps"])
        elif case["call"] == "host":
            s["ctx"].bve_back_rk4_step_host(*args)
        else:
            s["ctx"].bve_back_rk4_step(*args)
        return dict(vors=s["v"], vel=s["vel"], **({} if s["tr"] is None else {"tracers": s["tr"]}))
    if kind == "swe":
        for a, b in zip(s["f"], s["f0"]):
            a.copy_(b)
        if s["tr"] is not None:
            s["tr"].copy_(s["t0"])
        args = (*s["xyza"], *s["f"], *s["vel"], s["tr"], *s["base"])
        if case["call"] == "run":
            s["ctx"].swe_run(*args, nsteps=case["steps"])
        else:
            s["ctx"].swe_back_rk4_step_2(*args)
        return dict(fields=s["f"], vel=s["vel"], **({} if s["tr"] is None else {"tracers": s["tr"]}))
    if kind == "adjoint":
        s["ctx"].bve_adjoint_step(*s["xyza"], s["v"], s["bar"], s["out"])
        return s["out"]
    if kind == "ensemble":
        s["v"].copy_(s["v0"])
        s["batch"].run(*s["xyza"], s["v"], s["vel"], nsteps=case["steps"])
        return dict(vors=s["v"], vel=s["vel"])
    s["ctx"].poisson_fmm(s["xyza"][3], s["f"], s["out"])
    return s["out"]


# ------------------------------------------------------------------ work ----

@functools.lru_cache(maxsize=64)
def pairs(levels, degree, theta, proxy, leaf):
    """Pair evaluations of one velocity evaluation by the interaction list (proxy 0: the reference's method)."""
    q = (degree + 1) ** 2
    if not proxy:
        return len(sb.dual_tree_traversal(levels, sb.cubed_sphere_panels_init(levels), theta)) * q * q
    points, tree = q, levels
    while points * 4 <= leaf and tree > 1:
        points, tree = points * 4, tree - 1
    near = sb.dual_tree_traversal_flagged(tree, sb.cubed_sphere_panels_init(tree), theta)[1]
    return int(near.sum()) * points ** 2 + int((near == 0).sum()) * (proxy + 1) ** 4


def pairs_of(case, theta=None, proxy=None):
    if case.get("method") == "direct":
        return particles(case) ** 2
    return pairs(case["levels"], case["degree"], case["theta"] if theta is None else float(theta),
                 case.get("proxy", 0) if proxy is None else int(proxy), case.get("leaf", 0))


def work(case):
    """17 operations per Biot-Savart pair, 41 per shallow-water pair, 4 stages a step; the transposed pair of
    the adjoint (strength and position adjoints) 40; 8 and a logarithm (20) per Poisson pair."""
    kind = case["kind"]
    if kind == "direct":
        return dict(bytes=8 * (6 * case["targets"] + 4 * case["sources"]), flops=17 * case["targets"] * case["sources"])
    n = particles(case)
    if kind == "bve":
        fields = 4 + 1 + 1 + 3 + 2 * case["tracers"]
        return dict(bytes=8 * n * fields, flops=4 * 17 * pairs_of(case) * case["steps"])
    if kind == "swe":
        return dict(bytes=8 * n * (4 + 6 + 3 + 3 + 2 * case["tracers"]), flops=4 * 41 * pairs_of(case) * case["steps"])
    if kind == "adjoint":
        return dict(bytes=8 * n * 7, flops=4 * (17 + 40) * pairs_of(case))
    if kind == "ensemble":
        theta, degree, _ = members_of(case, 0)
        return dict(bytes=8 * n * (4 + 5 * case["members"]),
                    flops=4 * 17 * case["steps"] * sum(pairs_of(case, t, d) for t, d in zip(theta, degree)))
    return dict(bytes=8 * n * 3, flops=28 * pairs_of(case))


# ----------------------------------------------------------------- exact ----

def rows(n):
    return max(1, min(n, int(2e8 // n)))


class BiotSavart(torch.autograd.Function):
    """u_i = -1/(4 pi) sum_j w_j x_i cross y_j / (1 - x_i.y_j + eps), x and y [n][3]."""

    @staticmethod
    def forward(ctx, x, y, w):
        ctx.save_for_backward(x, y, w)
        a = torch.empty_like(x)
        m, wy = rows(len(y)), w[:, None] * y
        for k in range(0, len(x), m):
            a[k:k + m] = torch.mm(x[k:k + m], y.T).neg_().add_(1 + EPS).reciprocal_() @ wy
        return -K4 * torch.linalg.cross(x, a)

    @staticmethod
    def backward(ctx, ubar):
        x, y, w = ctx.saved_tensors
        abar = -K4 * torch.linalg.cross(ubar, x)
        wb, yb = torch.zeros_like(w), torch.zeros_like(y)
        m = rows(len(y))
        for k in range(0, len(x), m):
            xs, ab = x[k:k + m], abar[k:k + m]
            r = torch.mm(xs, y.T).neg_().add_(1 + EPS).reciprocal_()
            p = torch.mm(ab, y.T).mul_(r)
            wb += p.sum(0)
            yb += w[:, None] * (r.T @ ab + p.mul_(r).T @ xs)
        return None, yb, wb


def divergent(x, y, w):
    """1/(4 pi) sum_j w_j (y_j - x_i (x_i.y_j)) / (1 - x_i.y_j + eps)."""
    a, m, wy = torch.empty_like(x), rows(len(y)), w[:, None] * y
    for k in range(0, len(x), m):
        a[k:k + m] = torch.mm(x[k:k + m], y.T).neg_().add_(1 + EPS).reciprocal_() @ wy
    return K4 * (a - x * (x * a).sum(1, keepdim=True))


def unit(p):
    return p / p.norm(dim=1, keepdim=True)


def face_coordinates(p):
    x, y, z = p.unbind(1)
    ax, ay, az = x.abs(), y.abs(), z.abs()
    face = torch.where((ax >= ay) & (ax >= az), torch.where(x >= 0, 0, 2),
                       torch.where((ay >= ax) & (ay >= az), torch.where(y >= 0, 1, 3), torch.where(z >= 0, 4, 5)))

    def pick(*v):
        return torch.stack(v, 1).gather(1, face[:, None])[:, 0]

    den = pick(x, y, x, y, z, z)
    return face, torch.atan(pick(y, -x, y, -x, y, -y) / den), torch.atan(pick(z, z, -z, -z, -x, -x) / den)


def interpolate(p, fields, levels, degree):
    """The panel-wise barycentric interpolation of fields [leaf * q][k] at the points p."""
    face, xi, eta = face_coordinates(p)
    n, leaf, f = 2 ** (levels - 1), face, []
    cell = [((t.detach() / (math.pi / 4) + 1) * 0.5 * n).floor().long().clamp(0, n - 1) for t in (xi, eta)]
    for b in range(levels - 2, -1, -1):
        up = [(c >> b) & 1 for c in cell]
        leaf = 4 * leaf + torch.where(up[1] == 1, 1 - up[0], 2 + up[0])
    i = torch.arange(degree + 1, device=p.device, dtype=torch.float64)
    node = torch.cos(math.pi * i / degree)
    wt = (-1.0) ** i * torch.where((i == 0) | (i == degree), 0.5, 1.0)
    for t, c in zip((xi, eta), cell):
        d = (t / (math.pi / 4) + 1) * n - 2 * c - 1  # the panel's own coordinate in [-1, 1]
        dl = d[:, None] - node
        prod = torch.stack([wt[k] * dl[:, [j for j in range(degree + 1) if j != k]].prod(1) for k in range(degree + 1)], 1)
        f.append(prod / prod.sum(1, keepdim=True))
    basis = (f[0][:, :, None] * f[1][:, None, :]).flatten(1)
    at = fields.view(-1, basis.shape[1], fields.shape[1])
    return torch.stack([(at[leaf, :, k] * basis).sum(1) for k in range(fields.shape[1])], 1)


def departure(x, v, dt, levels, degree):
    k1 = v[3]
    k2 = interpolate(unit(x - 0.5 * dt * k1), v[2], levels, degree)
    k3 = interpolate(unit(x - 0.5 * dt * k2), v[1], levels, degree)
    k4 = interpolate(unit(x - dt * k3), v[0], levels, degree)
    p = x  # the weights' signs are the reference's
    for c, k in ((-1 / 6, k1), (1 / 3, k2), (1 / 3, k3), (1 / 6, k4)):
        p = unit(p + c * dt * k)
    return p


def bve_step(case, x, area, vors, tracers, dt):
    v = []
    for h in (0.0, 0.5 * dt, 0.5 * dt, dt):
        y = unit(x + h * v[-1]) if v else x
        v.append(BiotSavart.apply(x, y, area * (vors + 2 * OMEGA * (x[:, 2] - y[:, 2]))))
    p = departure(x, v, dt, case["levels"], case["degree"])
    fields = vors[:, None] if tracers is None else torch.cat([vors[:, None], tracers], 1)
    new = interpolate(p, fields, case["levels"], case["degree"])
    return new[:, 0] + 2 * OMEGA * (p[:, 2] - x[:, 2]), new[:, 1:], v[0]


@functools.lru_cache(maxsize=2)
def stencils(levels, degree):
    """Panel tables of the finite-difference tendencies: derivative matrices along each direction, the filter's
    matrix, the nodes' tangents and the map of points to distinct positions."""
    g = grid(levels, degree)
    n1 = degree + 1
    t = g["node"]
    D = np.zeros((n1, n1))

    def end(a, b, c):
        h, r = abs(a - b), (a - c) / (a - b)
        return np.array([-1 - 1 / r, r / (r - 1), -1 / (r * r - r)]) / h

    D[0, :3] = end(t[0], t[1], t[2])
    D[degree, degree - 2:] = -end(t[0], t[1], t[2])[::-1]
    for i in range(1, degree):
        d1, d2 = t[i - 1] - t[i], t[i] - t[i + 1]
        h, r = min(d1, d2), max(d1, d2) / min(d1, d2)
        w = (-r / (r + 1), (r - 1) / r, 1 / (r * r + r)) if d1 < d2 else (-1 / (r * r + r), (1 - r) / r, r / (r + 1))
        D[i, i - 1:i + 2] = np.array(w) / h
    c = 0.0005
    F = np.zeros((n1, n1))
    for i in range(n1):
        a, b = (1, 2) if i == 0 else (degree - 1, degree - 2) if i == degree else (i - 1, i + 1)
        da, db = abs(t[i] - t[a]), abs(t[i] - t[b])
        F[i, b] += 0.25 * c / (da + db) * da
        F[i, a] += 0.25 * c / (da + db) * db
    key = np.round(np.stack([g[k].ravel() for k in "xyz"], 1) * 1e9).astype(np.int64)
    where = np.unique(key, axis=0, return_inverse=True)[1].reshape(-1)
    scale = 2.0 * 2 ** (levels - 1) / (math.pi / 2)  # d(panel coordinate)/d(xi)
    return cuda(D * scale), cuda(F), cuda(np.tan(g["XI"])), cuda(np.tan(g["ETA"])), cuda(where)


def unify(f, where):
    total = torch.zeros((int(where.max()) + 1,) + f.shape[1:], dtype=f.dtype, device=f.device).index_add_(0, where, f)
    count = torch.zeros(len(total), dtype=f.dtype, device=f.device).index_add_(0, where, torch.ones_like(f[:, 0]))
    return (total / count[:, None])[where]


def tendencies(case, x, v, vors, divs, h):
    D, F, Xn, Yn, _ = stencils(case["levels"], case["degree"])
    n1 = case["degree"] + 1
    face, xi, eta = face_coordinates(x)
    X, Y = torch.tan(xi), torch.tan(eta)
    rho = (x[:, 0] ** 2 + x[:, 1] ** 2).sqrt()
    lon = (x[:, 0] * v[:, 1] - x[:, 1] * v[:, 0]) / rho
    col = ((x[:, 0] * v[:, 0] + x[:, 1] * v[:, 1]) * x[:, 2] - rho ** 2 * v[:, 2]) / rho
    C, E, s = (1 + X * X).sqrt(), (1 + Y * Y).sqrt(), (1 + X * X + Y * Y).sqrt()
    rr = 1 / (X * X + Y * Y).sqrt() * torch.where(face == 4, 1.0, -1.0)
    pole = x[:, 2].abs() >= 1 - 1e-16
    side = face <= 3
    a = torch.where(side, C * E / s * lon, rr * (E * X * col - E * Y / s * lon))
    b = torch.where(side, X * Y / s * lon - col, rr * (C * Y * col + C * X / s * lon))
    a, b = torch.where(pole, v[:, 0], a), torch.where(pole, v[:, 1], b)
    grid2 = lambda f: f.view(-1, n1, n1)  # noqa: E731
    dx = lambda f: torch.einsum("ij,pjk->pik", D, f)  # noqa: E731
    de = lambda f: torch.einsum("kj,pij->pik", D, f)  # noqa: E731
    fil = lambda f: (1 - 0.0005) * f + torch.einsum("ij,pjk->pik", F, f) + torch.einsum("kj,pij->pik", F, f)  # noqa: E731
    Xn, Yn = grid2(Xn), grid2(Yn)
    C2, E2, d2 = 1 + Xn * Xn, 1 + Yn * Yn, 1 + Xn * Xn + Yn * Yn
    Cn, En = C2.sqrt(), E2.sqrt()
    absvor = vors + 2 * OMEGA * x[:, 2]
    p, q = grid2(a * absvor), grid2(b * absvor)
    curl = -d2.sqrt() * (Xn * Yn / (Cn * En) * (de(q) / En - dx(p) / Cn) - de(p) / En + dx(q) / Cn)

    def lap(f):
        fx, fe = dx(f), de(f)
        return d2 * (dx(fx) / C2 + de(fe) / E2 + 2 * Xn * Yn / (C2 * E2) * 0.5 * (de(fx) + dx(fe)))

    hx, hy = grid2(h * a) / d2.sqrt(), grid2(h * b) / d2.sqrt()
    hdiv = d2 ** 1.5 / (Cn * En) * (dx(hx) / Cn + de(hy) / En)
    dt = (fil(curl) - fil(lap(grid2(h))) - fil(lap(grid2(0.5 * (v * v).sum(1))))).reshape(-1)
    flat = 1 - x[:, 2].abs() < 1e-5
    zero = torch.zeros_like(dt)
    return torch.stack([-divs * absvor - 2 * OMEGA * v[:, 2], torch.where(flat, zero, dt),
                        torch.where(flat, zero, hdiv.reshape(-1))], 1)


def swe_step(case, x, area, f, tracers, dt):
    where = stencils(case["levels"], case["degree"])[4]
    vors, divs, h = f
    v, T = [], []
    for hd, ht in ((0.0, 0.0), (0.5 * dt, 0.5 * dt), (0.5 * dt, 0.5 * dt), (dt, 0.5 * dt)):
        t = T[-1] if T else torch.zeros_like(x)
        y = unit(x + hd * v[-1]) if v else x
        u = BiotSavart.apply(x, y, area * (1 + ht * divs) * (vors + ht * t[:, 0]))
        u = u + divergent(x, x, area * (divs + ht * t[:, 1]))
        v.append(u if v else unify(u, where))
        if len(T) < 3:
            T.append(unify(tendencies(case, x, v[-1], vors, divs, h + ht * t[:, 2]), where))
    arrival = vors + dt * T[0][:, 0]
    p = departure(x, v, dt, case["levels"], case["degree"])
    fields = arrival[:, None] if tracers is None else torch.cat([arrival[:, None], tracers], 1)
    new = interpolate(p, fields, case["levels"], case["degree"])
    return [new[:, 0], divs + dt * T[0][:, 1], h + dt * T[0][:, 2]], new[:, 1:], v[0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "direct":
        t, s, w = scattered(case, seed)
        return tuple(BiotSavart.apply(cuda(t.T), cuda(s.T), cuda(w)).unbind(1))
    g = grid(case["levels"], case["degree"])
    shape = g["x"].shape
    x = torch.stack([a.reshape(-1) for a in on_gpu(case["levels"], case["degree"])[:3]], 1)
    area = cuda(g["area"].ravel())
    if kind == "adjoint":
        v, bar = (cuda(a.ravel()) for a in vortex(g, seed))
        v.requires_grad_()
        with torch.enable_grad():
            new = bve_step(case, x, area, v, None, ADJ_DT)[0]
            return torch.autograd.grad(new, v, bar)[0].view(shape)
    if kind == "poisson":
        w, m = area * cuda(smooth(g, np.random.default_rng(seed), 1.0).ravel()), rows(len(x))
        out = torch.empty_like(w)
        for k in range(0, len(x), m):
            d = torch.mm(x[k:k + m], x.T).neg_().add_(1.0)
            out[k:k + m] = -K4 * (torch.where(d > 1e-15, d, 1.0).log_() @ w)
        return out.view(shape)
    if kind == "ensemble":
        both = [bve_step(case, x, area, cuda(v.ravel()), None, DT) for v in members_of(case, seed)[2]]
        return dict(vors=torch.stack([b[0].view(shape) for b in both]),
                    vel=torch.stack([b[2].T.reshape((3,) + shape) for b in both]))
    tr = tracers_of(g, case["tracers"])
    tr = None if tr is None else cuda(tr).view(-1, case["tracers"])
    if kind == "bve":
        v = cuda(rossby_haurwitz(g, seed).ravel())
        for _ in range(case["steps"]):
            v, new, vel = bve_step(case, x, area, v, tr, DT)
            tr = None if tr is None else new
        out = dict(vors=v.view(shape))
    else:
        f = [cuda(a.ravel()) for a in balanced(g, seed)]
        where = stencils(case["levels"], case["degree"])[4]
        for _ in range(case["steps"]):
            f, new, vel = swe_step(case, x, area, f, tr, SWE_DT)
            tr = None if tr is None else new
            if case["call"] == "run":
                f = list(unify(torch.stack(f, 1), where).unbind(1))
        out = dict(fields=[a.view(shape) for a in f])
    out["vel"] = [a.view(shape) for a in vel.unbind(1)]
    if tr is not None:
        out["tracers"] = tr.view(shape + (case["tracers"],))
    return out
