"""The calls a program makes of this package, as cases that can be timed and compared.

A case is one evaluation of a built FMM: the points are fixed and the handle is kept, as a
solver's matrix-vector product, a time step on fixed geometry or a gradient step does, and
the charges are what changes.  `prepare` makes points and charges from a seed and builds
the handle; `run` is one call of a public entry point:

    device     Fmm.evaluate_device      device charges and outputs, on the handle's stream
    host       Fmm.evaluate             numpy charges and outputs (float64)
    host32     Fmm.evaluate             the same with float32 charges and outputs
    helmholtz  Fmm.helmholtz_evaluate_device
    vjp        Fmm.vjp                  gradients of the potentials (numpy)

`clouds` > 0 builds that many clouds of uneven sizes as one batch, `graph` replays the
device evaluation from a CUDA graph, `targets` > 0 is a target set of its own (0: the
targets are the sources).
"""
import math

import numpy as np
import torch

import fmm_b200 as F

SHAPES = ("cube", "sphere", "plummer", "gaussians")


def _case(name, call, shape, n, p, leaf, precision, *, vectors=1, gradients=True, targets=0, clouds=0, k=0.0,
          graph=False):
    c = {"call": call, "shape": shape, "n": n, "targets": targets, "clouds": clouds, "p": p, "leaf": leaf,
         "precision": precision, "vectors": vectors, "gradients": gradients, "k": k, "graph": graph}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small system solved by many products: launches and latency are all there is
        _case("small f64", "device", "cube", 2500, 4, 48, "f64", gradients=False, graph=True),
        # an ordinary particle step, small enough that the tree's levels are launch bound
        _case("particles mixed", "device", "plummer", 30011, 6, 64, "mixed", graph=True),
        # the plain f64 configuration: cube of 1e5, order 6, 64 a leaf, potentials
        _case("cube 1e5 f64", "device", "cube", 100000, 6, 64, "f64", gradients=False),
        # the published f64 configuration at 1e6: order 8, forces
        _case("cube 1e6 f64", "device", "cube", 1000000, 8, 64, "f64"),
        # several right-hand sides in f64 at a high order, sources and targets apart
        _case("apart f64 m4", "device", "sphere", 60013, 10, 80, "f64", vectors=4, targets=41017),
        # the same particles as 1e6 in mixed precision, through the host call in float32
        _case("cube 1e6 host32", "host32", "cube", 1000000, 8, 64, "mixed"),
        # the large surface configuration: 4e6 points on a sphere, order 8, 128 a leaf
        _case("sphere 4e6 mixed", "device", "sphere", 4000000, 8, 128, "mixed", graph=True),
        # the order that reaches 1e-6 on a surface
        _case("sphere 1e6 p11", "device", "sphere", 1000003, 11, 128, "mixed"),
        # many uneven clouds, 16 charge vectors each
        _case("batch m16 mixed", "device", "cube", 700001, 6, 64, "mixed", vectors=16, gradients=False, clouds=24,
              graph=True),
        # the Helmholtz kernel in both precisions
        _case("helmholtz mixed", "helmholtz", "cube", 200000, 10, 96, "mixed", k=20.0),
        _case("helmholtz f64", "helmholtz", "cube", 40009, 6, 96, "f64", k=8.0),
        # energy and forces of a clustered system, differentiated
        _case("vjp mixed", "vjp", "gaussians", 200000, 8, 64, "mixed"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(("device", "device", "device", "device", "host", "host32", "helmholtz", "batch", "vjp"))
    precision = rng.choice(("f64", "mixed"))
    shape = rng.choice(SHAPES)
    p = rng.randint(3, 11)
    leaf = rng.randint(32, 160)
    graph = rng.random() < 0.5
    gradients = rng.random() < 0.6
    if call == "batch":
        return _case(None, "device", shape, size(20000, 500000), rng.randint(3, 8), leaf, precision,
                     vectors=rng.choice((1, 3, 4, 8, 16)), gradients=False, clouds=rng.randint(2, 40), graph=graph)
    if call == "helmholtz":
        f64 = precision == "f64"
        return _case(None, call, shape, size(3000, 60000 if f64 else 200000), rng.randint(4, 8 if f64 else 10), leaf,
                     precision, gradients=gradients, k=round(rng.uniform(1.0, 20.0), 3))
    if call == "vjp":
        return _case(None, call, shape, size(3000, 300000), min(p, 9), leaf, precision)
    vectors = rng.choice((1, 1, 1, 2, 3, 4)) if call == "device" else 1
    n = size(1000, (400000 if precision == "f64" else 1500000) // vectors)
    targets = size(1000, n) if n > 2000 and rng.random() < 0.3 else 0
    return _case(None, call, shape, n, p, leaf, precision, vectors=vectors, gradients=gradients, targets=targets,
                 graph=graph and call == "device")


# ---- inputs --------------------------------------------------------------------------


def _points(shape, n, rng):
    if shape == "cube":
        return rng.random((n, 3))
    if shape == "sphere":
        x = rng.standard_normal((n, 3))
        return x / np.linalg.norm(x, axis=1, keepdims=True)
    if shape == "plummer":  # scale radius 0.1, cut at r = 5
        u = rng.random(n) * (1.0 + 0.02 ** 2) ** -1.5
        r = 0.1 / np.sqrt(np.maximum(u, 1e-12) ** (-2.0 / 3.0) - 1.0)
        x = rng.standard_normal((n, 3))
        return x * (np.minimum(r, 5.0) / np.linalg.norm(x, axis=1))[:, None]
    centres = rng.random((32, 3))  # 32 Gaussians, sigma log-uniform in [0.005, 0.05]
    sigma = 0.005 * 10.0 ** rng.random(32)
    g = rng.integers(0, 32, n)
    return centres[g] + sigma[g, None] * rng.standard_normal((n, 3))


def _cloud_sizes(case):
    """Sizes of a batch's clouds: log-uniform over a factor 50, the same for every seed."""
    rng = np.random.default_rng(case["n"] * 64 + case["clouds"])
    w = 50.0 ** rng.random(case["clouds"])
    return np.maximum(1, (w / w.sum() * case["n"]).astype(np.int64)).tolist()


def _inputs(case, seed):
    """(clouds of sources, targets or None, charges (ns, m), cotangent or None) on the host."""
    rng = np.random.default_rng([seed, case["n"], case["p"]])
    if case["clouds"]:
        shapes = [SHAPES[i % 3] for i in range(case["clouds"])]
        clouds = [_points(s, c, rng) for s, c in zip(shapes, _cloud_sizes(case))]
    else:
        clouds = [_points(case["shape"], case["n"], rng)]
    targets = _points(case["shape"], case["targets"], rng) if case["targets"] else None
    ns = sum(len(c) for c in clouds)
    nt = len(targets) if targets is not None else ns
    m = case["vectors"]
    q = rng.standard_normal((ns, m))
    if case["call"] == "helmholtz":
        q = q + 1j * rng.standard_normal((ns, m))
    if case["call"] == "host32":
        q = q.astype(np.float32)
    w = rng.standard_normal((m, nt)) if case["call"] == "vjp" else None
    return clouds, targets, q, w


def prepare(case, seed):
    clouds, targets, q, w = _inputs(case, seed)
    b = (F.FmmBuilder(case["p"]).vectors(case["vectors"]).max_points_per_leaf(case["leaf"])
         .gradients(case["gradients"]).precision(case["precision"]))
    fmm = b.build_batch(clouds) if case["clouds"] else b.build(clouds[0], targets)
    s = {"call": case["call"], "fmm": fmm, "k": case["k"], "q": q, "w": w}
    if case["call"] in ("device", "helmholtz"):
        dtype = torch.complex128 if case["call"] == "helmholtz" else torch.float64
        m, nt = case["vectors"], fmm.ntargets
        s["q"] = torch.from_numpy(q).cuda()
        s["potential"] = torch.zeros((m, nt), dtype=dtype, device="cuda")
        s["gradient"] = torch.zeros((m, nt, 3), dtype=dtype, device="cuda") if case["gradients"] else None
        torch.cuda.synchronize()
        if case["graph"]:
            fmm.set_graph(True)
        if case["call"] == "helmholtz":  # the first call of a wavenumber builds its tables
            run(s)
            fmm.synchronize()
    return s


def run(state):
    call, fmm = state["call"], state["fmm"]
    if call in ("device", "helmholtz"):
        q, phi, g = state["q"], state["potential"], state["gradient"]
        gp = None if g is None else g.data_ptr()
        if call == "device":  # work that reads the outputs is ordered after fmm.stream
            fmm.evaluate_device(q.data_ptr(), phi.data_ptr(), gp)
        else:
            fmm.helmholtz_evaluate_device(state["k"], q.data_ptr(), phi.data_ptr(), gp)
        return {"potential": phi} if g is None else {"potential": phi, "gradient": g}
    if call == "vjp":
        dq, dxs, dxt = fmm.vjp(state["q"], state["w"])
        return {"dcharges": dq, "dsources": dxs, "dtargets": dxt}
    out = fmm.evaluate(state["q"])
    return {"potential": out.potential} if out.gradient is None else {"potential": out.potential,
                                                                      "gradient": out.gradient}


# ---- what a pass needs ---------------------------------------------------------------


def work(case):
    """Inputs read once and outputs written once; the operations of the fast multipole
    method at the case's order and leaf size: near pairs (27 leaf neighbours in a volume,
    about 11 on a surface or in a cluster, leaves about 0.4 full), dense translations
    (189 or about 30 a box) and leaf expansions."""
    n, m, nc = case["n"], case["vectors"], (case["p"] + 1) ** 2
    nt = case["targets"] or n
    z = 2 if case["call"] == "helmholtz" else 1
    size = 4 if case["call"] == "host32" else 8
    comps = 4 if case["gradients"] else 1
    fill = 0.4 * case["leaf"]
    volume = case["shape"] == "cube" and not case["clouds"]
    near, vlist = (27, 189) if volume else (11, 30)
    boxes = max(1.0, 1.15 * n / fill)
    pair = (15 if case["gradients"] else 10) * (2 if z == 2 else 1)
    flops = nt * min(n, near * fill) * pair * m + boxes * vlist * 2 * nc * nc * m * z * z
    flops += (n + nt * comps) * 4 * nc * m * z
    nbytes = 24 * (n + case["targets"]) + size * z * m * (n + comps * nt)
    if case["call"] == "vjp":  # the forward gradients, the transpose pass, and their products
        flops *= 2
        nbytes = 24 * n + 8 * (m * (2 * n + 2 * nt) + 3 * (n + nt))
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    # measured against the same evaluation with its sums in another order (the points
    # permuted, so every leaf sums its own in another order): f64 up to 7.3e-16, 3.9e-15 at
    # one value; mixed (f32 expansions and pairs, f64 sums a target) up to 2.6e-7, 3.8e-6 at
    # one value.  Each bound is at least four times that.
    if case["precision"] == "f64":
        return {"rel": 5e-15, "max": 3e-14}
    return {"rel": 1e-6, "max": 2e-5}


# ---- the same numbers in plain torch, 64 bits ------------------------------------------


def _kernel_sums(src, tgt, q, k, gradients):
    """sum_j G(t - s_j) q_j and its gradient at t: (m, nt) and (m, nt, 3); coincident pairs
    left out.  src, tgt, q on the GPU."""
    m = q.shape[1]
    phi = torch.zeros((m, len(tgt)), dtype=q.dtype, device="cuda")
    g = torch.zeros((m, len(tgt), 3), dtype=q.dtype, device="cuda") if gradients else None
    step = max(1, int(4e7) // len(src))
    for a in range(0, len(tgt), step):
        t = tgt[a:a + step]
        d = [t[:, i, None] - src[None, :, i] for i in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        inv = torch.where(r2 > 0, r2.rsqrt(), torch.zeros_like(r2))
        del r2
        if k:
            r = torch.where(inv > 0, 1.0 / inv, torch.zeros_like(inv))
            wave = torch.polar(inv, k * r)
        else:
            wave = inv
        phi[:, a:a + step] = (wave @ q).T
        if gradients:
            rad = wave * (torch.complex(-torch.ones_like(inv), k * r) if k else -1.0) * (inv * inv)
            for i in range(3):
                g[:, a:a + step, i] = ((rad * d[i]) @ q).T
    f = 1.0 / (4.0 * math.pi)
    return phi * f, None if g is None else g * f


def exact(case, seed):
    n, nt, m = case["n"], case["targets"] or case["n"], case["vectors"]
    pairs = sum(c * c for c in _cloud_sizes(case)) if case["clouds"] else n * nt
    weight = (2 if case["call"] == "vjp" else 1) * (3 if case["call"] == "helmholtz" else 1) * (1 + m / 8)
    if pairs * weight > 1.2e11:
        return None
    clouds, targets, q, w = _inputs(case, seed)
    wide = np.complex128 if case["call"] == "helmholtz" else np.float64
    qd = torch.from_numpy(np.ascontiguousarray(q.astype(wide))).cuda()
    src = [torch.from_numpy(c).cuda() for c in clouds]
    tgt = [torch.from_numpy(targets).cuda()] if targets is not None else src
    if case["call"] == "vjp":
        wd = torch.from_numpy(w).cuda()
        _, grad = _kernel_sums(src[0], tgt[0], qd, 0.0, True)
        psi, gpsi = _kernel_sums(tgt[0], src[0], wd.T.contiguous(), 0.0, True)
        return {"dcharges": psi.T.contiguous().cpu().numpy(),
                "dsources": (qd.T[:, :, None] * gpsi).sum(0).cpu().numpy(),
                "dtargets": (wd[:, :, None] * grad).sum(0).cpu().numpy()}
    phis, grads, at = [], [], 0
    for s, t in zip(src, tgt):
        phi, g = _kernel_sums(s, t, qd[at:at + len(s)], case["k"], case["gradients"])
        at += len(s)
        phis.append(phi)
        grads.append(g)
    out = {"potential": torch.cat(phis, dim=1)}
    if case["gradients"]:
        out["gradient"] = torch.cat(grads, dim=1)
    if case["call"] in ("host", "host32"):
        out = {k: v.cpu().numpy() for k, v in out.items()}
    return out
