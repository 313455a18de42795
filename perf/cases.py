"""Performance cases: the work users have this library do, through its public entry points.

Four kinds of pass, each on seeded synthetic inputs made on the GPU:

* ``step``   one new permeability field on a known mesh: set_kappa, setup, rhs, solve (what
             ``bench.py`` times and what ``run_case.py`` does once).  The solver object is kept from
             field to field, as a time loop or a Monte-Carlo run keeps it.
* ``solve``  one more right-hand side on a finished set-up.
* ``batch``  independent problems of different sizes set up and solved together, several right-hand
             sides each (``BatchSolver``).
* ``apply``  one operator product (the MatMult of a caller that runs its own Krylov method).
* ``train``  one training batch of the learned start's network: forward, loss, backward, and the
             gradients of every layer.

Solutions are asked for at a relative residual of 1e-12 (1e-10 on the large anisotropic field, the default
1e-8 on the layered one, where 64-bit residuals level off near 1e-10).  On the fracture fields the contrast is 1e8 and a
residual of 1e-8 leaves the solution's sixth digit to the path of the iteration; at 1e-12 the solution
itself is fixed to about 1e-10, so a caller who compares or differentiates solutions asks for that.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from premixfem_b200 import learned
from premixfem_b200.solver import BatchSolver, DarcySolver, options_string

RTOL = {"large": 1e-10, "layered": 1e-8}  # others 1e-12

# field -> (unit cells or unit cube, Dirichlet faces, volume source)
FIELDS = {
    "grf": ("cube", {"x+": 0.0}, "unit"),        # lognormal, sigma 2, correlation 0.1
    "box": ("cube", {"x-": 0.0}, "noise"),       # mild lognormal, N(0,1) source
    "fracture": ("cells", {"x-": 1.0, "x+": 0.0}, None),  # 1e4 fractures, 1e-4 barriers
    "large": ("cube", {"z-": 0.0}, "unit"),      # anisotropic lognormal sigma 3, 1e6 fractures
    "layered": ("spe", {}, "wells"),             # lognormal layers over 1e6 channels, no-flux walls
}


def listed():
    fr = {"field": "fracture", "tile": 16, "en1": 6, "en2": 4}
    return [
        # the smallest workload of the benchmark configurations: 32^3 lognormal field in 8^3 subdomains on
        # one rank, plain FP64; launches and host round trips count
        {"name": "grf32_step", "kind": "step", "field": "grf", "M": 32, "N": 32, "P": 32, "tile": 8,
         "en1": 4, "en2": 4, "precision": "fp64"},
        # another right-hand side on a small odd-sized box with ragged subdomains, W-cycle
        {"name": "box45x37x29_solve", "kind": "solve", "field": "box", "M": 45, "N": 37, "P": 29, "tile": 11,
         "en1": 4, "en2": 4, "precision": "mixed", "extra": "-use_W_cycle -si_lv2 2"},
        # the headline workload at half its edge: fracture network, mixed form, learned start
        dict(fr, name="fracture128_step", kind="step", M=128, N=128, P=128, precision="mixed", learned=True),
        # the headline workload: 16.7 M cells, 4 096 subdomains
        dict(fr, name="fracture256_step", kind="step", M=256, N=256, P=256, precision="mixed", learned=True),
        # more right-hand sides on the headline set-up (time steps, sensitivities)
        dict(fr, name="fracture256_solve", kind="solve", M=256, N=256, P=256, precision="mixed"),
        # a mesh that 16 does not divide, plain FP64: subdomains of 12 and 13 cells per axis
        dict(fr, name="fracture150_fp64_step", kind="step", M=150, N=150, P=150, precision="fp64", tile=13),
        # plain FP64 solve at a size of its own (the comparator of the benchmark's metric)
        dict(fr, name="fracture192_fp64_solve", kind="solve", M=192, N=192, P=192, precision="fp64"),
        # the SPE10-shaped layered field: pure Neumann with the constant null space, 60 x 220 x 85 cells
        {"name": "layered_step", "kind": "step", "field": "layered", "M": 60, "N": 220, "P": 85,
         "vranks": "2,2,1", "sd": "3,11,17", "en1": 4, "en2": 4, "precision": "fp64", "extra": "-ksp_constant_null_space"},
        # the large anisotropic field's options (eight vectors per subdomain) on 8.4 M cells
        {"name": "large_k8_step", "kind": "step", "field": "large", "M": 256, "N": 256, "P": 128, "tile": 16,
         "en1": 8, "en2": 4, "precision": "mixed"},
        # many small problems at once: 16 unit cubes of 24..80 cells per axis, four right-hand sides each
        {"name": "batch16", "kind": "batch", "count": 16, "lo": 24, "hi": 80, "rhs": 4, "en1": 4, "en2": 4,
         "precision": "mixed"},
        # the operator alone, for a caller's own Krylov method
        dict(fr, name="apply256", kind="apply", M=256, N=256, P=256, precision="mixed", en1=2, en2=2),
        # one training batch of the learned start (the batch size of learned.train)
        {"name": "train64", "kind": "train", "count": 64},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "solve", "solve", "batch", "apply", "train"])
    if kind == "train":
        return {"kind": "train", "count": rng.randint(8, 64)}
    if kind == "batch":
        hi = rng.randint(32, 80)
        return {"kind": "batch", "count": rng.randint(2, 16), "lo": 24, "hi": hi, "rhs": rng.randint(1, 4),
                "en1": rng.randint(3, 4), "en2": 4, "precision": rng.choice(["mixed", "fp64"])}
    field = rng.choice(["grf", "box", "fracture", "fracture", "large"])
    cells = _log_uniform(rng, 20, 200) ** 3
    shape = [rng.uniform(0.7, 1.4) for _ in range(3)]
    e = (cells / (shape[0] * shape[1] * shape[2])) ** (1.0 / 3.0)
    M, N, P = (min(256, max(18, int(round(s * e)))) for s in shape)
    if rng.random() < 0.4:  # the aligned shapes that configurations favour
        M, N, P = (max(16, 16 * int(round(v / 16.0))) for v in (M, N, P))
    c = {"kind": kind, "field": field, "M": M, "N": N, "P": P, "tile": rng.choice([8, 12, 13, 16, 16]),
         "en1": rng.choice([4, 4, 6, 6, 8]), "en2": 4, "precision": rng.choice(["mixed", "mixed", "fp64"])}
    if kind == "apply":
        c.update(en1=2, en2=2)
    if kind == "step" and field == "fracture" and c["precision"] == "mixed" and c["tile"] == 16:
        c.update(en1=6, learned=True)
    elif rng.random() < 0.25:
        c["extra"] = rng.choice(["-use_W_cycle", "-si_lv1 2", "-si_lv2 2", "-use_2level", "-eg_op 1", "-no_shift_A_cc"])
        if c["extra"] == "-use_2level" and M * N * P > 130 ** 3:
            c["extra"] = "-use_W_cycle"
    return c


# ---------------------------------------------------------------------------
# inputs

def _gen(seed, stream=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * stream + seed)


def _grf(shape, spacing, sigma, corr, seed, stream=0, embed=1):
    """Gaussian random field, exponential covariance, on a periodic grid ``embed`` times the domain."""
    ext = [max(2, s * embed) for s in shape]
    d = [torch.minimum(torch.arange(n, device="cuda", dtype=torch.float64),
                       n - torch.arange(n, device="cuda", dtype=torch.float64)) * h / c
         for n, h, c in zip(ext, spacing, corr)]
    r = torch.sqrt(d[0][:, None, None] ** 2 + d[1][None, :, None] ** 2 + d[2][None, None, :] ** 2)
    lam = torch.fft.rfftn(torch.exp(-r)).real.clamp_(min=0.0)
    w = torch.randn(ext, dtype=torch.float64, device="cuda", generator=_gen(seed, stream))
    f = torch.fft.irfftn(torch.fft.rfftn(w) * torch.sqrt(lam), s=ext)[:shape[0], :shape[1], :shape[2]]
    return sigma * (f - f.mean()) / f.std()


def _fractures(k, rng, count, lo, hi, value):
    """Axis-aligned one-cell-thick rectangles of in-plane extent U{lo..hi}."""
    dims = k.shape
    for _ in range(count):
        normal = int(rng.integers(0, 3))
        sl = [None, None, None]
        for a in range(3):
            n = 1 if a == normal else min(int(rng.integers(lo, hi + 1)), dims[a])
            s = int(rng.integers(0, dims[a] - n + 1))
            sl[a] = slice(s, s + n)
        k[tuple(sl)] = value


def _barriers(k, rng, share, value, lo=2, hi=6):
    """Boxes of 2..6 cells per axis until about ``share`` of the cells are covered."""
    count = max(1, int(share * k.numel() / (0.5 * (lo + hi)) ** 3))
    size = torch.from_numpy(rng.integers(lo, hi + 1, size=(count, 3))).cuda()
    at = torch.from_numpy(rng.integers(0, 1 << 30, size=(count, 3))).cuda()
    dims = torch.tensor(k.shape, device="cuda")
    at = at % (dims - size).clamp(min=1)
    o = torch.stack(torch.meshgrid(*[torch.arange(hi, device="cuda")] * 3, indexing="ij"), -1).reshape(1, -1, 3)
    inside = (o < size[:, None]).all(-1)
    c = torch.minimum(at[:, None] + o, dims - 1)
    flat = (c[..., 0] * dims[1] + c[..., 1]) * dims[2] + c[..., 2]
    k.view(-1)[flat[inside]] = value


def _layered(M, N, P, seed):
    """Lognormal layers on top (35 of 85), sinuous channels of contrast 1e6 below."""
    smooth = P * 35 // 85
    rng = np.random.default_rng(seed)
    k = torch.empty((P, N, M), dtype=torch.float64, device="cuda")
    for z in range(smooth):
        k[z] = torch.exp(_grf((1, N, M), (1.0,) * 3, 1.5, (1.0, 8.0, 8.0), seed, stream=1 + z, embed=2)[0])
    xs, yy = np.arange(M), np.arange(N)
    for z in range(smooth, P):
        mask = np.zeros((N, M), dtype=bool)
        for _ in range(int(rng.integers(3, 7))):
            c = rng.uniform(0, M) + rng.uniform(2, 10) * np.sin(2 * np.pi * yy / rng.uniform(30, 120)
                                                                + rng.uniform(0, 2 * np.pi))
            mask |= np.abs(xs[None, :] - c[:, None]) < int(rng.integers(3, 7)) / 2.0
        k[z] = torch.from_numpy(np.where(mask, 1e3, 1e-3)).cuda()
    return k


def _kappa(case, seed):
    M, N, P = case["M"], case["N"], case["P"]
    shape = (P, N, M)
    rng = np.random.default_rng(seed)
    f = case["field"]
    if f == "layered":
        return _layered(M, N, P, seed)
    if f == "fracture":
        n = min(shape)
        k = torch.exp(_grf(shape, (1.0,) * 3, 0.5, (8.0,) * 3, seed))
        _fractures(k, rng, 200, max(2, 32 * n // 256), max(3, 160 * n // 256), 1e4)
        _barriers(k, rng, 0.05, 1e-4)
        return k
    h = (1.0 / P, 1.0 / N, 1.0 / M)
    if f == "large":
        k = torch.exp(_grf(shape, h, 3.0, (0.02, 0.1, 0.1), seed))
        n = max(shape)
        _fractures(k, rng, max(1, 400 * n * n // (512 * 512)), max(2, n // 16), max(3, n // 2), 1e6)
        return k
    sigma, corr = (2.0, 0.1) if f == "grf" else (1.0, 0.2)
    return torch.exp(_grf(shape, h, sigma, (corr,) * 3, seed, embed=2))


def _domain(case):
    M, N, P = case["M"], case["N"], case["P"]
    return {"cells": (float(M), float(N), float(P)), "cube": (1.0, 1.0, 1.0),
            "spe": (20.0 * M, 10.0 * N, 2.0 * P)}[FIELDS[case["field"]][0]]


def _source(case, seed):
    M, N, P = case["M"], case["N"], case["P"]
    kind = FIELDS[case["field"]][2]
    s = torch.zeros((P, N, M), dtype=torch.float64, device="cuda")
    if kind == "unit":
        s.fill_(1.0 / (M * N * P))
    elif kind == "noise":
        s = torch.randn((P, N, M), dtype=torch.float64, device="cuda", generator=_gen(seed, 91)) / (M * N * P)
    elif kind == "wells":
        s[:, 0, 0] = 1.0 / P
        s[:, N - 1, M - 1] = -1.0 / P
    if case["kind"] == "solve" and kind != "noise":  # another right-hand side: wells of its own
        rng = np.random.default_rng(seed + 7)
        for sign in (1.0, -1.0):
            s[:, int(rng.integers(0, N)), int(rng.integers(0, M))] += sign * (1.0 if kind is None else 1.0 / P)
    return s.reshape(-1)


def _options(case):
    """Subdomains of about ``tile`` cells per axis, at most four per virtual rank and axis."""
    o = {"en_lv1": case["en1"], "en_lv2": case["en2"], "pmf_precision": case["precision"], "ksp_rtol": RTOL.get(case.get("field"), 1e-12)}
    if case.get("vranks"):
        o["pmf_vranks"], o["pmf_sd"] = case["vranks"], case["sd"]
    elif case["kind"] != "batch":
        v, s = [], []
        for n in (case["M"], case["N"], case["P"]):
            subs = max(2, -(-n // case["tile"]))
            v.append(-(-subs // 4))
            s.append(-(-subs // v[-1]))
        o["pmf_vranks"], o["pmf_sd"] = tuple(v), tuple(s)
    if case.get("learned"):
        o["pmf_learned"] = learned.DEFAULT_WEIGHTS
    return options_string(o) + (" " + case["extra"] if case.get("extra") else "")


def _batch_problems(case, seed):
    """The problems' meshes belong to the case (they set its size), the fields and sources to the seed."""
    sizes = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    rng = np.random.default_rng(seed)
    probs, srcs = [], []
    for q in range(case["count"]):
        M, N, P = (int(v) for v in sizes.integers(case["lo"], case["hi"] + 1, size=3))
        c = rng.uniform(0.05, 0.2)
        k = torch.exp(_grf((P, N, M), (1.0 / P, 1.0 / N, 1.0 / M), rng.uniform(1.0, 3.0), (c,) * 3, seed,
                           stream=100 + q, embed=2))
        probs.append({"dom": (1.0, 1.0, 1.0), "mesh": (M, N, P), "dirichlet": {"x+": 0.0}, "kappa": k})
        g = _gen(seed, 1000 + q)
        meas = 1.0 / (M * N * P)
        srcs.append([torch.full((P, N, M), meas, dtype=torch.float64, device="cuda")] +
                    [torch.randn((P, N, M), dtype=torch.float64, device="cuda", generator=g) * meas
                     for _ in range(case["rhs"] - 1)])
    return probs, srcs


def _pack(s, arrays):
    M, N, P = s.mesh
    out = torch.zeros((P, N, M), dtype=torch.float64, device="cuda")
    for (m, n, p), z0, a in zip(s.meshes, s.z0, arrays):
        out[z0:z0 + p, :n, :m] = a
    return out.reshape(-1)


def _train_inputs(case, seed):
    """Patches as the set-up makes them: log-permeability minus its mean over four, the masks, and smooth
    orthonormal target vectors (the shape of a subdomain's lowest modes)."""
    B = case["count"]
    g = _gen(seed, 5)
    ax = (torch.arange(16, device="cuda") + 0.5) / 16.0
    x = torch.zeros((B, 16, 16, 16, learned.CH), device="cuda")
    logk = 0.5 * torch.randn((B, 4, 4, 4), device="cuda", generator=g)
    logk = torch.nn.functional.interpolate(logk[:, None], size=(16, 16, 16), mode="trilinear")[:, 0]
    for b in range(B):  # a fracture plane and a barrier in most patches
        p = [int(v) for v in torch.randint(0, 16, (4,), device="cuda", generator=g).tolist()]
        if p[0] < 10:
            logk[b].transpose(0, p[1] % 3)[p[2]] = math.log(1e4)
        if p[3] < 12:
            logk[b, p[3]:p[3] + 4, p[2] % 12:p[2] % 12 + 3, p[1] % 12:p[1] % 12 + 3] = math.log(1e-4)
    x[..., :3] = ((logk - logk.mean((1, 2, 3), keepdim=True)) / 4.0)[..., None]
    x[..., 4] = 1.0
    modes = []
    for a, b_, c in ((0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (0, 1, 1)):
        modes.append(torch.cos(math.pi * a * ax)[None, None, :] * torch.cos(math.pi * b_ * ax)[None, :, None] *
                     torch.cos(math.pi * c * ax)[:, None, None])
    v = torch.stack(modes, -1).reshape(1, learned.VOX, 6).double()
    v = v * (1.0 + 0.3 * torch.tanh(logk.reshape(B, learned.VOX, 1).double())) + \
        0.05 * torch.randn((B, learned.VOX, 6), device="cuda", generator=g, dtype=torch.float64)
    m = torch.exp(0.2 * logk.reshape(B, learned.VOX).double()).clamp(0.1, 10.0)
    q, _ = torch.linalg.qr(torch.sqrt(m)[..., None] * v)
    v = q / torch.sqrt(m)[..., None]
    return (x.reshape(B, learned.VOX, learned.CH).to(torch.bfloat16).contiguous(), v.float().contiguous(),
            m.float().contiguous())


# ---------------------------------------------------------------------------
# preparation and one pass

def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, v, m = _train_inputs(case, seed)
        y = torch.empty((case["count"], learned.VOX, learned.CH), dtype=torch.float32, device="cuda")
        return {"kind": kind, "net": learned.Net(path=learned.DEFAULT_WEIGHTS), "x": x, "V": v, "M": m, "y": y,
                "dy": torch.empty_like(y), "loss": torch.empty(case["count"], device="cuda")}
    if kind == "batch":
        probs, srcs = _batch_problems(case, seed)
        s = BatchSolver(probs, [tuple(max(2, -(-n // 8)) for n in p["mesh"]) for p in probs], _options(case))
        return {"kind": kind, "s": s, "k": _pack(s, [p["kappa"] for p in probs]),
                "src": [_pack(s, [v[i] for v in srcs]) for i in range(case["rhs"])]}
    k = _kappa(case, seed).reshape(-1)
    s = DarcySolver(_domain(case), (case["M"], case["N"], case["P"]), _options(case))
    for face, value in FIELDS[case["field"]][1].items():
        s.set_dirichlet(face, value)
    src = _source(case, seed)
    torch.cuda.synchronize()
    if kind == "step":
        return {"kind": kind, "s": s, "k": k, "src": src}
    s.set_kappa(k, k, k)
    s.setup()
    if kind == "apply":
        return {"kind": kind, "s": s,
                "x": torch.randn(s.n, dtype=torch.float64, device="cuda", generator=_gen(seed, 17))}
    return {"kind": kind, "s": s, "b": s.rhs(src)}


def run(state):
    kind = state["kind"]
    if kind == "train":
        net = state["net"]
        net.forward(state["x"], state["y"])
        learned.loss_and_grad(state["y"], state["V"], state["M"], 6, state["loss"], state["dy"])
        net.backward(state["dy"])
        return {"y": state["y"], "loss": state["loss"], "grads": [net.grads(i) for i in range(9)]}
    s = state["s"]
    if kind == "apply":
        return s.apply_A(state["x"])
    if kind == "solve":
        return s.solve(state["b"])[0]
    s.set_kappa(state["k"], state["k"], state["k"])
    s.setup()
    if kind == "batch":
        return [s.solve(s.rhs(src))[0] for src in state["src"]]
    return s.solve(s.rhs(state["src"]))[0]


# ---------------------------------------------------------------------------
# what a pass cannot do without

# iterations that the method itself needs on these fields (typical counts: conjugate gradients to the residuals above, local
# eigensolves from a random and from the learned start)
PCG_ITS = {"grf": 30, "box": 25, "fracture": 100, "large": 220, "layered": 240}
EIG_ITS, EIG_ITS_LEARNED = 28, 22


def _eig_work(n, m, w, its):
    # per iteration: the basis (3m columns) and the operator read, the block and its directions (2m) written
    return its * n * (5.0 * m * w + 40.0), its * n * (4.0 * 3 * m * 3 * m + 60.0 * m)


def _solve_work(n, k, w, its, levels):
    # CG: z, p, four operator arrays, p, w, x, r; cycle: two level-1 visits per side, restriction, prolongation
    return its * n * (112.0 + 24.0 + w * (12.0 + 2.0 * k)) * levels, its * n * (60.0 + 8.0 * k)


def work(case):
    kind = case["kind"]
    if kind == "train":
        flops = 2.0 * 4096 * (27 * 16 * 32 + 27 * 32 * 32 + 32 * 16 + 64 * 32) + \
            2.0 * 512 * (8 * 32 * 64 + 27 * 64 * 64 + 96 * 64) + 2.0 * 64 * (8 * 64 * 96 + 27 * 96 * 96)
        return {"bytes": case["count"] * 4096.0 * (2 * 16 + 4 * 16 * 3 + 4 * 6 + 4) + 532976 * 6.0,
                "flops": 3.0 * case["count"] * flops}
    if kind == "batch":
        sizes = np.random.default_rng([case["count"], case["lo"], case["hi"]])
        n = float(sum(np.prod(sizes.integers(case["lo"], case["hi"] + 1, size=3)) for _ in range(case["count"])))
        field, solves = "box", case["rhs"]
    else:
        n, field, solves = float(case["M"] * case["N"] * case["P"]), case["field"], 1
    if kind == "apply":
        return {"bytes": 48.0 * n, "flops": 13.0 * n}
    w = 4.0 if case["precision"] == "mixed" else 8.0
    levels = 2 if "-si_lv1 2" in case.get("extra", "") else 1
    b, f = _solve_work(n, case["en1"], w, solves * PCG_ITS[field], levels)
    if kind != "solve":
        eb, ef = _eig_work(n, case["en1"] + 2, w, EIG_ITS_LEARNED if case.get("learned") else EIG_ITS)
        b, f = b + eb + n * 24.0, f + ef
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the results in 64 bits, without the library

def _operator(k, dom, dirichlet):
    """Face transmissibilities (low side of each cell), diagonal and boundary right-hand side, (z, y, x)."""
    P, N, M = k.shape
    h = (dom[2] / P, dom[1] / N, dom[0] / M)
    vol = h[0] * h[1] * h[2]
    t, diag, rhs = [], torch.zeros_like(k), torch.zeros_like(k)
    for a in range(3):
        f = (vol / h[a]) ** 2 / vol
        lo, hi = k.narrow(a, 0, k.shape[a] - 1), k.narrow(a, 1, k.shape[a] - 1)
        ta = torch.zeros_like(k)
        ta.narrow(a, 1, k.shape[a] - 1).copy_(f * 2.0 / (1.0 / lo + 1.0 / hi))
        diag += ta
        diag.narrow(a, 0, k.shape[a] - 1).add_(ta.narrow(a, 1, k.shape[a] - 1))
        t.append(ta)
        for end, face in ((0, "zyx"[a] + "-"), (k.shape[a] - 1, "zyx"[a] + "+")):
            if face in dirichlet:
                tb = f * 2.0 * k.narrow(a, end, 1)
                diag.narrow(a, end, 1).add_(tb)
                rhs.narrow(a, end, 1).add_(tb * dirichlet[face])
    return t, diag, rhs


def _matvec(t, diag, x):
    y = diag * x
    for a in range(3):
        n = x.shape[a] - 1
        ta = t[a].narrow(a, 1, n)
        y.narrow(a, 1, n).sub_(ta * x.narrow(a, 0, n))
        y.narrow(a, 0, n).sub_(ta * x.narrow(a, 1, n))
    return y


def _block_solver(k, dom, dirichlet):
    """Block elimination along the longest axis: Cholesky factors of the planes' Schur complements.
    Returns solve(b)."""
    t, diag, _ = _operator(k, dom, dirichlet)
    ax = int(np.argmax(k.shape))
    order = (ax, *[a for a in range(3) if a != ax])
    tp = [t[a].permute(order).contiguous() for a in order]
    dp = diag.permute(order).contiguous()
    L, n1, n2 = dp.shape
    n = n1 * n2
    idx = torch.arange(n, device=k.device).reshape(n1, n2)
    fac, inv = [], None
    for i in range(L):
        S = torch.zeros((n, n), dtype=torch.float64, device=k.device)
        S.view(-1)[torch.arange(n, device=k.device) * (n + 1)] = dp[i].reshape(-1)
        for ta, p, q in ((tp[1][i][1:], idx[1:], idx[:-1]), (tp[2][i][:, 1:], idx[:, 1:], idx[:, :-1])):
            S[p.reshape(-1), q.reshape(-1)] = -ta.reshape(-1)
            S[q.reshape(-1), p.reshape(-1)] = -ta.reshape(-1)
        if i:
            c = tp[0][i].reshape(-1)
            S -= c[:, None] * inv * c[None, :]
        fac.append(torch.linalg.cholesky(S))
        if i + 1 < L:
            inv = torch.cholesky_inverse(fac[-1])

    def once(b):
        bp = b.permute(order).reshape(L, n, 1).clone()
        for i in range(1, L):
            bp[i] += tp[0][i].reshape(-1, 1) * torch.cholesky_solve(bp[i - 1], fac[i - 1])
        x = torch.empty_like(bp)
        x[L - 1] = torch.cholesky_solve(bp[L - 1], fac[L - 1])
        for i in range(L - 2, -1, -1):
            x[i] = torch.cholesky_solve(bp[i] + tp[0][i + 1].reshape(-1, 1) * x[i + 1], fac[i])
        back = [order.index(a) for a in range(3)]
        return x.reshape(L, n1, n2).permute(back).contiguous()

    def solve(b):
        x = once(b)
        for _ in range(4):
            x = x + once(b - _matvec(t, diag, x))
        return x

    return solve


def _block_cost(mesh):
    a, b, c = sorted(mesh)
    return 3.0 * c * float(a * b) ** 3, 8.0 * c * float(a * b) ** 2  # operations, bytes of the factors


def _bf(a):
    return a.to(torch.bfloat16).to(torch.float64)


class _Round(torch.autograd.Function):
    """Activations are stored in BF16; gradients pass as they are."""

    @staticmethod
    def forward(ctx, a):
        return _bf(a)

    @staticmethod
    def backward(ctx, g):
        return g


def _exact_train(case, seed):
    """The network in 64 bits with its BF16 weights and activations, the subspace loss, and the gradients."""
    x, V, Mw = _train_inputs(case, seed)
    net = learned.Net(path=learned.DEFAULT_WEIGHTS)
    B = case["count"]
    W, b = [], []
    for i in range(9):
        w_, b_ = net.weights(i)
        W.append(_bf(torch.from_numpy(w_).cuda()).requires_grad_())
        b.append(torch.from_numpy(b_).cuda().double().requires_grad_())
    net.close()
    layers = [("c3", 16, -1), ("d2", 16, -1), ("c3", 8, -1), ("d2", 8, -1), ("c3", 4, -1), ("u2", 4, 3),
              ("u2", 8, 1), ("c3", 16, -1), ("c1", 16, -1)]
    acts = [x.double().reshape(B, 16, 16, 16, -1)]
    F = torch.nn.functional
    for i, (typ, s, skip) in enumerate(layers):
        a = acts[-1]
        if typ == "c3":
            p = F.pad(a, (0, 0, 1, 1, 1, 1, 1, 1))
            z = sum(p[:, dz:dz + s, dy:dy + s, dx:dx + s] @ W[i][dz * 9 + dy * 3 + dx]
                    for dz in range(3) for dy in range(3) for dx in range(3))
        elif typ == "d2":
            z = sum(a[:, t >> 2::2, (t >> 1) & 1::2, t & 1::2] @ W[i][t] for t in range(8))
        elif typ == "u2":
            z = torch.stack([a @ W[i][t] for t in range(8)], 4)  # B z y x 8 c
            z = z.reshape(B, s, s, s, 2, 2, 2, -1).permute(0, 1, 4, 2, 5, 3, 6, 7).reshape(B, 2 * s, 2 * s, 2 * s, -1)
        else:
            z = a @ W[i][0]
        z = z + b[i]
        if skip >= 0:
            z = z + acts[skip]
        acts.append(z if i == 8 else _Round.apply(torch.relu(z)))
    y = acts[-1].reshape(B, learned.VOX, -1)
    yk, v, m = y[..., :6], V.double(), Mw.double()[..., None]
    G, H = yk.transpose(1, 2) @ (m * yk), yk.transpose(1, 2) @ (m * v)
    r = v - yk @ torch.linalg.solve(G, H)
    loss = (m * r * r).sum((1, 2)) / 6.0
    grads = torch.autograd.grad(loss.mean(), W + b)
    return {"y": y.detach(), "loss": loss.detach(), "grads": [(grads[i], grads[9 + i]) for i in range(9)]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "batch":
        probs, srcs = _batch_problems(case, seed)
        if sum(_block_cost(p["mesh"])[0] for p in probs) > 2e14:
            return None
        z0, z = [], 0
        for p in probs:
            z0.append(z)
            z += p["mesh"][2] + 1
        shape = (z, max(p["mesh"][1] for p in probs), max(p["mesh"][0] for p in probs))
        out = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(case["rhs"])]
        for p, src, a in zip(probs, srcs, z0):
            M, N, P = p["mesh"]
            solve = _block_solver(p["kappa"], p["dom"], p["dirichlet"])
            for i in range(case["rhs"]):
                out[i][a:a + P, :N, :M] = solve(src[i])
        return [o.reshape(-1) for o in out]
    dom, faces = _domain(case), FIELDS[case["field"]][1]
    mesh = (case["M"], case["N"], case["P"])
    if kind == "apply":
        t, diag, _ = _operator(_kappa(case, seed), dom, faces)
        x = torch.randn(mesh[0] * mesh[1] * mesh[2], dtype=torch.float64, device="cuda", generator=_gen(seed, 17))
        return _matvec(t, diag, x.reshape(diag.shape)).reshape(-1)
    flops, size = _block_cost(mesh)
    if flops > 2e14 or size > 6e10 or not faces:  # pure Neumann: the elimination loses the solution's digits
        return None
    k = _kappa(case, seed)
    b = _source(case, seed).reshape(k.shape) + _operator(k, dom, faces)[2]
    return _block_solver(k, dom, faces)(b).reshape(-1)
