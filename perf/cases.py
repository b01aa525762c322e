"""The calls a user of this framework makes, as cases that can be timed.

Three kinds of program use libllg.so:

* a program that integrates a film with the library's own BDF integrator
  ("run"), or many films at once ("batch");
* a program that drives the operator callbacks from its own CVODE, which per
  Newton iteration forms the iterate and evaluates f ("residual"), per Krylov
  iteration applies Jv and the preconditioner and orthogonalises ("krylov"),
  and per preconditioner refresh sets the block inverse up ("setup");
* a program that needs the demagnetising field alone ("demag"), or trains and
  applies the learned preconditioner ("learned_apply", "learned_grad").

prepare() holds what such a program holds before the call: a context with its
geometry and demag plan, and device vectors made from the seed.  run() is one
pass.  exact() states the same operators in plain torch, in 64 bits.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "gpu-micromagnetics-irregular_b200"))
import llg  # noqa: E402

DEV = "cuda"


# ── the cases ───────────────────────────────────────────────────────────
def listed():
    return [
        # the smallest call: one Newton residual of the 128x64 local film
        # (free edges, no demag) from a user's own CVODE; launches and latency
        {"name": "residual-local-128x64", "kind": "residual", "shape": "bulk", "ng": 128, "ny": 64,
         "demag": "off", "precision": "fp64", "strength": 0.0},
        # the same film integrated by the library: every kernel is a few us, so
        # launches and read-backs count
        {"name": "run-local-128x64", "kind": "run", "shape": "bulk", "ng": 128, "ny": 64, "demag": "off",
         "precision": "fp64", "strength": 0.0, "gs": "auto", "krylov": "fp64", "outputs": 20},
        # the benchmark film (square hole, open demag) in the plain FP64 form
        {"name": "run-film-1536x512-fp64", "kind": "run", "shape": "hole", "ng": 1536, "ny": 512, "demag": "open",
         "precision": "fp64", "strength": 4.0, "gs": "classical", "krylov": "fp64", "outputs": 20},
        # the same in the form the benchmark quotes: mixed demag, FP32 Krylov basis
        {"name": "run-film-1536x512-mixed32", "kind": "run", "shape": "hole", "ng": 1536, "ny": 512,
         "demag": "open", "precision": "mixed", "strength": 4.0, "gs": "classical", "krylov": "fp32",
         "outputs": 20},
        # Voronoi polycrystal (window and per-cell axes) at a ragged size with
        # the default options: above 500,000 unknowns these pick modified
        # Gram-Schmidt, as CVODE programs of the reference do
        {"name": "run-polycrystal-720x400-fp64", "kind": "run", "shape": "polycrystal", "ng": 720, "ny": 400,
         "demag": "open", "precision": "fp64", "strength": 1.0, "gs": "auto", "krylov": "fp64", "outputs": 20},
        # one Newton residual of the benchmark film from a user's own CVODE
        {"name": "residual-film-1536x512-fp64", "kind": "residual", "shape": "hole", "ng": 1536, "ny": 512,
         "demag": "open", "precision": "fp64", "strength": 4.0},
        # the compact circle on the 2048x2048 grid (about 20 % of the cells
        # active, index lists, periodic mixed demag): the largest single call
        {"name": "residual-compact-2048-mixed", "kind": "residual", "shape": "circle", "ng": 2048, "ny": 2048,
         "demag": "periodic", "precision": "mixed", "strength": 2.0},
        # one Krylov iteration of a user's own CVODE on the benchmark film:
        # Jv, the preconditioner and classical Gram-Schmidt against 3 vectors
        {"name": "krylov-film-1536x512", "kind": "krylov", "shape": "hole", "ng": 1536, "ny": 512,
         "demag": "open", "precision": "fp64", "strength": 4.0, "basis": 3},
        # the demag field alone at an odd size (750x450 transforms: factors 2, 3, 5)
        {"name": "demag-375x225-fp64", "kind": "demag", "shape": "bulk", "ng": 375, "ny": 225, "demag": "open",
         "precision": "fp64", "strength": 2.5},
        # the batched mixed workload: 16 films of 256x256 .. 1024x512 advanced
        # together from the host thread pool
        {"name": "batch-16-mixed", "kind": "batch", "count": 16, "outputs": 5},
        # the learned preconditioner on the compact circle, one application
        {"name": "learned-apply-2048", "kind": "learned_apply", "shape": "circle", "ng": 2048, "ny": 2048},
        # one training step of it: forward, loss and backward on 16 patches of 32x32
        {"name": "learned-grad-16x32", "kind": "learned_grad", "patches": 16, "side": 32},
    ]


def _smooth(n):
    """Whether n has no prime factor above 64 (the transform lengths accepted)."""
    for p in range(2, 64):
        while n % p == 0:
            n //= p
    return n == 1


def _size(rng, lo, hi):
    """A length between lo and hi, spread over its logarithm, even or odd."""
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if rng.random() < 0.3:
            n = max(lo, min(hi, 1 << int(round(math.log2(n)))))
        if _smooth(n):
            return n


def draw(rng):
    kind = rng.choice(["residual", "residual", "krylov", "setup", "demag", "demag", "run", "learned_grad"])
    if kind == "learned_grad":
        return {"kind": kind, "patches": rng.randint(1, 32), "side": rng.randint(8, 64)}
    # 1,536 x 1,024 at most (the transforms are twice that in open mode), 33 x 17 at least
    c = {"kind": kind, "shape": rng.choice(["bulk", "hole", "circle", "polycrystal"]),
         "ng": _size(rng, 33, 1536), "ny": _size(rng, 17, 1024),
         "demag": rng.choice(["open", "open", "periodic"]) if kind == "demag" else
         rng.choice(["off", "open", "open", "periodic"]),
         "precision": rng.choice(["fp64", "fp64", "mixed"]),
         "strength": round(rng.uniform(1.0, 4.0), 3)}
    if c["demag"] == "off":
        c["precision"], c["strength"] = "fp64", 0.0
    if kind == "demag":
        c["shape"] = "bulk"
    if kind == "krylov":
        c["basis"] = rng.randint(1, 5)
    if kind == "run":
        c["ng"], c["ny"] = min(c["ng"], 768), min(c["ny"], 512)
        c["gs"] = rng.choice(["auto", "classical"])
        c["krylov"] = rng.choice(["fp64", "fp32"]) if c["gs"] == "classical" else "fp64"
        c["outputs"] = rng.randint(1, 4)
    return c


# ── inputs ──────────────────────────────────────────────────────────────
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _params(case):
    shape = case["shape"]
    kw = dict(demag_mode={"off": llg.DEMAG_OFF, "open": llg.DEMAG_OPEN, "periodic": llg.DEMAG_PERIODIC}[case["demag"]],
              demag_strength=case["strength"], demag_precision=llg.DEMAG_MIXED if case["precision"] == "mixed"
              else llg.DEMAG_FP64)
    if case["demag"] != "off":
        kw["norm_kind"] = llg.NORM_REG
    if case["demag"] == "periodic":
        kw["bc"] = llg.BC_PERIODIC
    if shape == "circle":
        kw["exec_model"] = llg.EXEC_COMPACT
    if shape == "polycrystal":
        kw["windowed"] = 1
    return llg.default_params(case["ng"], case["ny"], **kw)


def _geometry(case, seed):
    """Active cells (None: all) and, for a polycrystal, window and axes."""
    ng, ny, shape = case["ng"], case["ny"], case["shape"]
    if shape == "bulk":
        return {}
    if shape == "polycrystal":
        grains = max(3, min(72, ng * ny // 4000))
        g = llg.default_geom(ng, ny, geometry_kind=llg.GEOM_POLYCRYSTAL, num_grains=grains, dead_grain_frac=0.16,
                             grain_z_bias=1.0, hole_seed=seed % 100000 + 1)
        d = llg.build_geometry_device(g)
        return {"w": d["w"], "msk3": d["msk3"], "nsk3": d["nsk3"]}
    # cell-centre predicates of the two cut shapes
    x = torch.arange(ng, device=DEV, dtype=torch.float64) - 0.5 * (ng - 1)
    yv = torch.arange(ny, device=DEV, dtype=torch.float64)[:, None] - 0.5 * (ny - 1)
    if shape == "hole":   # square of side 0.25 ny in the middle
        act = ~((x.abs() <= 0.125 * ny) & (yv.abs() <= 0.125 * ny))
    else:                 # ellipse of half axes 0.25 ng, 0.25 ny
        act = (x / (0.25 * ng)) ** 2 + (yv / (0.25 * ny)) ** 2 <= 1.0
    return {"act": act.reshape(-1)}


def _make_context(case, geo, stream=None):
    ctx = llg.Context(_params(case), stream)
    if case["shape"] == "polycrystal":
        ctx.set_window(*(geo[k].cpu().numpy() for k in ("w", "msk3", "nsk3")))
    elif case["shape"] == "circle":
        act = geo["act"].cpu().numpy()
        ids = np.arange(act.size, dtype=np.int32)
        ctx.set_active_ids(ids[act], ids[~act])
    elif case["shape"] == "hole":
        ctx.set_mask(np.tile(geo["act"].cpu().numpy().astype(np.float64), 3))
    return ctx


def _state(case, geo, seed):
    """A film's magnetisation: a vortex on the circle, else domains along x with
    their walls, every component jittered by 0.01, |m| = 1; 0 in the holes."""
    g, ng, ny = _gen(seed), case["ng"], case["ny"]
    x = torch.arange(ng, device=DEV, dtype=torch.float64)[None, :].expand(ny, ng)
    y = torch.arange(ny, device=DEV, dtype=torch.float64)[:, None].expand(ny, ng)
    if case["shape"] == "circle":
        m = torch.stack([-(y - 0.5 * (ny - 1)), x - 0.5 * (ng - 1), torch.full_like(x, 0.1 * ng)])
    elif case["shape"] == "polycrystal":
        s = torch.tanh((0.5 * ng - x) / 6.0)
        m = torch.stack([s, 0.3 * (1 - s * s), 0.1 * torch.ones_like(x)])
    else:
        m = torch.stack([torch.ones_like(x), 0.05 * torch.sin(0.07 * y), torch.zeros_like(x)])
    m = m / m.norm(dim=0).clamp_min(1e-3)
    m = m + 0.01 * (2 * torch.rand(m.shape, generator=g, device=DEV, dtype=torch.float64) - 1)
    m = m / m.norm(dim=0)
    if "act" in geo:
        m = m * geo["act"].reshape(ny, ng)
    if "w" in geo:
        m = m * (geo["w"].reshape(ny, ng) > 0)
    return m.reshape(-1).contiguous()


def _vectors(case, seed):
    """What one Newton or Krylov iteration of a user's CVODE holds."""
    n3 = 3 * case["ng"] * case["ny"]
    g = _gen(seed + 1)
    rnd = lambda s: s * torch.randn(n3, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    geo = _geometry(case, seed)
    v = {"geo": geo, "zn0": _state(case, geo, seed), "gamma": 0.02}
    if case["kind"] == "residual":
        v["ycor"] = rnd(1e-4)
    elif case["kind"] == "krylov":
        v["v"] = rnd(1e-3)
        q = torch.linalg.qr(torch.randn(n3, case["basis"], generator=g, device=DEV, dtype=torch.float64))[0]
        v["basis"] = [q[:, k].contiguous() for k in range(case["basis"])]
    elif case["kind"] == "setup":
        v["r"] = rnd(1e-3)
    return v


def _opts(case):
    gs = {"auto": llg.GS_AUTO, "classical": llg.GS_CLASSICAL}[case["gs"]]
    return llg.default_solver_opts(gs_type=gs, mxstep=5000,
                                   krylov_precision=llg.KRYLOV_FP32 if case["krylov"] == "fp32" else llg.KRYLOV_FP64)


def _patches(case, seed):
    nb, P = case["patches"], case["side"]
    g = np.random.default_rng(int(seed) + 5)
    m = g.standard_normal((nb, 3, P, P)).astype(np.float32) * 0.2
    m[:, 0] += 1.0
    m /= np.sqrt((m * m).sum(axis=1, keepdims=True))
    u = (1e-3 * g.standard_normal((nb, 3, P, P))).astype(np.float32)
    x = (u * 0.9 + 1e-4 * g.standard_normal((nb, 3, P, P))).astype(np.float32)
    return {"w": (0.05 * g.standard_normal(llg.LEARNED_NWEIGHTS)).astype(np.float32), "u": u, "m": m, "x": x,
            "ewt": (1e4 * (0.5 + g.random((nb, 3, P, P)))).astype(np.float32),
            "mask": (g.random((nb, P, P)) < 0.9).astype(np.float32),
            "gamma": (0.01 + 0.02 * g.random(nb)).astype(np.float32)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "learned_grad":
        return {"case": case, "p": _patches(case, seed)}
    if kind == "batch":
        insts = llg.config4_instances(case["count"])
        b = llg.Batch([i["params"] for i in insts])
        y0, g = [], _gen(seed)
        for ctx, inst in zip(b.ctx, insts):   # the workload's films, their states jittered by the seed
            y = torch.from_numpy(llg.setup_instance(ctx, inst)).to(DEV).reshape(3, -1)
            on = y.norm(dim=0) > 0
            y = y + 0.01 * (2 * torch.rand(y.shape, generator=g, device=DEV, dtype=torch.float64) - 1)
            y0.append((y / y.norm(dim=0) * on).reshape(-1))
        return {"case": case, "batch": b, "y0": y0, "out": [torch.empty_like(y) for y in y0],
                "opts": llg.default_solver_opts(gs_type=llg.GS_CLASSICAL)}
    if kind == "learned_apply":
        c = dict(case, demag="off", precision="fp64", strength=0.0)
        geo = _geometry(c, seed)
        p = _params(c)
        p.precond_kind = llg.PREC_LEARNED
        ctx = llg.Context(p)
        act = geo["act"].cpu().numpy()
        ids = np.arange(act.size, dtype=np.int32)
        ctx.set_active_ids(ids[act], ids[~act])
        g = _gen(seed + 2)
        m = _state(c, geo, seed)
        z = 1e-3 * torch.randn(m.numel(), generator=g, device=DEV, dtype=torch.float64)
        w = (0.05 * np.random.default_rng(seed).standard_normal(llg.LEARNED_NWEIGHTS)).astype(np.float32)
        ctx.learned_set_weights(w)
        return {"case": case, "ctx": ctx, "z": z, "m": m, "ewt": 1.0 / (1e-4 * m.abs() + 1e-6),
                "out": torch.empty_like(z)}
    s = _vectors(case, seed)
    s["case"] = case
    s["ctx"] = ctx = _make_context(case, s["geo"])
    new = lambda: torch.zeros_like(s["zn0"])  # noqa: E731
    if kind == "run":
        s["opts"], s["y"] = _opts(case), new()
    elif kind == "demag":
        s["h"] = new()
    elif kind == "residual":
        s["y"], s["ydot"] = new(), new()
    else:   # the iterate at which the Jacobian stands, its f and the block inverse
        s["y"], s["ydot"] = s["zn0"].clone(), new()
        ctx.rhs(0.0, s["y"], s["ydot"])
        if kind == "krylov":
            ctx.psetup(0.0, s["y"], s["ydot"], 0, s["gamma"])
            s.update(Jv=new(), u=new(), z=new(), w=new())
        else:
            s["z"] = new()
    return s


# ── one pass ────────────────────────────────────────────────────────────
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "residual":   # y = zn0 + ycor, then f(y) (normalises y in place)
        s["ctx"].linear_combination((1.0, 1.0), (s["zn0"], s["ycor"]), s["y"])
        s["ctx"].rhs(0.0, s["y"], s["ydot"])
        return {"y": s["y"], "ydot": s["ydot"]}
    if kind == "krylov":     # w = P^-1 (I - gamma J) v orthogonalised against the basis
        ctx = s["ctx"]
        ctx.jtv(s["v"], s["Jv"], 0.0, s["y"], s["ydot"])
        ctx.linear_combination((1.0, -s["gamma"]), (s["v"], s["Jv"]), s["u"])
        ctx.psolve(0.0, s["y"], s["ydot"], s["u"], s["z"], s["gamma"])
        d = ctx.dot_multi(s["z"], s["basis"])
        ctx.linear_combination([1.0] + [-x for x in d], [s["z"]] + s["basis"], s["w"])
        return {"Jv": s["Jv"], "z": s["z"], "dots": np.array(d), "w": s["w"],
                "norm": np.array(ctx.dot_multi(s["w"], [s["w"]]))}
    if kind == "setup":
        s["ctx"].psetup(0.0, s["y"], s["ydot"], 0, s["gamma"])
        s["ctx"].psolve(0.0, s["y"], s["ydot"], s["r"], s["z"], s["gamma"])
        return s["z"]
    if kind == "demag":
        s["ctx"].demag_apply(s["zn0"], s["h"])
        return s["h"]
    if kind == "run":        # from the initial state, output every 0.1
        s["ctx"].integrator_init(0.0, s["zn0"], s["opts"])
        for k in range(1, case["outputs"] + 1):
            s["ctx"].integrate(0.1 * k, s["y"])
        return s["y"]
    if kind == "batch":
        s["batch"].integrator_init(0.0, s["y0"], s["opts"])
        for k in range(1, case["outputs"] + 1):
            s["batch"].integrate(0.1 * k, s["out"])
        return s["out"]
    if kind == "learned_apply":
        n2 = s["ctx"].learned_apply(s["z"], s["m"], s["ewt"], 0.02, s["out"])
        return {"out": s["out"], "norm2": np.array(n2)}
    p = s["p"]
    loss, grad, z = llg.learned_loss_grad(p["w"], p["u"], p["m"], p["mask"], p["ewt"], p["x"], p["gamma"])
    return {"loss": loss, "grad": grad, "z": z}


# ── what a pass cannot do without ───────────────────────────────────────
def _demag_work(case):
    """Field of one state: the state in, the tensor spectra once (even in both
    frequencies in open mode, in y in periodic mode), the field out; FFT flops."""
    ng, ny = case["ng"], case["ny"]
    if case["demag"] == "off":
        return 0.0, 0.0
    k = 2 if case["demag"] == "open" else 1
    px, py = k * ng, k * ny
    e = 4 if case["precision"] == "mixed" else 8
    hx = px // 2 + 1
    rows = 2 * 3 * ny * 2.5 * px * math.log2(px)
    cols = 2 * 3 * hx * 5.0 * py * math.log2(py)
    tensor = hx * (py // 2 + 1) * 4 * e
    return tensor, rows + cols + 28.0 * hx * py


def work(case):
    kind = case["kind"]
    if kind == "learned_grad":
        px = case["patches"] * case["side"] ** 2
        return {"bytes": 4.0 * (px * 17 + 2 * 4032), "flops": 3 * 2.0 * 4032 * px}
    if kind == "batch":
        # about 20 BDF steps for each 0.1 of an instance, of 150,000 cells on average
        n = case["count"] * 0.15e6
        return {"bytes": case["outputs"] * 20 * n * 700.0, "flops": case["outputs"] * 20 * n * 1500.0}
    n = float(case["ng"] * case["ny"])
    if kind == "learned_apply":
        return {"bytes": 97.0 * n, "flops": 2 * 4032.0 * n * math.pi * 0.0625}
    db, df = _demag_work(case)
    extra = {"polycrystal": 56.0, "bulk": 0.0}.get(case["shape"], 1.0) * n
    if kind == "demag":
        return {"bytes": 48 * n + db, "flops": df}
    if kind == "residual":
        return {"bytes": 96 * n + extra + db, "flops": 80 * n + df}
    if kind == "krylov":   # v, y, block inverse, basis in; Jv, z, w out
        return {"bytes": (48 + 72 + 72 + 24 * case["basis"]) * n + extra, "flops": (200 + 12 * case["basis"]) * n}
    if kind == "setup":    # y, field, r in; block inverse and z out
        return {"bytes": (72 + 72 + 24) * n + extra, "flops": 400 * n}
    # a BDF step cannot do without one residual, the history in and out, two
    # Krylov iterations and their basis; about 8 steps in each 0.1
    steps = 8.0 * case["outputs"]
    kb = 4 if case["krylov"] == "fp32" else 8
    per = 96 * n + db + 2 * 3 * 24 * n + 2 * (48 + 9 * kb + 3 * 4 * kb) * n + extra
    return {"bytes": steps * per, "flops": steps * (df + 800 * n)}


# ── the same operators in plain torch, 64 bits ──────────────────────────
def _tensor(case):
    """The film's demag tensor (xx, yy, zz, xy) at every displacement of the
    transform grid: the closed-form integrals over a cell of side 0.99998 and
    thickness 1 seen from the 81 points (0.1 i, 0.1 j), |i|, |j| <= 4, averaged."""
    k = 2 if case["demag"] == "open" else 1
    px, py = k * case["ng"], k * case["ny"]

    def disp(n):
        i = torch.arange(n, device=DEV)
        return torch.where(i <= n - 1 - n // 2, i, i - n).double()

    dx, dy = disp(px)[None, :], disp(py)[:, None]
    acc = torch.zeros(4, py, px, device=DEV, dtype=torch.float64)
    for jy in range(-4, 5):
        for ix in range(-4, 5):
            X = [dx + 0.1 * ix - 0.49999, dx + 0.1 * ix + 0.49999]
            Y = [dy + 0.1 * jy - 0.49999, dy + 0.1 * jy + 0.49999]
            lz = {}
            for i in (0, 1):
                for j in (0, 1):
                    r = torch.sqrt(X[i] ** 2 + Y[j] ** 2 + 0.25)
                    for q, Z in ((0, -0.5), (1, 0.5)):
                        sg = -1.0 if (i + j + q) & 1 else 1.0
                        acc[0] += sg * torch.atan(Z * Y[j] / (X[i] * r))
                        acc[1] += sg * torch.atan(Z * X[i] / (Y[j] * r))
                        acc[2] += sg * torch.atan(X[i] * Y[j] / (Z * r))
                    lz[i, j] = torch.log((r + 0.5) / (r - 0.5))
            acc[3] += lz[0, 0] - lz[1, 0] - lz[0, 1] + lz[1, 1]
    acc /= 81.0
    if k == 2:   # displacements that a zero-padded convolution never uses
        acc[:, :, px // 2] = 0
        acc[:, py // 2, :] = 0
    return acc


def _demag(case, T, m):
    ny, ng = case["ny"], case["ng"]
    py, px = T.shape[1:]
    M = torch.fft.rfft2(m, s=(py, px))
    N = torch.fft.rfft2(T)
    H = torch.stack([N[0] * M[0] + N[3] * M[1], N[3] * M[0] + N[1] * M[1], N[2] * M[2]])
    return case["strength"] * torch.fft.irfft2(H, s=(py, px))[:, :ny, :ng]


def _nbsum(f, periodic):
    if periodic:
        return f.roll(1, -1) + f.roll(-1, -1) + f.roll(1, -2) + f.roll(-1, -2)
    out = torch.zeros_like(f)
    out[..., 1:] += f[..., :-1]
    out[..., :-1] += f[..., 1:]
    out[..., 1:, :] += f[..., :-1, :]
    out[..., :-1, :] += f[..., 1:, :]
    return out


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


class _Film:
    """Exchange 1, easy axis with constant 0.1, applied field (0, 0, 0.05), damping 0.02."""

    def __init__(self, case, geo):
        self.case, ny, ng = case, case["ny"], case["ng"]
        self.periodic = case["demag"] == "periodic"
        self.windowed = "w" in geo
        if self.windowed:
            self.w = geo["w"].reshape(ny, ng)
            self.axis = geo["msk3"].reshape(3, ny, ng)
            self.gate = self.w
        else:
            self.w = 1.0
            self.axis = torch.tensor([1.0, 0, 0], device=DEV, dtype=torch.float64).reshape(3, 1, 1)
            self.gate = geo["act"].reshape(ny, ng).double() if "act" in geo else 1.0
        self.T = _tensor(case) if case["demag"] != "off" else None

    def grid(self, v):
        return v.reshape(3, self.case["ny"], self.case["ng"])

    def normalised(self, y):
        return y / (y.norm(dim=0) + 1e-3) if self.case["demag"] != "off" else y

    def local(self, m):   # exchange and anisotropy
        return _nbsum(self.w * m, self.periodic) + 0.1 * (m * self.axis).sum(0) * self.axis

    def field(self, m):
        h = self.local(m)
        h[2] += 0.05
        return h + _demag(self.case, self.T, self.w * m) if self.T is not None else h

    def f(self, m):
        h = self.field(m)
        return self.gate * (_cross(h, m) + 0.02 * (h - (m * h).sum(0) * m))

    def jv(self, m, v):
        h, dh = self.local(m), self.local(v)
        d = (v * h).sum(0) + (m * dh).sum(0)
        return self.gate * (_cross(h, v) + _cross(dh, m) + 0.02 * (dh - d * m - (m * h).sum(0) * v))

    def psolve(self, m, gamma, r):
        """(I - gamma J_cell)^-1 r, J_cell the cell's own block with the self-demag term."""
        h = self.field(m)
        n0 = self.case["strength"] * self.T[:3, 0, 0] if self.T is not None else torch.zeros(3, device=DEV)
        ax = self.axis.expand_as(m)
        cols = []
        mh = (m * h).sum(0)
        for b in range(3):
            e = torch.zeros_like(m)
            e[b] = 1.0
            kb = 0.1 * ax * ax[b] + self.w * n0[b] * e
            eb = h[b] + (kb * m).sum(0)
            J = _cross(kb, m) + _cross(h, e) + 0.02 * (kb - eb * m - mh * e)
            cols.append(e - gamma * self.w * J)
        A = torch.stack(cols, 1).permute(2, 3, 0, 1)   # [ny, ng, a, b]
        z = torch.linalg.solve(A, r.permute(1, 2, 0)[..., None])[..., 0].permute(2, 0, 1)
        return z if self.windowed else z * self.gate


def _net(w, f):
    sizes = [(16, 9, 3, 3), (16, 16, 3, 3), (3, 16, 3, 3)]
    k = 0
    for s in sizes:
        n = math.prod(s)
        f = torch.nn.functional.conv2d(f, w[k:k + n].reshape(s), padding=1)
        k += n
    return f


def exact(case, seed):
    kind = case["kind"]
    if kind in ("run", "batch", "learned_apply"):   # (learned_apply rounds its network to BF16 on purpose)
        return None
    if kind == "learned_grad":
        p = {k: torch.from_numpy(v).to(DEV).double() for k, v in _patches(case, seed).items()}
        w = p["w"].requires_grad_()
        cr = lambda a, b: torch.linalg.cross(a, b, dim=1)  # noqa: E731
        mask = p["mask"][:, None]
        mu = cr(p["m"], p["u"])
        feat = torch.cat([p["u"], mu, cr(p["m"], mu)], 1) * mask
        z = (p["u"] + p["gamma"][:, None, None, None] * _net(w, feat)) * mask
        inner = (slice(None), slice(None), slice(3, -3), slice(3, -3))
        num = ((p["ewt"] * (z - p["x"]))[inner] ** 2).sum((1, 2, 3))
        den = ((p["ewt"] * p["x"])[inner] ** 2).sum((1, 2, 3))
        loss = (num / den).mean()
        loss.backward()
        return {"loss": loss.detach(), "grad": w.grad, "z": z.detach()}
    v = _vectors(case, seed)
    film = _Film(case, v["geo"])
    if kind == "demag":
        return _demag(case, film.T, film.grid(v["zn0"])).reshape(-1)
    if kind == "residual":
        y = film.normalised(film.grid(v["zn0"] + v["ycor"]))
        return {"y": y.reshape(-1), "ydot": film.f(y).reshape(-1)}
    y = film.normalised(film.grid(v["zn0"]))
    if kind == "setup":
        return film.psolve(y, v["gamma"], film.grid(v["r"])).reshape(-1)
    Jv = film.jv(y, film.grid(v["v"]))
    z = film.psolve(y, v["gamma"], film.grid(v["v"]) - v["gamma"] * Jv).reshape(-1)
    d = torch.stack([torch.dot(z, b) for b in v["basis"]])
    w = z - sum(d[k] * b for k, b in enumerate(v["basis"]))
    return {"Jv": Jv.reshape(-1), "z": z, "dots": d, "w": w, "norm": torch.dot(w, w).reshape(1)}
