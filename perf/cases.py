"""Timed cases of the velocity solver, through its public entry points.

``listed()`` holds the cases, ``draw(rng)`` one more of the same ranges.
Each case has a ``kind``:

* ``solve``: a velocity solve.  ``entry = "host"`` is what a host model does
  every time step (new geometry, host arrays in and out: plan, upload, Picard
  loop, download); ``entry = "resident"`` a problem kept on the device, started
  from a velocity, run and read back.  ``maxiter`` caps the Picard iterations
  (a time-stepping model starts close to the answer and takes few), 200 PCG
  iterations per linear solve are the reference's cap;
* ``pcg``: the linear solver alone on a matrix held by the caller (the
  drop-in for the reference's own PCG calls);
* ``residual``: the allocation-free residual on the caller's device arrays;
* ``guess``: the learned initial velocity of a batch of domains;
* ``train``: one training step of the network behind it.

Every input is made from the seed.
"""
import ctypes
import math
import os

import numpy as np
import torch

from cism_b200 import configs, guess, net, solver

_WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(solver.__file__)), "weights", "unet_marine.bin")


def _solve(name, family, n, **kw):
    case = {"name": name, "kind": "solve", "family": family, "n": n, "nz": 11, "batch": 1, "entry": "resident",
            "mixed": False, "sia": False, "chrongear": False, "learned": False, "approx": 0, "law": 0,
            "maxiter": 5, "pcg_cap": 200, "relative_residual": False, "sizes": 3}
    case.update(kw)
    return case


def listed():
    return [
        # the allocation-free residual inside a time step: the dome of the
        # 31 x 31 x 10 workload, and the periodic slab of 160 x 160 x 11
        {"name": "residual_dome", "kind": "residual", "n": 31, "nz": 10, "periodic": 1},
        {"name": "residual_slab", "kind": "residual", "n": 160, "nz": 11, "periodic": 1},
        # the smallest whole solve: the 31 x 31 x 10 dome to convergence from
        # rest, standard PCG, diagonal preconditioner
        _solve("dome_converged", "dome", 31, nz=10, entry="host", maxiter=100),
        # the periodic slab of 160 x 160 x 11, FP64, standard PCG
        _solve("slab_fp64", "slab", 160, maxiter=3),
        # a time step of the 400 x 400 x 11 marine sheet in FP64 with the
        # reference's default preconditioner, from host arrays
        _solve("marine400_fp64", "marine", 400, sia=True, chrongear=True, entry="host", maxiter=2),
        # the held-out marine evaluation set: four 256 x 256 x 11 sheets in
        # one resident problem, mixed precision, learned start
        _solve("marine256x4_mixed", "marine", 256, batch=4, sia=True, chrongear=True, mixed=True, learned=True,
               maxiter=3, relative_residual=True),
        # the ensemble of uneven domes and slabs, mixed, batched, host arrays
        _solve("ensemble16_mixed", "ensemble", 96, batch=16, sia=True, chrongear=True, mixed=True, entry="host",
               maxiter=5, relative_residual=True),
        # the depth-integrated solve with a velocity-dependent sliding law
        _solve("diva128_sliding", "marine", 128, approx=configs.APPROX_DIVA, law=configs.BABC_COULOMB_POWERLAW_SCHOOF,
               chrongear=True, entry="host", maxiter=10),
        # a caller's own matrix: the 48 x 48 x 11 slab's first system
        {"name": "pcg_slab", "kind": "pcg", "n": 48, "nz": 11, "sia": True, "chrongear": True, "maxiters": 200},
        # the learned start alone, four 256 x 256 sheets
        {"name": "guess256x4", "kind": "guess", "n": 256, "nz": 11, "batch": 4},
        # one training step of that network: batch 8 of 128 x 128 grids
        {"name": "train128x8", "kind": "train", "n": 128, "batch": 8, "periodic": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["residual", "solve3d", "solve3d", "solve3d", "solve2d", "pcg", "guess", "train"])
    if kind == "residual":
        return {"kind": "residual", "n": _log(rng, 12, 160), "nz": rng.randint(3, 14), "periodic": rng.randint(0, 1)}
    if kind == "pcg":
        return {"kind": "pcg", "n": rng.randint(12, 56), "nz": rng.randint(4, 13), "sia": rng.random() < 0.5,
                "chrongear": rng.random() < 0.5, "maxiters": rng.choice([50, 200])}
    if kind == "guess":
        return {"kind": "guess", "n": rng.randint(48, 256), "nz": 11, "batch": rng.randint(1, 4)}
    if kind == "train":
        return {"kind": "train", "n": 8 * rng.randint(6, 18), "batch": rng.randint(2, 6), "periodic": rng.randint(0, 1)}
    if kind == "solve2d":
        case = _solve("", rng.choice(["marine", "slab"]), _log(rng, 32, 160), chrongear=rng.random() < 0.5,
                      approx=rng.choice([configs.APPROX_SSA, configs.APPROX_L1L2, configs.APPROX_DIVA]),
                      law=rng.choice([0, configs.BABC_POWERLAW, configs.BABC_COULOMB_POWERLAW_SCHOOF]),
                      entry=rng.choice(["host", "resident"]), maxiter=rng.randint(2, 10))
    else:
        family = rng.choice(["dome", "slab", "marine", "ensemble"])
        mixed = rng.random() < 0.5
        n = {"dome": _log(rng, 15, 64), "slab": _log(rng, 24, 160), "marine": _log(rng, 40, 300),
             "ensemble": rng.randint(32, 80)}[family]
        case = _solve("", family, n, nz=rng.choice([6, 8, 10, 11, 11, 14]), mixed=mixed, sia=rng.random() < 0.6,
                      chrongear=rng.random() < 0.6, entry=rng.choice(["host", "resident"]), maxiter=rng.randint(1, 3),
                      batch=rng.randint(3, 10) if family == "ensemble" else 1, sizes=rng.randint(1, 1000),
                      relative_residual=rng.random() < 0.5)
    case.pop("name")
    return case


# ---------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------
def _models(case, seed):
    rng = np.random.default_rng(seed)
    n, nz = case["n"], case.get("nz", 11)
    if case["family"] == "dome":
        ms = [configs.dome(n=n, nz=nz, radius=0.4 * n * 2000.0, hmax=float(rng.uniform(1500.0, 2500.0)),
                           flwa=1.0e-16 * float(rng.uniform(0.5, 2.0)))]
    elif case["family"] == "slab":
        ms = [configs.random_slab(rng, n=n, nz=nz)]
    elif case["family"] == "ensemble":
        # the sizes and shapes are the case's; friction and rate factor follow the seed
        ms = [m.copy(beta_external=m.beta_external * float(rng.uniform(0.7, 1.4)),
                     flwa=m.flwa * float(rng.uniform(0.7, 1.4)))
              for m in configs.ensemble(count=case["batch"], seed=case["sizes"], lo=max(16, n // 3), hi=n, nz=nz)]
    else:
        ms = [configs.marine(n=n, dx=2000.0 if 128 < n <= 300 else 4000.0, nz=nz, seed=seed + 7919 * i)
              for i in range(case.get("batch", 1))]
    out = []
    for i, m in enumerate(ms):
        if case.get("law"):
            m = configs.with_sliding(m, case["law"], seed=seed + i)
        m = m.copy(which_precond=configs.PRECOND_SIA if case.get("sia") else configs.PRECOND_DIAG,
                   which_sparse=configs.SPARSE_PCG_CHRONGEAR if case.get("chrongear") else configs.SPARSE_PCG_STANDARD,
                   maxiter_nonlinear=case.get("maxiter", 100), pcg_maxiters=case.get("pcg_cap", 200),
                   approx_2d=case.get("approx", 0),
                   which_resid=(configs.RESID_L2NORM_RELATIVE if case.get("relative_residual")
                                else configs.RESID_MAXU))
        out.append(m)
    return out


def _start(m, case):
    """Rest, or for a capped solve the shallow-ice velocity (a start near the answer)."""
    if case["maxiter"] >= 100:
        return guess.zero_guess(m)
    u, v = guess.sia_guess(m)
    speed = np.maximum(np.sqrt(u * u + v * v), 1.0e-30)
    f = np.minimum(1.0, 2000.0 / speed)  # a shelf without friction has no shallow-ice balance
    return u * f, v * f


_loaded = {}


def _context(learned):
    ctx = solver.default_context()
    if learned and not _loaded:
        ctx.load_guess(_WEIGHTS)
        _loaded["unet"] = True
    return ctx


def _prepare_solve(case, seed):
    learned = bool(case.get("learned"))
    ctx = _context(learned)
    ms = _models(case, seed)
    preps, us, vs = [], [], []
    for m in ms:
        u0, v0 = _start(m, case)
        p, u, v = solver.prepare(m, u0, v0, solver.MIXED if case["mixed"] else solver.FP64,
                                 guess_mode=solver.GUESS_LEARNED if learned else solver.GUESS_GIVEN)
        preps.append(p)
        us.append(u)
        vs.append(v)
    s = {"kind": "solve", "entry": case["entry"], "ctx": ctx, "preps": preps, "us": us, "vs": vs,
         "learned": learned, "diva": case["approx"] == configs.APPROX_DIVA}
    if s["diva"]:  # the solve writes this state back: every pass starts from the same one
        s["state"] = [{k: p.arrays[k].copy() for k in ("uvel_2d", "vvel_2d", "btractx", "btracty")} for p in preps]
    if case["entry"] == "resident":
        s["problem"] = ctx.problem(preps)
    return s


def _run_solve(s):
    if s["diva"]:
        for p, st in zip(s["preps"], s["state"]):
            for k, a in st.items():
                p.arrays[k][...] = a
    n = len(s["preps"])
    if s["entry"] == "host":
        if n == 1:
            u, v, e, _ = s["ctx"].solve_prepared(s["preps"][0], s["us"][0], s["vs"][0])
            us, vs, es = [u], [v], [e]
        else:
            us, vs, es, _ = s["ctx"].batch_solve(s["preps"], s["us"], s["vs"], want_efvs=True)
    else:
        p = s["problem"]
        if s["learned"]:
            p.set_guess([None] * n, [None] * n)
        else:
            p.set_guess(s["us"], s["vs"])
        p.run()
        us, vs, es = p.get(want_efvs=True)
    return {"u": us, "v": vs, "efvs": es}


def _prepare_pcg(case, seed):
    ctx = _context(False)
    m = configs.random_slab(np.random.default_rng(seed), n=case["n"], nz=case["nz"])
    u0, v0 = guess.sia_guess(m)
    p, u, v = solver.prepare(m, u0, v0)
    A, bu, bv, _ = ctx.assemble(p, u, v)
    return {"kind": "pcg", "ctx": ctx, "m": m, "active": p.arrays["active_vertex"], "A": A, "b": (bu, bv),
            "x": (u, v), "precond": 2 if case["sia"] else 1, "variant": 3 if case["chrongear"] else 2,
            "maxiters": case["maxiters"]}


def _run_pcg(s):
    xu, xv, err, _, _ = s["ctx"].pcg_solve(s["m"], s["active"], s["A"], *s["b"], *s["x"], precond=s["precond"],
                                           variant=s["variant"], maxiters=s["maxiters"])
    return {"xu": xu, "xv": xv}


def _residual_inputs(case, seed):
    """A system in the reference's layout on the device: blocks of a stiffness
    matrix's magnitudes (a strong diagonal, neighbours of both signs), a round
    ice sheet in the middle of the grid."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    n, nz = case["n"], case["nz"]
    V = n + 3
    A = [torch.randn((V, V, nz, 27), generator=g, device="cuda", dtype=torch.float64) * 1.0e4 for _ in range(4)]
    A[0][..., 13] += 2.0e5
    A[3][..., 13] += 2.0e5
    vec = [torch.randn((V, V, nz), generator=g, device="cuda", dtype=torch.float64) * s for s in (300.0, 300.0, 1e7, 1e7)]
    c = torch.arange(V, device="cuda", dtype=torch.float64) - (V - 1) / 2
    active = (c[:, None] ** 2 + c[None, :] ** 2 <= (0.45 * n) ** 2).to(torch.int32).contiguous()
    return V, nz, A, vec, active


def _prepare_residual(case, seed):
    V, nz, A, vec, active = _residual_inputs(case, seed)
    out = [torch.empty((V, V, nz), device="cuda", dtype=torch.float64) for _ in range(2)]
    norms = torch.empty(3, device="cuda", dtype=torch.float64)
    f = solver.lib().bp_residual_noalloc
    f.argtypes = [ctypes.c_int] * 4 + [ctypes.c_void_p] * 13
    f.restype = ctypes.c_int
    _context(False)
    return {"kind": "residual", "f": f, "dims": (V + 1, V + 1, nz, case["periodic"]), "active": active, "A": A,
            "vec": vec, "out": out, "norms": norms}


def _run_residual(s):
    rc = s["f"](*s["dims"], s["active"].data_ptr(), *[a.data_ptr() for a in s["A"]],
                *[a.data_ptr() for a in s["vec"]], *[a.data_ptr() for a in s["out"]], s["norms"].data_ptr(),
                torch.cuda.current_stream().cuda_stream)
    if rc != 0:
        raise RuntimeError(f"bp_residual_noalloc: status {rc}")
    return {"ru": s["out"][0], "rv": s["out"][1], "norms": s["norms"]}


def _prepare_guess(case, seed):
    ctx = _context(True)
    preps = []
    for i in range(case["batch"]):
        m = configs.marine(n=case["n"], dx=2000.0, nz=case["nz"], seed=seed + 7919 * i)
        preps.append(solver.prepare(m, guess_mode=solver.GUESS_LEARNED)[0])
    return {"kind": "guess", "problem": ctx.problem(preps)}


def _run_guess(s):
    p = s["problem"]
    p.set_guess([None] * p.n, [None] * p.n)
    us, vs = p.get_guess()
    return {"u": us, "v": vs}


def _layer_shapes():
    """(cin, cout, 3 x 3) of the network's convolutions in order."""
    c = net.CHANNELS
    out, cin = [], net.N_IN
    for ch in c:
        out += [(cin, ch, True), (ch, ch, True)]
        cin = ch
    for lv in range(len(c) - 2, -1, -1):
        out += [(c[lv + 1] + c[lv], c[lv], True), (c[lv], c[lv], True)]
    return out + [(c[0], 24, False)]


def _train_inputs(case, seed):
    """Weights, a batch of smooth normalised fields, targets and the ice mask."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def rand(*shape):
        return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)

    B, n = case["batch"], case["n"]
    w = [rand(co, (9 if k3 else 1) * ci) * math.sqrt(2.0 / ((9 if k3 else 1) * ci)) for ci, co, k3 in _layer_shapes()]
    b = [0.1 * rand(co) for _, co, _ in _layer_shapes()]

    def smooth(ch):
        low = rand(B, ch, max(2, n // 8), max(2, n // 8))
        up = torch.nn.functional.interpolate(low, size=(n, n), mode="bilinear", align_corners=False)
        return (up + 0.1 * rand(B, ch, n, n)).permute(0, 2, 3, 1).contiguous()

    x = smooth(net.N_IN).to(torch.bfloat16)
    t = smooth(24)
    c = torch.arange(n, device="cuda", dtype=torch.float32) - (n - 1) / 2
    mask = (c[:, None] ** 2 + c[None, :] ** 2 <= (0.45 * n) ** 2).to(torch.float32).expand(B, n, n).contiguous()
    return w, b, x, t, mask


def _prepare_train(case, seed):
    w, b, x, t, mask = _train_inputs(case, seed)
    model = net.UNet(n_out=24)
    for cv, wi, bi in zip(model.convs(), w, b):
        cv.w.copy_(wi)
        cv.b.copy_(bi)
        cv.refresh()
    return {"kind": "train", "model": model, "x": x, "t": t, "mask": mask, "periodic": case["periodic"], "step": 0}


def _run_train(s):
    m = s["model"]
    s["step"] += 1
    y = m.forward(s["x"], s["periodic"], train=True)
    loss, dy = net.mse(y, s["t"], s["mask"])
    m.backward(dy)
    m.adam(6.0e-4, s["step"])
    return {"loss": loss, "y": y, "gw": [c.gw for c in m.convs()], "gb": [c.gb for c in m.convs()],
            "w": [c.w for c in m.convs()], "b": [c.b for c in m.convs()]}


_PREPARE = {"solve": _prepare_solve, "pcg": _prepare_pcg, "residual": _prepare_residual, "guess": _prepare_guess,
            "train": _prepare_train}
_RUN = {"solve": _run_solve, "pcg": _run_pcg, "residual": _run_residual, "guess": _run_guess, "train": _run_train}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed) % (1 << 31))


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------
def _columns(case):
    """Active columns per domain (an estimate for the drawn geometries)."""
    n = case["n"]
    f = {"dome": math.pi * 0.4 ** 2, "slab": 1.0, "marine": math.pi * 0.45 ** 2 * (14.0 / 15.0),
         "ensemble": 0.5 * (1.0 + math.pi * 0.4 ** 2)}[case.get("family", "slab")]
    side2 = n * n if case.get("family") != "ensemble" else ((n + max(16, n // 3)) / 2.0) ** 2
    return f * side2


def work(case):
    kind = case["kind"]
    if kind == "residual":
        V = case["n"] + 3
        rows = math.pi * (0.45 * case["n"]) ** 2 * case["nz"]
        return {"bytes": rows * (4 * 27 * 8 + 4 * 8) + V * V * case["nz"] * 16.0, "flops": rows * (27 * 8 + 8)}
    if kind == "pcg":
        N = case["n"] ** 2 * case["nz"]
        its = case["maxiters"]
        return {"bytes": N * (864.0 + 64.0 + its * (448.0 + 12 * 16.0)), "flops": N * its * (27 * 8 + 30.0)}
    if kind in ("guess", "train"):
        px = case["batch"] * (8 * ((case["n"] + 7) // 8)) ** 2
        lv = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0]
        flops = by = 0.0
        for k, (ci, co, k3) in zip(lv, _layer_shapes()):
            p = px / 4.0 ** k
            flops += 2.0 * p * ci * co * (9 if k3 else 1)
            by += 2.0 * p * (ci + co)  # BF16 activations, read once and written once
        if kind == "guess":
            return {"bytes": by + px * case["nz"] * 16.0, "flops": flops}
        return {"bytes": 3.0 * by, "flops": 3.0 * flops}
    levels = 1 if case["approx"] else case["nz"]
    N = _columns(case) * case["batch"] * levels
    # converged runs: about 30 Picard iterations of 75 PCG iterations
    picard, its = (case["maxiter"], case["pcg_cap"]) if case["maxiter"] < 100 else (30, 75)
    offsets = 5 if case["approx"] else 14
    matrix = (offsets - 1) * 16.0 + 32.0 if case["mixed"] else offsets * 32.0
    vec = 12 * 16.0 + (48.0 if case["sia"] else 0.0)
    asm = offsets * 32.0 + 640.0
    return {"bytes": N * picard * (asm + its * (matrix + vec)) + 6.0 * 8.0 * N,
            "flops": N * picard * ((300.0 if case["approx"] else 18.1e3) + its * (offsets * 2 * 8.0 + 30.0))}


# ---------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------
def _exact_residual(case, seed):
    V, nz, A, vec, active = _residual_inputs(case, int(seed) % (1 << 31))
    xu, xv, bu, bv = vec
    pad = torch.nn.functional.pad
    Xu, Xv = pad(xu, (1, 1, 1, 1, 1, 1)), pad(xv, (1, 1, 1, 1, 1, 1))
    yu, yv = torch.zeros_like(xu), torch.zeros_like(xv)
    for m in range(27):
        i, j, k = m % 3, (m // 3) % 3, m // 9
        su, sv = Xu[j:j + V, i:i + V, k:k + nz], Xv[j:j + V, i:i + V, k:k + nz]
        yu += A[0][..., m] * su + A[1][..., m] * sv
        yv += A[2][..., m] * su + A[3][..., m] * sv
    lo = 2 if case["periodic"] else 1
    own = torch.zeros((V, V), dtype=torch.bool, device="cuda")
    own[lo:V - 1, lo:V - 1] = True
    rows = (own & (active != 0))[..., None]
    ru, rv = torch.where(rows, yu - bu, 0.0), torch.where(rows, yv - bv, 0.0)
    nr = (ru.square().sum() + rv.square().sum()).sqrt()
    nb = torch.where(rows, bu.square() + bv.square(), 0.0).sum().sqrt()
    return {"ru": ru, "rv": rv, "norms": torch.stack([nr, nb, nr / nb])}


def _exact_train(case, seed):
    w, b, x, t, mask = _train_inputs(case, int(seed) % (1 << 31))
    F = torch.nn.functional
    W = [v.double().requires_grad_() for v in w]
    Bi = [v.double().requires_grad_() for v in b]
    shapes = _layer_shapes()
    mode = "circular" if case["periodic"] else "constant"

    def conv(h, i, act=True):
        ci, co, k3 = shapes[i]
        if k3:
            k = W[i].view(co, 3, 3, ci).permute(0, 3, 1, 2)
            h = F.conv2d(F.pad(h, (1, 1, 1, 1), mode=mode), k, Bi[i])
        else:
            h = F.conv2d(h, W[i].view(co, ci, 1, 1), Bi[i])
        return F.gelu(h) if act else h

    h, skips, i = x.double().permute(0, 3, 1, 2), [], 0
    for lv in range(len(net.CHANNELS)):
        if lv:
            h = F.avg_pool2d(h, 2)
        h = conv(conv(h, i), i + 1)
        i += 2
        skips.append(h)
    for lv in range(len(net.CHANNELS) - 2, -1, -1):
        h = torch.cat([F.interpolate(h, scale_factor=2, mode="nearest"), skips[lv]], dim=1)
        h = conv(conv(h, i), i + 1)
        i += 2
    y = conv(h, i, act=False).permute(0, 2, 3, 1)
    m = mask.double()[..., None]
    loss = (((y - t.double()) * m) ** 2).sum() / (mask.double().sum() * t.shape[-1])
    loss.backward()
    none = [None] * len(W)
    return {"loss": float(loss.detach()), "y": y.detach().contiguous(), "gw": [v.grad for v in W],
            "gb": [v.grad for v in Bi], "w": none, "b": none}


def exact(case, seed):
    """In 64 bits for the residual and the network; a velocity solve's result
    depends on where its iterations stop, so it has no such value."""
    if case["kind"] == "residual":
        return _exact_residual(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None
